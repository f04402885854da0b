"""The register split of the CTA-pair attention backward against what the compiler launches it with."""

import os
import re
import subprocess

import pytest

from teletron_b200 import build


def test_the_blocks_registers_cover_the_split(tmp_path):
    """``setmaxnreg.inc`` waits for registers that the block was launched with, and for ever if they are too few."""
    src = os.path.join(build.SRC, "attn_bwd_pair_tcgen05.cu")
    try:
        nvcc = build.find_nvcc()
    except RuntimeError:
        pytest.skip("needs nvcc")
    r = subprocess.run([nvcc] + build.NVCC_FLAGS + ["-Xptxas", "-v", "-I", build.SRC, "-c", src, "-o", str(tmp_path / "x.o")],
                       capture_output=True, text=True, check=True)
    used = int(re.search(r"Compiling entry function '\S*attn_bwd_pair_kernel.*?Used (\d+) registers", r.stderr, re.S).group(1))
    text = open(src).read()
    value = {k: int(v) for k, v in re.findall(r"(kRegs\w+) = (\d+)", text)}
    groups = int(re.search(r"kGroups = (\d+)", text).group(1))
    assert used == value["kRegsLaunch"]
    assert 128 * (value["kRegsMisc"] + groups * value["kRegsSoftmax"] + 2 * value["kRegsDrain"]) <= (384 + 128 * groups) * used
