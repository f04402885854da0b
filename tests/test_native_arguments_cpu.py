"""What the C entries refuse before they touch a device.  The pointers are made up, so nothing here runs where there is one."""

import pytest
import torch

from teletron_b200.ops import _lib
from teletron_b200.ops._lib import c_float, c_int, c_size

pytestmark = pytest.mark.skipif(torch.cuda.is_available() or not _lib.available(), reason="needs the library and no device")

ARG, BASE = 1, 1 << 20


def _attn_bwd(out=BASE, lse=BASE, dq=BASE, pitch=192, work=None, S=130, route=0):
    p = _lib.ctypes.c_void_p
    floats = 2 * 256 * 130 if work is None else work
    return _lib.lib().tt_attn_bwd_fused(p(BASE), p(BASE), p(BASE), p(out), p(BASE), p(lse), p(BASE), c_size(floats), p(dq), p(BASE), p(BASE),
                                        c_int(1), c_int(2), c_int(S), c_int(S), c_int(0), c_int(0), c_int(pitch), c_float(0.1), c_int(route), p(BASE), p(0))


def test_attention_backward_takes_and_refuses_what_it_did():
    """Statistics in rows of a multiple of 64, 16-byte aligned; the forward's output is read in 8-byte pieces."""
    assert _attn_bwd() != ARG and _attn_bwd(out=BASE + 8) != ARG
    assert _attn_bwd(pitch=130) == ARG and _attn_bwd(pitch=128) == ARG and _attn_bwd(lse=BASE + 4) == ARG
    assert _attn_bwd(out=BASE + 4) == ARG and _attn_bwd(dq=BASE + 8) == ARG and _attn_bwd(work=2 * 256 * 130 - 1) == ARG
    assert _attn_bwd(route=3) == ARG and _attn_bwd(route=-1) == ARG


def _gemm2(K, epi, entry="tt_gemm2_bf16"):
    lib = _lib.lib()
    if entry == "tt_gemm2_bf16_splitk":
        return lib.tt_gemm2_bf16_splitk(BASE, BASE, BASE, 0, 0, 256, 256, K, 256, 256, 256, 1, 1, epi, 2, BASE, BASE, 0)
    return lib.tt_gemm2_bf16(BASE, BASE, BASE, 0, 0, 256, 256, K, 256, 256, 256, 1, 1, epi, BASE, 0)


def test_only_the_adding_epilogue_takes_any_row_count():
    assert _gemm2(128, 0) != ARG and _gemm2(128, 0, "tt_gemm2_bf16_splitk") != ARG
    assert _gemm2(7, 5) != ARG and _gemm2(129, 5) != ARG
    assert _gemm2(7, 0) == ARG and _gemm2(129, 0) == ARG and _gemm2(129, 0, "tt_gemm2_bf16_splitk") == ARG


@pytest.mark.parametrize("heads,S,pairs", [
    (1, 128, False), (24, 256, False), (1, 257, True), (2, 384, True), (3, 1237, True), (48, 1237, True), (24, 32656, True), (3, 119056, True),
    (150, 257, False), (48, 1152, False), (768, 512, True), (160, 33, False), (4, 129, False)])
def test_backward_kernel_by_measured_costs(heads, S, pairs):
    """On 148 SMs: pairs but for one or two key tiles, odd tiles over many heads, and a wave that only a pair would start."""
    from teletron_b200.ops.attn_bwd_tcgen05 import uses_pairs
    assert uses_pairs(heads, S) is pairs
