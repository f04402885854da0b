"""Python side of the tcgen05 GEMM (``csrc/gemm_tcgen05.cu``).

``gemm(a, b, layout, bias, epi, aux)`` computes ``C[M, N]`` in bf16 with fp32 accumulation:

* layout ``"nt"``: ``a [M, K] @ b [N, K]^T``;  ``"nn"``: ``a [M, K] @ b [K, N]``;  ``"tn"``: ``a [K, M]^T @ b [K, N]``.
* ``epi`` 0: ``+ bias``; 1 / 2: ``gelu_erf / gelu_tanh(acc + bias)`` with the pre-activation written to a
  second output; 3 / 4: ``acc * gelu'(aux)`` (activation backward fused into a data-gradient product).

The kernel's waits are bounded; if one runs out it records a status word that :func:`check_status` turns
into :class:`teletron_b200.ops._lib.CommTimeoutError` (the CUDA context stays usable).
"""

from __future__ import annotations

import functools
import os
from typing import Dict, Optional, Tuple

import torch

from . import _lib
from ._lib import call

BF16 = torch.bfloat16
_LAYOUTS = {"nt": (0, 0), "nn": (0, 1), "tn": (1, 1)}
# CTA-pair kernel (thread-block cluster of 2, 256 x 256 tiles) for products with at least one tile per pair of SMs;
# TELETRON_B200_GEMM_2CTA=0 keeps everything on the single-CTA kernel
PAIR_KERNEL = os.environ.get("TELETRON_B200_GEMM_2CTA", "1") != "0"
PAIR_MIN_TILES = 74
COUNTERS = {"pair": 0, "single": 0, "split": 0, "add": 0}       # "add": those of "pair" that added to their output
# What a split product takes the host to issue: a scratch allocation and a second launch on top of the 12.4 us of the others.
SPLIT_ISSUE_US = 17.5


def use_pair_kernel(M: int, N: int) -> bool:
    return PAIR_KERNEL and ((M + 255) // 256) * ((N + 255) // 256) >= PAIR_MIN_TILES


@functools.lru_cache(maxsize=4096)
def _plan(M: int, N: int, K: int) -> Tuple[bool, int]:
    """``(pair, splits)`` for a product with fewer than PAIR_MIN_TILES 256 x 256 tiles.

    Costs in microseconds as measured over M = 40 .. 1280, N = 3072 .. 12288, K = 3072 .. 15360 with weights from HBM: a
    64-wide k-block of a wave of 128 x 128 tiles (148 of them, one an SM) takes 0.22 us, 0.26 when waves follow one another
    (32 KB through L2 per SM set the pace); a wave of 74 pair tiles takes 0.30 (four times the tile on twice the SMs: the
    tensor core does); a split product adds a second launch and one write and read of its fp32 slices.  Examples, single /
    pair / best split: 256 x 3072 x 12288 45.7 / 62.2 / 25.5 (6 splits); 256 x 12288 x 3072 28.1 / 23.0 / 29.0;
    256 x 9216 x 3072 17.4 / 22.0 / 21.6; 1024 x 3072 x 12288 85.8 / 67.8 / 61.1 (3); 512 x 3072 x 4096 18.8 / 25.9 / 18.8.  cuBLAS
    takes 21.8, 18.9, 14.7, 55.3 and 13.1 for these, and 8.0 where the best here is 14.0 (256 x 3072 x 3072).

    A product that is through before a split one could be issued is not split: 40 x 3072 x 3072 would take 11.6 us instead of
    12.6, but calls in a row one every 17.5 us instead of every 12.6."""
    kb, t1, t2 = (K + 63) // 64, ((M + 127) // 128) * ((N + 127) // 128), ((M + 255) // 256) * ((N + 255) // 256)
    waves = (t1 + 147) // 148
    best = (4 + waves * kb * (0.22 if waves == 1 else 0.26), False, 1)
    for s in range(1, min(16, kb // 4) + 1):
        if s == 2 and best[0] < SPLIT_ISSUE_US:
            break
        cost = 5 + ((t2 * s + 73) // 74) * ((kb + s - 1) // s) * 0.30
        if s > 1:
            cost += 5 + 0.13e-6 * (s * ((M + 31) // 32 * 32) * N * 8)
        if cost < best[0]:
            best = (cost, True, s)
    return best[1:]


_STATUS: Dict[torch.device, torch.Tensor] = {}


def status_tensor(device: torch.device) -> torch.Tensor:
    t = _STATUS.get(device)
    if t is None:
        t = _STATUS[device] = torch.zeros(4, dtype=torch.int32, device=device)
    return t


def check_status(device: Optional[torch.device] = None) -> None:
    """Synchronise and raise if any GEMM / attention launch on ``device`` abandoned a bounded wait."""
    for dev, t in _STATUS.items():
        if device is not None and dev != device:
            continue
        code = int(t[0].item())
        if code:
            t.zero_()
            raise _lib.CommTimeoutError(f"a tcgen05 kernel on {dev} gave up a bounded wait (status {code})")


def _rowmajor(t: torch.Tensor) -> bool:
    if t.dim() != 2:
        return False
    s0, s1 = t.stride()
    return s1 == 1 and s0 >= t.shape[1] and s0 % 8 == 0 and t.data_ptr() % 16 == 0


def _dims(a: torch.Tensor, b: torch.Tensor, layout: str) -> Tuple[int, int, int]:
    if layout == "nt":
        (M, K), (N, K2) = a.shape, b.shape
    elif layout == "nn":
        (M, K), (K2, N) = a.shape, b.shape
    else:
        (K, M), (K2, N) = a.shape, b.shape
    if K != K2:
        raise ValueError(f"contraction mismatch for {layout}: {tuple(a.shape)} x {tuple(b.shape)}")
    return M, N, K


def supported(a: torch.Tensor, b: torch.Tensor, layout: str) -> bool:
    if not (_lib.available() and a.is_cuda and a.dtype == BF16 and b.dtype == BF16 and _rowmajor(a) and _rowmajor(b)):
        return False
    M, N, K = _dims(a, b, layout)
    if N % 8 or K % 8 or (layout == "tn" and M % 8):
        return False
    return M >= 1 and N >= 8 and K >= 8


def gemm(a: torch.Tensor, b: torch.Tensor, layout: str, bias: Optional[torch.Tensor] = None, epi: int = 0,
         aux: Optional[torch.Tensor] = None, out: Optional[torch.Tensor] = None):
    """Returns ``C`` (and the pre-activation tensor for ``epi`` 1 / 2)."""
    M, N, K = _dims(a, b, layout)
    a_mn, b_mn = _LAYOUTS[layout]
    dev = a.device
    c = out if out is not None else torch.empty(M, N, dtype=BF16, device=dev)
    if epi and c.stride(0) != N and M > 1:      # the kernels walk the pre-activation with the pitch of C
        raise _lib.NativeError("an epilogue with a pre-activation needs a contiguous output")
    if epi in (1, 2):
        aux = torch.empty(M, N, dtype=BF16, device=dev)
    elif epi in (3, 4):
        if aux is None or aux.shape != (M, N) or not aux.is_contiguous():
            raise _lib.NativeError("epilogue 3/4 needs a contiguous [M, N] pre-activation tensor")
    if bias is not None:
        bias = _lib.check(bias.contiguous(), BF16, "bias")
    pair, splits = use_pair_kernel(M, N), 1
    if PAIR_KERNEL and not pair:
        pair, splits = _plan(M, N, K)
    args = (a.data_ptr(), b.data_ptr(), c.data_ptr(), None if bias is None else bias.data_ptr(), None if aux is None else aux.data_ptr(),
            M, N, K, a.stride(0), b.stride(0), c.stride(0), a_mn, b_mn, epi)
    if splits > 1:
        COUNTERS["split"] += 1
        scratch = torch.empty(splits * ((M + 31) // 32 * 32) * N, dtype=torch.float32, device=dev)
        call("tt_gemm2_bf16_splitk", *args, splits, scratch.data_ptr(), status_tensor(dev).data_ptr(), _lib.raw_stream())
    else:
        COUNTERS["pair" if pair else "single"] += 1
        call("tt_gemm2_bf16" if pair else "tt_gemm_bf16", *args, status_tensor(dev).data_ptr(), _lib.raw_stream())
    return (c, aux) if epi in (1, 2) else c


def add_supported(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor) -> bool:
    """``out += a.T @ b`` in the product's epilogue: any row count, and no split over K (a split product has a pass of its own that
    could add, but a gradient with so few tiles is small)."""
    if not (PAIR_KERNEL and _lib.available() and a.is_cuda and a.dtype == BF16 and b.dtype == BF16 and out.dtype == BF16 and _rowmajor(a)
            and _rowmajor(b) and _rowmajor(out)):
        return False
    (K, M), (K2, N) = a.shape, b.shape
    return (K == K2 >= 1 and tuple(out.shape) == (M, N) and M % 8 == 0 and N % 8 == 0 and min(M, N) >= 8
            and (use_pair_kernel(M, N) or _plan(M, N, K)[1] == 1))


def gemm_add(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor) -> None:
    """``out += a.T @ b``: the product is rounded to bf16, then added with one more rounding, as a separate addition would."""
    (K, M), N = a.shape, b.shape[1]
    COUNTERS["pair"] += 1
    COUNTERS["add"] += 1
    call("tt_gemm2_bf16", a.data_ptr(), b.data_ptr(), out.data_ptr(), None, None, M, N, K, a.stride(0), b.stride(0), out.stride(0), 1, 1, 5,
         status_tensor(a.device).data_ptr(), _lib.raw_stream())


def two_supported(a: torch.Tensor, a2: torch.Tensor, b: torch.Tensor) -> bool:
    """``[a | a2] @ b.T`` without the concatenation: the seam has to lie between two 64-wide k-blocks."""
    return (PAIR_KERNEL and a2.dtype == BF16 and a2.is_cuda and _rowmajor(a2) and a.dim() == 2 and a.shape[0] == a2.shape[0]
            and a.shape[1] % 64 == 0 and a2.shape[1] % 8 == 0 and a2.shape[1] > 0 and a.shape[1] + a2.shape[1] == b.shape[1]
            and supported(a, b[:, :a.shape[1]], "nt"))


def gemm_two(a: torch.Tensor, a2: torch.Tensor, b: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Always on the CTA-pair kernel: what the single-CTA kernel gains on a short product is less than the concatenation costs."""
    (M, k1), N, K = a.shape, b.shape[0], b.shape[1]
    c = torch.empty(M, N, dtype=BF16, device=a.device)
    if bias is not None:
        bias = _lib.check(bias.contiguous(), BF16, "bias")
    splits = 1 if use_pair_kernel(M, N) else _plan(M, N, K)[1]
    COUNTERS["pair" if splits == 1 else "split"] += 1
    scratch = None if splits == 1 else torch.empty(splits * ((M + 31) // 32 * 32) * N, dtype=torch.float32, device=a.device)
    call("tt_gemm2_bf16_two", a.data_ptr(), a2.data_ptr(), b.data_ptr(), c.data_ptr(), None if bias is None else bias.data_ptr(), M, N, K, k1,
         a.stride(0), a2.stride(0), b.stride(0), c.stride(0), splits, None if scratch is None else scratch.data_ptr(),
         status_tensor(a.device).data_ptr(), _lib.raw_stream())
    _lib.LAUNCHES += splits > 1      # the pass over the slices
    return c
