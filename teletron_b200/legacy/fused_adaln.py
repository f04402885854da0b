"""``fused_adaln`` with the reference's entry points (``teletron_op/fused_adaln/adaln_ops.cpp:52-65``), served by the
sm_100a LayerNorm + modulation kernels.  Unlike the reference's binding (``adaln_ops.cpp:6-50``) every argument is
checked for dtype, device, contiguity and shape, any column count that is a multiple of 8 is accepted, and launches go
to the caller's current stream.

``torch_launch_adaln_forward(out, x, scale, shift, x_norm, invvar, rows, cols, eps)`` writes
``out = LN(x) * (1 + scale) + shift``, ``x_norm = LN(x)`` and ``invvar = rstd``;
``torch_launch_adaln_backward(dx, dscale, dshift, dout, x_norm, scale, invvar, rows, cols)`` consumes them."""

import torch

from ..ops import _lib
from ..ops._lib import c_float, c_int, c_long, call, check, ptr, stream

BF16 = torch.bfloat16


def torch_launch_adaln_forward(out, x, scale, shift, x_norm, invvar, rows: int, cols: int, eps: float = 1e-6):
    for t, n in ((out, "out"), (x, "x"), (scale, "scale"), (shift, "shift"), (x_norm, "x_norm")):
        check(t, BF16, n)
    check(invvar, torch.float32, "invvar")
    if x.numel() != rows * cols or scale.numel() != cols or shift.numel() != cols or x_norm.numel() != rows * cols:
        raise _lib.NativeError("shape mismatch")
    _check_rows(invvar, rows, cols, out)
    call("tt_adaln_fwd", ptr(x), ptr(scale), ptr(shift), ptr(out), ptr(x_norm), ptr(invvar), c_long(rows), c_int(cols), c_float(eps),
         stream())


def _check_rows(invvar, rows, cols, *full):
    """One statistic per row, and whole [rows, cols] buffers behind every pointer the kernels walk."""
    if invvar.numel() != rows or (invvar.dim() != 1 and rows != 1):
        raise _lib.NativeError("invvar: expected one value per row")
    if any(t.numel() < rows * cols for t in full):
        raise _lib.NativeError("shape mismatch")


def torch_launch_adaln_backward(dx, dscale, dshift, dout, x_norm, scale, invvar, rows: int, cols: int):
    for t, n in ((dx, "dx"), (dscale, "dscale"), (dshift, "dshift"), (dout, "dout"), (x_norm, "x_norm"), (scale, "scale")):
        check(t, BF16, n)
    check(invvar, torch.float32, "invvar")
    if dx.numel() != rows * cols or min(scale.numel(), dscale.numel(), dshift.numel()) < cols:
        raise _lib.NativeError("shape mismatch")
    if invvar.shape == (1,) and rows > 1:
        invvar = invvar.repeat(rows)        # one statistic for all rows
    _check_rows(invvar, rows, cols, dout, x_norm)
    nblk = _lib.lib().tt_norm_partial_blocks(c_long(rows), c_int(1))
    partials = torch.empty(nblk * 2 * cols, dtype=torch.float32, device=dx.device)
    call("tt_adaln_bwd", ptr(dout), ptr(x_norm), ptr(scale), ptr(invvar), ptr(dx), ptr(partials), ptr(dscale), ptr(dshift),
         c_long(rows), c_int(cols), stream())
