"""tcgen05 flash attention against an fp32 PyTorch softmax attention."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["fused", "split"])
def bwd_variant(request):
    """Run a backward test on the one-pass kernel (dQ by fp32 reductions) and on the deterministic two-kernel split."""
    from teletron_b200.ops import attn_bwd_tcgen05 as AB
    was = AB.set_fused(request.param == "fused")
    before = dict(AB.COUNTERS)
    yield request.param
    assert AB.COUNTERS[request.param] > before[request.param]
    AB.set_fused(was)


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()


def _ref(q, k, v, kv_len=None, scale=None):
    qf, kf, vf = q.float(), k.float(), v.float()
    s = qf @ kf.transpose(-1, -2) * (scale or 1.0 / math.sqrt(q.shape[-1]))
    if kv_len is not None:
        s[..., kv_len:] = float("-inf")
    p = s.softmax(-1)
    o = p @ vf
    B, H, S, D = q.shape
    return o.transpose(1, 2).reshape(B, S, H * D), torch.logsumexp(s, -1)


@pytest.mark.parametrize("B,H,S,kv_len", [(1, 2, 256, None), (1, 3, 1000, None), (2, 2, 513, None), (1, 2, 900, 777),
                                          (1, 1, 128, None), (1, 2, 3000, None), (1, 1, 200, 130)])
def test_forward(B, H, S, kv_len):
    from teletron_b200.ops import attn_tcgen05 as A
    from teletron_b200.ops.gemm_tcgen05 import check_status
    g = torch.Generator(device="cuda").manual_seed(S + H)
    q, k, v = ((torch.randn(B, H, S, 128, device="cuda", generator=g) * s).bfloat16() for s in (1.0, 1.0, 1.0))
    out, lse, *_ = A.forward(q, k, v, kv_len, None)
    check_status()
    ro, rl = _ref(q, k, v, kv_len)
    assert _rel(out, ro) < 1.2e-2, _rel(out, ro)
    torch.testing.assert_close(lse[..., :S], rl, rtol=2e-3, atol=2e-3)


def test_forward_large_scores_trigger_rescale():
    """Keys ordered by growing norm so the row maximum keeps rising across KV tiles."""
    from teletron_b200.ops import attn_tcgen05 as A
    from teletron_b200.ops.gemm_tcgen05 import check_status
    g = torch.Generator(device="cuda").manual_seed(0)
    S = 1024
    q = (torch.randn(1, 2, S, 128, device="cuda", generator=g) * 2).bfloat16()
    ramp = torch.linspace(0.2, 6.0, S, device="cuda").view(1, 1, S, 1)
    k = (torch.randn(1, 2, S, 128, device="cuda", generator=g) * ramp).bfloat16()
    v = torch.randn(1, 2, S, 128, device="cuda", generator=g).bfloat16()
    out, lse, *_ = A.forward(q, k, v, None, None)
    check_status()
    ro, rl = _ref(q, k, v)
    assert _rel(out, ro) < 1.5e-2
    torch.testing.assert_close(lse[..., :S], rl, rtol=2e-3, atol=5e-3)


@pytest.mark.parametrize("S,kv_len", [(640, None), (300, 260), (128, None), (1000, None), (2100, 2000), (77, None)])
def test_autograd_matches_reference(S, kv_len, bwd_variant):
    from teletron_b200.ops import attn_tcgen05 as A
    from teletron_b200.ops import reference
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v = (torch.randn(1, 2, S, 128, device="cuda", generator=g).bfloat16().requires_grad_() for _ in range(3))
    d = torch.randn(1, S, 256, device="cuda", generator=g).bfloat16()
    o = A.attention(q, k, v, kv_len, None)
    o.backward(d)
    refs = [t.detach().float().requires_grad_() for t in (q, k, v)]
    ro = reference.attention(*refs, kv_len, None)
    ro.backward(d.float())
    assert _rel(o, ro) < 1.2e-2
    for a, r in zip((q, k, v), refs):
        assert _rel(a.grad, r.grad) < 2e-2


@pytest.mark.parametrize("S,kv_len,mask", [(900, None, (40, 256)), (700, 650, (100, 130)), (640, None, (128, 256)), (400, 390, (3, 5))])
def test_masked_key_range_forward_and_backward(S, kv_len, mask, bwd_variant):
    """Padded text tokens that sit at the head of the sequence: keys in [lo, hi) are masked on top of the key length,
    including a range that covers a whole 128-key tile."""
    from teletron_b200.ops import attn_tcgen05 as A
    from teletron_b200.ops import reference
    from teletron_b200.ops.gemm_tcgen05 import check_status
    g = torch.Generator(device="cuda").manual_seed(7)
    q, k, v = (torch.randn(1, 2, S, 128, device="cuda", generator=g).bfloat16().requires_grad_() for _ in range(3))
    d = torch.randn(1, S, 256, device="cuda", generator=g).bfloat16()
    o = A.attention(q, k, v, kv_len, None, mask)
    o.backward(d)
    check_status()
    refs = [t.detach().float().requires_grad_() for t in (q, k, v)]
    ro = reference.attention(*refs, kv_len, None, mask)
    ro.backward(d.float())
    assert _rel(o, ro) < 1.2e-2
    for a, r in zip((q, k, v), refs):
        assert torch.isfinite(a.grad.float()).all()
        assert _rel(a.grad, r.grad) < 2e-2
    # masked keys receive no gradient at all
    assert float(k.grad[:, :, mask[0]:mask[1]].float().abs().max()) == 0.0
    assert float(v.grad[:, :, mask[0]:mask[1]].float().abs().max()) == 0.0


@pytest.mark.parametrize("S,kv_len,mask", [(256, None, None), (300, None, None), (700, 650, None), (384, None, (0, 128)), (640, 600, (100, 300))])
@pytest.mark.parametrize("scale", [0.0, -0.05, -0.6])
def test_scale_of_zero_and_below(S, kv_len, mask, scale, bwd_variant):
    """Masked keys stay out whatever the scale's sign is: with tiles that are whole, ragged, partly and wholly masked (the
    first one, too), and with scores (-0.6) whose range is beyond what exp2 takes without the running maximum."""
    from teletron_b200 import ops
    from teletron_b200.ops import reference
    from teletron_b200.ops.gemm_tcgen05 import check_status
    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v = (torch.randn(1, 2, S, 128, device="cuda", generator=g).bfloat16().requires_grad_() for _ in range(3))
    d = torch.randn(1, S, 256, device="cuda", generator=g).bfloat16()
    o = ops.attention(q, k, v, kv_len, scale, mask)
    o.backward(d)
    check_status()
    refs = [t.detach().double().requires_grad_() for t in (q, k, v)]
    ro = reference.attention(*refs, kv_len, scale, mask)
    ro.backward(d.double())
    assert _rel(o, ro) < 1.2e-2
    for a, r in zip((q, k, v), refs):
        assert _rel(a.grad, r.grad) < 2e-2


def test_forward_and_backward_are_bitwise_reproducible(bwd_variant):
    """The forward, dK and dV have a fixed accumulation order in both variants; so has dQ in the two-kernel split:
    repeated launches on the same inputs give the same bits (also a cheap detector of ordering races between the
    kernels' warp roles).  The one-pass variant adds the key tiles' dQ contributions in fp32 in no fixed order: there
    dQ repeats to rounding."""
    from teletron_b200.ops import attn_tcgen05 as A
    from teletron_b200.ops.gemm_tcgen05 import check_status
    g = torch.Generator(device="cuda").manual_seed(4)
    S, kv_len = 1500, 1400
    q, k, v = (torch.randn(1, 3, S, 128, device="cuda", generator=g).bfloat16() for _ in range(3))
    d = torch.randn(1, S, 384, device="cuda", generator=g).bfloat16()
    first = None
    for _ in range(5):
        qq, kk, vv = (t.clone().requires_grad_() for t in (q, k, v))
        o = A.attention(qq, kk, vv, kv_len, None)
        o.backward(d)
        res = (o.detach(), qq.grad, kk.grad, vv.grad)
        if first is None:
            first = res
        else:
            for i, (a, b) in enumerate(zip(res, first)):
                if i == 1 and bwd_variant == "fused":
                    assert _rel(a, b) < 2e-3
                else:
                    assert torch.equal(a, b)
    check_status()


@pytest.mark.parametrize("S,kv_len,mask,ramp", [(640, None, (0, 200), 1.0), (900, 777, (0, 256), 6.0), (1100, 1090, (300, 520), 6.0),
                                                (129, None, None, 1.0), (2049, None, None, 8.0)])
def test_forward_running_maximum_with_masked_tiles(S, kv_len, mask, ramp):
    """The first exponentials of a tile use the maximum before it: a first tile without a visible key, maxima that keep
    growing (the redo path) before, inside and after masked tiles, and a last tile of one key."""
    from teletron_b200.ops import attn_tcgen05 as A
    from teletron_b200.ops import reference
    g = torch.Generator(device="cuda").manual_seed(S)
    q = torch.randn(1, 2, S, 128, device="cuda", generator=g).bfloat16()
    k = (torch.randn(1, 2, S, 128, device="cuda", generator=g) * torch.linspace(0.3, ramp, S, device="cuda").view(1, 1, S, 1)).bfloat16()
    v = torch.randn(1, 2, S, 128, device="cuda", generator=g).bfloat16()
    out, lse, *_ = A.forward(q, k, v, kv_len, None, mask)
    ref = reference.attention(q.double(), k.double(), v.double(), kv_len, None, mask)
    assert _rel(out, ref) < 1.2e-2
    s = q.double() @ k.double().transpose(-1, -2) / math.sqrt(128)
    s[..., kv_len or S:] = float("-inf")
    if mask:
        s[..., mask[0]:mask[1]] = float("-inf")
    torch.testing.assert_close(lse[..., :S].double(), s.logsumexp(-1), rtol=1e-4, atol=1e-3)


@pytest.mark.parametrize("route", ["single CTAs", "CTA pairs"])
@pytest.mark.parametrize("B,H,S,kv_len,mask,scale", [
    (1, 1, 257, 200, None, None), (1, 2, 384, None, None, None), (2, 3, 300, None, (20, 90), None), (1, 1, 511, None, None, None),
    (1, 2, 513, 500, None, None), (1, 3, 1237, 1201, (180, 256), None), (1, 1, 2049, None, None, None),      # odd tiles, ragged chunks, masks over a tile's edge
    (1, 1, 129, None, None, None), (3, 50, 257, 250, (100, 130), None), (40, 4, 33, None, None, None),       # few tiles
    (1, 1, 1, None, None, None), (1, 2, 100, 90, (3, 7), None), (2, 1, 128, None, None, None), (1, 1, 256, None, None, None),  # one and two chunks
    (1, 2, 700, 650, (100, 300), -0.05), (1, 1, 300, None, (0, 30), 0.0)])                                  # masked keys outscore visible ones
def test_one_pass_backward_against_64_bits(B, H, S, kv_len, mask, scale, route):
    """Both kernels of the one-pass backward, forced, at the edges of their tiles.  bf16 P and dS (2^-9 each) under fp32 sums leave about
    3e-3; the two-kernel split differs from this by the order of sums only."""
    from teletron_b200.ops import attn_bwd_tcgen05 as AB, attn_tcgen05 as A
    from teletron_b200.ops.gemm_tcgen05 import check_status
    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v = (torch.randn(B, H, S, 128, device="cuda", generator=g).bfloat16() for _ in range(3))
    d = torch.randn(B, S, H * 128, device="cuda", generator=g).bfloat16()
    out, lse, qc, kc, vc, sc, kv = A.forward(q, k, v, kv_len, scale, mask)
    got = AB.backward(d, qc, kc, vc, out, lse, sc, kv, mask_range=mask or (0, 0), route=1 + (route == "CTA pairs"))
    check_status()
    qd, kd, vd = (t.double() for t in (q, k, v))
    dd = d.double().view(B, S, H, 128).transpose(1, 2)
    s = qd @ kd.transpose(-1, -2) * sc
    dead = torch.zeros(S, dtype=torch.bool, device="cuda")
    dead[kv:] = True
    if mask:
        dead[mask[0]:mask[1]] = True
    p = s.masked_fill(dead, float("-inf")).softmax(-1)
    ds = p * (dd @ vd.transpose(-1, -2) - (dd * (p @ vd)).sum(-1, keepdim=True)) * sc
    for a, r in zip(got, (ds @ kd, ds.transpose(-1, -2) @ qd, p.transpose(-1, -2) @ dd)):
        assert torch.isfinite(a).all()
        # one key, or a scale of zero: dQ and dK are zero, but for two fp32 sums of 128 products that should cancel
        assert _rel(a, r) < 5e-3 if r.abs().max() > 1e-9 else a.float().abs().max() < 1e-3


def test_backward_route_by_itself():
    """The call without a route takes the kernel that the rule names: the same bits in dK and dV, whose sums have an order."""
    from teletron_b200.ops import attn_bwd_tcgen05 as AB, attn_tcgen05 as A
    from teletron_b200.ops.gemm_tcgen05 import check_status
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for H, S in ((1, 257), (3, 1237), (150, 257), (4, 129)):
        g = torch.Generator(device="cuda").manual_seed(S)
        q, k, v = (torch.randn(1, H, S, 128, device="cuda", generator=g).bfloat16() for _ in range(3))
        d = torch.randn(1, S, H * 128, device="cuda", generator=g).bfloat16()
        out, lse, *_, sc, kv = A.forward(q, k, v, None, None)
        by_rule, single, pairs = (AB.backward(d, q, k, v, out, lse, sc, kv, route=r) for r in (0, 1, 2))
        for x, y in zip(by_rule[1:], (pairs if AB.uses_pairs(H, S, sms) else single)[1:]):
            assert torch.equal(x, y)
    check_status()


@pytest.mark.parametrize("S,scale", [(1, None), (63, None), (64, None), (129, -0.1), (250, None), (449, None), (1237, None)])
def test_forward_fills_the_padding_of_its_statistics(S, scale):
    """The log-sum-exp rows are S rounded up to 64 long; the forward itself writes +inf behind the last query."""
    from teletron_b200.ops import attn_tcgen05 as A
    from teletron_b200.ops.gemm_tcgen05 import check_status
    pitch = (S + 63) // 64 * 64
    junk = torch.full((2, 3, pitch), -7.0, device="cuda")
    del junk                                        # the allocator hands the same block out again
    q, k, v = (torch.randn(2, 3, S, 128, device="cuda").bfloat16() for _ in range(3))
    lse = A.forward(q, k, v, None, scale)[1]
    check_status()
    assert lse.shape[-1] == pitch and torch.isfinite(lse[..., :S]).all()
    assert (lse[..., S:] == float("inf")).all()
