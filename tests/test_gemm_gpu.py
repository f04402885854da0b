"""tcgen05 GEMM against an fp32 PyTorch matmul: all three operand layouts, tails in M / N / K, epilogues."""

import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(128, 256, 64), (256, 512, 128), (300, 384, 200), (1000, 3072, 3072), (77, 128, 1024), (4096, 9216, 256),
          (130, 8, 8), (2048, 264, 72)]


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()


def _mk(shape, g, k=1.0):
    return (torch.randn(*shape, device="cuda", generator=g) * k).bfloat16()


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
def test_layouts(M, N, K, layout):
    from teletron_b200.ops import gemm_tcgen05 as G
    if layout == "tn" and M % 8:
        pytest.skip("tn needs M % 8 == 0")
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    if layout == "nt":
        a, b = _mk((M, K), g), _mk((N, K), g)
        ref = a.float() @ b.float().t()
    elif layout == "nn":
        a, b = _mk((M, K), g), _mk((K, N), g)
        ref = a.float() @ b.float()
    else:
        a, b = _mk((K, M), g), _mk((K, N), g)
        ref = a.float().t() @ b.float()
    assert G.supported(a, b, layout)
    c = G.gemm(a, b, layout)
    G.check_status()
    assert c.shape == (M, N)
    assert _rel(c, ref) < 6e-3, _rel(c, ref)
    # tails must not be written outside the output
    assert torch.isfinite(c).all()


def test_bias_and_gelu_epilogues():
    from teletron_b200.ops import gemm_tcgen05 as G
    g = torch.Generator(device="cuda").manual_seed(0)
    M, N, K = 520, 768, 320
    a, w, bias = _mk((M, K), g), _mk((N, K), g, 0.05), _mk((N,), g)
    u_ref = a.float() @ w.float().t() + bias.float()
    c = G.gemm(a, w, "nt", bias)
    assert _rel(c, u_ref) < 6e-3
    for epi, approx in ((1, "none"), (2, "tanh")):
        y, u = G.gemm(a, w, "nt", bias, epi=epi)
        assert _rel(u, u_ref) < 6e-3
        assert _rel(y, torch.nn.functional.gelu(u_ref, approximate=approx)) < 8e-3
    # dgrad with fused activation backward: (dy @ W) * gelu'(u)
    dy, w2 = _mk((M, 256), g), _mk((256, N), g, 0.05)
    uu = _mk((M, N), g)
    for epi, approx in ((3, "none"), (4, "tanh")):
        got = G.gemm(dy, w2, "nn", epi=epi, aux=uu)
        uf = uu.float().requires_grad_()
        torch.nn.functional.gelu(uf, approximate=approx).backward(dy.float() @ w2.float())
        assert _rel(got, uf.grad) < 8e-3
    G.check_status()


def test_strided_views_and_determinism():
    from teletron_b200.ops import gemm_tcgen05 as G
    g = torch.Generator(device="cuda").manual_seed(1)
    big = _mk((512, 1024), g)
    a = big[:, 256:768]                       # row pitch 1024, 512 columns
    w = _mk((384, 512), g)
    assert G.supported(a, w, "nt")
    c1 = G.gemm(a, w, "nt")
    assert _rel(c1, a.float() @ w.float().t()) < 6e-3
    for _ in range(10):
        assert torch.equal(G.gemm(a, w, "nt"), c1)
    G.check_status()


def test_large_k_weight_gradient_shape():
    from teletron_b200.ops import gemm_tcgen05 as G
    g = torch.Generator(device="cuda").manual_seed(2)
    tokens = 8200
    dy, x = _mk((tokens, 1536), g, 0.1), _mk((tokens, 768), g)
    dw = G.gemm(dy, x, "tn")
    G.check_status()
    assert _rel(dw, dy.float().t() @ x.float()) < 6e-3


@pytest.mark.parametrize("M,N,K,layout", [(300, 264, 192, "nt"), (130, 136, 320, "nn"), (264, 520, 200, "tn")])
def test_output_window_is_the_only_memory_written(M, N, K, layout):
    """The output is a window inside a larger buffer pre-filled with a guard pattern: rows above and below, and the
    columns left and right of the window, must come back untouched (ragged last tiles must not spill)."""
    from teletron_b200.ops import gemm_tcgen05 as G
    g = torch.Generator(device="cuda").manual_seed(M + N)
    if layout == "nt":
        a, b = _mk((M, K), g), _mk((N, K), g)
        ref = a.float() @ b.float().t()
    elif layout == "nn":
        a, b = _mk((M, K), g), _mk((K, N), g)
        ref = a.float() @ b.float()
    else:
        a, b = _mk((K, M), g), _mk((K, N), g)
        ref = a.float().t() @ b.float()
    pad_r, pad_c = 5, 8                                   # the column offset keeps the window 16-byte aligned
    guard = torch.full((M + 2 * pad_r, N + 2 * pad_c), -777.0, device="cuda", dtype=torch.bfloat16)
    window = guard[pad_r:pad_r + M, pad_c:pad_c + N]
    if not G.supported(a, b, layout):
        pytest.skip("shape outside the kernel's gate")
    G.gemm(a, b, layout, out=window)
    G.check_status()
    assert _rel(window, ref) < 8e-3
    mask = torch.ones_like(guard, dtype=torch.bool)
    mask[pad_r:pad_r + M, pad_c:pad_c + N] = False
    assert bool((guard[mask] == -777.0).all())


PAIR_SHAPES = [(256, 256, 64), (2560, 2048, 512), (2313, 2056, 200), (4096, 9216, 256), (1100, 4360, 72)]


@pytest.mark.parametrize("M,N,K", PAIR_SHAPES)
@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
def test_cta_pair_kernel_layouts(M, N, K, layout):
    """The CTA-pair kernel (cluster of 2, tcgen05.mma.cta_group::2, 256 x 256 tiles) on whole tiles and on M / N / K tails,
    forced for every shape, against fp32; two runs give the same bits."""
    from teletron_b200.ops import gemm_tcgen05 as G
    if layout == "tn" and M % 8:
        pytest.skip("tn needs M % 8 == 0")
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    if layout == "nt":
        a, b = _mk((M, K), g), _mk((N, K), g)
        ref = a.float() @ b.float().t()
    elif layout == "nn":
        a, b = _mk((M, K), g), _mk((K, N), g)
        ref = a.float() @ b.float()
    else:
        a, b = _mk((K, M), g), _mk((K, N), g)
        ref = a.float().t() @ b.float()
    old = (G.PAIR_KERNEL, G.PAIR_MIN_TILES)
    G.PAIR_KERNEL, G.PAIR_MIN_TILES = True, 1
    try:
        n0 = G.COUNTERS["pair"]
        c = torch.full((M + 2, N), float("nan"), device="cuda", dtype=torch.bfloat16)       # rows beyond M must stay untouched
        G.gemm(a, b, layout, out=c[:M])
        c2 = G.gemm(a, b, layout)
        G.check_status()
        assert G.COUNTERS["pair"] == n0 + 2
    finally:
        G.PAIR_KERNEL, G.PAIR_MIN_TILES = old
    assert torch.isnan(c[M:].float()).all()
    assert torch.isfinite(c[:M].float()).all()
    assert _rel(c[:M], ref) < 6e-3, _rel(c[:M], ref)
    assert torch.equal(c[:M], c2)


def test_cta_pair_kernel_epilogues():
    from teletron_b200.ops import gemm_tcgen05 as G
    g = torch.Generator(device="cuda").manual_seed(3)
    M, N, K = 1032, 1544, 320
    a, w, bias = _mk((M, K), g), _mk((N, K), g, 0.05), _mk((N,), g)
    u_ref = a.float() @ w.float().t() + bias.float()
    old = (G.PAIR_KERNEL, G.PAIR_MIN_TILES)
    G.PAIR_KERNEL, G.PAIR_MIN_TILES = True, 1
    try:
        assert _rel(G.gemm(a, w, "nt", bias), u_ref) < 6e-3
        for epi, approx in ((1, "none"), (2, "tanh")):
            y, u = G.gemm(a, w, "nt", bias, epi=epi)
            assert _rel(u, u_ref) < 6e-3
            assert _rel(y, torch.nn.functional.gelu(u_ref, approximate=approx)) < 8e-3
        dy, w2 = _mk((M, 256), g), _mk((256, N), g, 0.05)
        uu = _mk((M, N), g)
        for epi, approx in ((3, "none"), (4, "tanh")):
            got = G.gemm(dy, w2, "nn", epi=epi, aux=uu)
            uf = uu.float().requires_grad_()
            torch.nn.functional.gelu(uf, approximate=approx).backward(dy.float() @ w2.float())
            assert _rel(got, uf.grad) < 8e-3
        G.check_status()
    finally:
        G.PAIR_KERNEL, G.PAIR_MIN_TILES = old


@pytest.mark.parametrize("M,N,K,splits", [(33, 72, 512, 2), (256, 264, 4104, 6), (130, 520, 1032, 5), (520, 136, 2056, 16), (8, 8, 264, 2),
                                            (2504, 520, 1032, 5)])
@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
def test_split_k(M, N, K, splits, layout, monkeypatch):
    """Ragged rows, columns and k-blocks (a last range shorter than the others, ranges that would be empty), every epilogue
    the layout has, an output window, and the same bits twice.  The last size has more (tile, range) units than CTA pairs
    and an odd number of boxes in some, so that the staging boxes alternate from one unit to the next."""
    from teletron_b200.ops import gemm_tcgen05 as G
    if layout == "tn" and M % 8:
        pytest.skip("tn needs M % 8 == 0")
    monkeypatch.setattr(G, "_plan", lambda *a: (True, splits))
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = _mk((K, M) if layout == "tn" else (M, K), g)
    b = _mk((N, K) if layout == "nt" else (K, N), g, 0.05)
    ref = (a.double().t() if layout == "tn" else a.double()) @ (b.double().t() if layout == "nt" else b.double())
    before = G.COUNTERS["split"]
    guard = torch.full((M + 2, N + 16), -777.0, device="cuda", dtype=torch.bfloat16)
    c = G.gemm(a, b, layout, out=guard[1:M + 1, 8:N + 8])
    assert G.COUNTERS["split"] == before + 1
    for r0 in range(0, M, 32):                   # one bf16 rounding (2^-9 relative, 1.7e-3 in norm) and fp32 sums
        assert _rel(c[r0:r0 + 32], ref[r0:r0 + 32]) < 3e-3
    guard[1:M + 1, 8:N + 8] = -777.0
    assert bool((guard == -777.0).all())
    assert torch.equal(G.gemm(a, b, layout), G.gemm(a, b, layout))
    if layout == "nt":
        bias = _mk((N,), g)
        assert _rel(G.gemm(a, b, "nt", bias), ref + bias.double()) < 3e-3
        for epi, approx in ((1, "none"), (2, "tanh")):
            y, u = G.gemm(a, b, "nt", bias, epi=epi)
            assert _rel(u, ref + bias.double()) < 3e-3
            assert _rel(y, torch.nn.functional.gelu(ref + bias.double(), approximate=approx)) < 4e-3
    elif layout == "nn":
        aux = _mk((M, N), g)
        for epi, approx in ((3, "none"), (4, "tanh")):
            ud = aux.double().requires_grad_()
            torch.nn.functional.gelu(ud, approximate=approx).backward(ref)
            assert _rel(G.gemm(a, b, "nn", epi=epi, aux=aux), ud.grad) < 4e-3
    G.check_status()


@pytest.mark.parametrize("M,k1,k2,N,splits", [(300, 64, 72, 264, 1), (1031, 384, 1536, 768, 1), (8, 128, 64, 8, 1), (257, 320, 2040, 136, 4)])
def test_two_operands_side_by_side(M, k1, k2, N, splits, monkeypatch):
    """``[a | a2] @ b.T`` from two tensors (one of them a strided view): the seam inside a split's range, ragged ends, with
    the same k order as the concatenated product and therefore the same bits when that takes the same kernel."""
    from teletron_b200.ops import gemm_tcgen05 as G
    monkeypatch.setattr(G, "_plan", lambda *a: (True, splits))
    g = torch.Generator(device="cuda").manual_seed(M)
    a, wide, b, bias = _mk((M, k1), g), _mk((M, k2 + 16), g), _mk((N, k1 + k2), g, 0.05), _mk((N,), g)
    a2 = wide[:, 8:8 + k2]
    assert G.two_supported(a, a2, b)
    c = G.gemm_two(a, a2, b, bias)
    cat = torch.cat([a, a2], dim=1)
    assert _rel(c, cat.double() @ b.double().t() + bias.double()) < 3e-3
    assert torch.equal(c, G.gemm(cat, b, "nt", bias))
    assert not G.two_supported(a[:, :k1 - 8], a2, b[:, 8:])
    G.check_status()


@pytest.mark.parametrize("M,N,K,pair", [(40005, 64, 64, False), (40005, 72, 72, False), (30005, 320, 64, True), (20013, 264, 64, True)])
def test_epilogue_boxes_over_many_tiles(M, N, K, pair, monkeypatch):
    """Short products with an odd number of 64-column boxes in some tiles, several tiles a CTA: the two staging boxes of a
    warp alternate over tile boundaries.  With a pre-activation beside the output a tile's count of boxes is even."""
    from teletron_b200.ops import gemm_tcgen05 as G
    monkeypatch.setattr(G, "use_pair_kernel", lambda *a: pair)
    monkeypatch.setattr(G, "_plan", lambda *a: (pair, 1))
    g = torch.Generator(device="cuda").manual_seed(N)
    a, w, bias = _mk((M, K), g), _mk((N, K), g, 0.05), _mk((N,), g)
    ref = a.float() @ w.float().t() + bias.float()
    for _ in range(3):
        assert _rel(G.gemm(a, w, "nt", bias), ref) < 3e-3
        y, u = G.gemm(a, w, "nt", bias, epi=1)
        assert _rel(u, ref) < 3e-3 and _rel(y, torch.nn.functional.gelu(ref)) < 4e-3
    G.check_status()


@pytest.mark.parametrize("M,N,K,kind", [(256, 9216, 3072, "single"), (40, 3072, 3072, "single"), (256, 12288, 3072, "pair"),
                                        (250, 3072, 12288, "split"), (1024, 3072, 12288, "split")])
def test_small_products_as_planned(M, N, K, kind):
    """The kernel that the rule picks for the size, for one product and for two operands side by side."""
    from teletron_b200.ops import gemm_tcgen05 as G
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, b, bias = _mk((M, K), g), _mk((N, K), g, 0.05), _mk((N,), g)
    ref = a.float() @ b.float().t() + bias.float()
    before = dict(G.COUNTERS)
    c = G.gemm(a, b, "nt", bias)
    assert {k: v - before[k] for k, v in G.COUNTERS.items() if v != before[k]} == {kind: 1}
    before = dict(G.COUNTERS)
    c2 = G.gemm_two(a[:, :1024], a[:, 1024:], b, bias)
    assert {k: v - before[k] for k, v in G.COUNTERS.items() if v != before[k]} == {"split" if kind == "split" else "pair": 1}
    for r0 in range(0, M, 32):
        assert _rel(c[r0:r0 + 32], ref[r0:r0 + 32]) < 3e-3 and _rel(c2[r0:r0 + 32], ref[r0:r0 + 32]) < 3e-3
    G.check_status()


@pytest.mark.parametrize("K,M,N", [(1, 512, 3072), (7, 264, 520), (64, 256, 256), (250, 3072, 1024), (1000, 8, 4096), (333, 4096, 2056)])
def test_weight_gradient_added_in_the_epilogue(K, M, N):
    """``out += a.T @ b`` rounds the product to bf16 and adds with one more rounding: the bits of a separate addition of this kernel's
    product (which added to zeros gives that).  Any row count; columns beside the window stay as they are."""
    from teletron_b200.ops import gemm
    from teletron_b200.ops.gemm_tcgen05 import add_supported, check_status
    g = torch.Generator(device="cuda").manual_seed(K)
    a, b = (torch.randn(K, n, device="cuda", generator=g).bfloat16() for n in (M, N))
    whole = torch.randn(M, N + 64, device="cuda", generator=g).bfloat16()
    before, out = whole.clone(), whole[:, 8:8 + N]
    assert add_supported(a, b, out) and gemm.gemm_tn_add(a, b, out)
    check_status()
    ref = before[:, 8:8 + N].double() + (a.double().t() @ b.double()).bfloat16().double()
    assert (out.double() - ref).abs().max() <= 2 ** -7 * ref.abs().max()
    assert (out.double() - ref).norm() < 4e-3 * ref.norm()          # 2^-9 per rounding
    assert torch.equal(whole[:, :8], before[:, :8]) and torch.equal(whole[:, 8 + N:], before[:, 8 + N:])
    product = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
    assert gemm.gemm_tn_add(a, b, product)
    assert torch.equal(out, before[:, 8:8 + N] + product)


def test_flat_gradient_buffers_receive_products_only_where_autograd_accumulates():
    """Parameters in a flat buffer: ``backward`` adds each weight gradient exactly once per pass (four products: the merged projection has
    two halves); ``autograd.grad``, hooks on the parameter or on its node, and a side stream see gradients as before."""
    from teletron_b200 import ops
    from teletron_b200.ops.gemm_tcgen05 import COUNTERS
    from teletron_b200.parallel.grad_buffer import DistributedDataParallel

    def additions(f):
        n0 = COUNTERS["add"]
        f()
        return COUNTERS["add"] - n0

    class Net(torch.nn.Module):
        def __init__(self):
            super().__init__()
            g = torch.Generator(device="cuda").manual_seed(3)
            mk = lambda *s: torch.nn.Parameter((torch.randn(*s, device="cuda", generator=g) * 0.05).bfloat16())  # noqa: E731
            self.w1, self.b1, self.w2, self.w3 = mk(1024, 256), mk(1024), mk(256, 1024), mk(256, 512)

        def forward(self, x):
            h = ops.linear(ops.linear(x, self.w1, self.b1, "gelu"), self.w2)
            return ops.linear_merged(h, x, self.w3)

    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(1, 37, 256, device="cuda", generator=g).bfloat16()
    dy = torch.randn(1, 37, 256, device="cuda", generator=g).bfloat16()
    plain, net = Net(), Net()
    ddp = DistributedDataParallel(net, None)
    names = ("w1", "b1", "w2", "w3")
    for _ in range(2):                                       # two micro-batches
        plain(x).backward(dy)
        assert additions(lambda: ddp(x).backward(dy)) == 4
    for n in names:
        torch.testing.assert_close(getattr(net, n).grad, getattr(plain, n).grad, rtol=1.6e-2, atol=1e-2)
    kept = {n: getattr(net, n).grad.clone() for n in names}
    n0 = COUNTERS["add"]
    got = torch.autograd.grad(net(x), [net.w1, net.w2, net.w3], dy)
    assert COUNTERS["add"] == n0
    want = torch.autograd.grad(plain(x), [plain.w1, plain.w2, plain.w3], dy)
    for a, b in zip(got, want):
        torch.testing.assert_close(a, b, rtol=1.6e-2, atol=1e-2)
    assert all(torch.equal(getattr(net, n).grad, kept[n]) for n in names)          # collected, not accumulated
    seen = []
    h1 = net.w1.register_hook(lambda t: seen.append("w1"))
    h2 = net.w2.register_post_accumulate_grad_hook(lambda p: seen.append("w2"))
    assert additions(lambda: net(x).backward(dy)) == 2          # w3's
    assert sorted(seen) == ["w1", "w2"]
    h1.remove()
    h2.remove()
    node = net.w3.expand_as(net.w3).grad_fn.next_functions[0][0]
    h3 = node.register_hook(lambda _, g: seen.append(g[0].shape))
    assert additions(lambda: net(x).backward(dy)) == 2          # w1's and w2's
    assert seen[2:] == [net.w3.shape]
    h3.remove()
    del node
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        assert additions(lambda: net(x).backward(dy)) == 0
    torch.cuda.current_stream().wait_stream(side)
    assert additions(lambda: net(x).backward(dy, inputs=[net.b1])) == 0
    assert additions(lambda: net(x).backward(dy, inputs=[net.w2])) == 1
    for _ in range(3):
        plain(x).backward(dy)
    plain(x).backward(dy, inputs=[plain.w2])
    for n in ("w1", "w2", "w3"):
        torch.testing.assert_close(getattr(net, n).grad, getattr(plain, n).grad, rtol=1.6e-2, atol=2e-2)


def test_flat_gradient_buffers_of_the_two_stream_projection():
    """One autograd node with two weights: both products are added, each to its own buffer, in any row count."""
    from teletron_b200 import ops
    from teletron_b200.ops.gemm_tcgen05 import COUNTERS, check_status
    from teletron_b200.parallel.grad_buffer import DistributedDataParallel
    heads, S, T = 2, 45, 11
    H = heads * 128

    class Net(torch.nn.Module):
        def __init__(self):
            super().__init__()
            g = torch.Generator(device="cuda").manual_seed(13)
            for i in (1, 2):
                for n, shape, k in (("w", (3 * H, H), 0.05), ("b", (3 * H,), 0.1), ("qw", (128,), 0.2), ("kw", (128,), 0.2)):
                    setattr(self, f"{n}{i}", torch.nn.Parameter(_mk(shape, g, k)))

        def forward(self, x, y):
            return ops.joint_qkv_projection(x, self.w1, self.b1, self.qw1, self.kw1, cos, sin, y, self.w2, self.b2, self.qw2, self.kw2, heads)

    g = torch.Generator(device="cuda").manual_seed(14)
    x, y = _mk((1, S, H), g), _mk((1, T, H), g)
    ang = torch.rand(S, 64, device="cuda", generator=g) * 6.28
    cos, sin = ang.cos().repeat_interleave(2, 1), ang.sin().repeat_interleave(2, 1)
    d = [_mk((1, heads, S + T, 128), g) for _ in range(3)]
    plain, net = Net(), Net()
    ddp = DistributedDataParallel(net, None)
    for _ in range(2):
        torch.autograd.backward(plain(x, y), d)
        n0 = COUNTERS["add"]
        torch.autograd.backward(ddp(x, y), d)
        assert COUNTERS["add"] == n0 + 2
    check_status()
    for (n, a), (_, b) in zip(net.named_parameters(), plain.named_parameters()):
        assert _rel(a.grad, b.grad) < 4e-3, n


def test_flat_gradient_added_before_an_accumulation_node_of_another_stream_runs():
    """The node was created under a side stream, which is all that the caller of ``backward`` waits for: the product that the default
    stream adds meanwhile has to come before it."""
    from teletron_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(7)
    x, dy = (torch.randn(64, 256, device="cuda", generator=g).bfloat16() for _ in range(2))
    w = torch.nn.Parameter(torch.zeros(256, 256, device="cuda", dtype=torch.bfloat16))
    w.grad = torch.zeros_like(w)
    w.flat_grad = True
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        node = w.expand_as(w).grad_fn.next_functions[0][0]
    ops.linear(x, w).backward(dy)
    torch.cuda.synchronize()
    want = w.grad.clone()
    w.grad.zero_()
    y = ops.linear(x, w)
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)              # the product waits behind this, ~50 ms
    with torch.cuda.stream(side):
        y.backward(dy)
        got = w.grad.clone()
    torch.cuda.synchronize()
    assert torch.equal(got, want) and want.any()
    assert node.variable is w
