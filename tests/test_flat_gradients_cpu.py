"""Weight gradients that a product adds to a flat gradient buffer itself: whoever could see a gradient on its way to the buffer still
does.  The product is a stand-in on the CPU; the decision is the one of the kernels' autograd functions."""

import pytest
import torch

from teletron_b200.ops import _lib, cuda_ops, gemm


class _Product(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w):
        ctx.save_for_backward(x, w)
        return x @ w.t()

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        return dy @ w, cuda_ops._weight_grad(ctx, w, dy, x)


@pytest.fixture
def added(monkeypatch):
    """Weights whose gradient a product has added itself, in order."""
    log = []

    def add(a, b, out):
        log.append(tuple(out.shape))
        out.data.add_((a.t() @ b).to(out.dtype))        # through raw pointers: autograd does not see it
        return True
    monkeypatch.setattr(gemm, "gemm_tn_add", add)
    monkeypatch.setattr(_lib, "raw_stream", lambda: 0)
    return log


def _weight(rows=4):
    w = torch.nn.Parameter(torch.randn(rows, 4).bfloat16())
    w.grad = torch.zeros_like(w)
    w.flat_grad = True
    return w


def _node(w):
    return w.expand_as(w).grad_fn.next_functions[0][0]


X = torch.randn(3, 4).bfloat16()


def test_product_is_added_where_nobody_looks(added):
    w = _weight()
    for _ in range(2):
        _Product.apply(X, w).sum().backward()
    assert added == [(4, 4)] * 2
    torch.testing.assert_close(w.grad, (2 * X.sum(0)).expand(4, 4).bfloat16(), rtol=2 ** -7, atol=2 ** -7)


@pytest.mark.parametrize("register", ["register_hook", "register_prehook"])
@pytest.mark.parametrize("held", [True, False])
def test_hooks_on_the_accumulation_node_see_the_gradient(added, register, held):
    """The form that data-parallel wrappers use: a hook on the node that accumulates, which the wrapper keeps alive, or which lives as
    long as the graph."""
    w, seen = _weight(), []

    def hook(*grads):
        seen.append(grads[-1][0] if register == "register_hook" else grads[0][0])
    node = _node(w)
    if held:
        getattr(node, register)(hook)
        y = _Product.apply(X, w)
    else:
        y = _Product.apply(X, w)
        getattr(y.grad_fn.next_functions[1][0], register)(hook)
        del node
    y.sum().backward()
    assert added == [] and len(seen) == 1 and seen[0] is not None
    assert torch.equal(seen[0], w.grad)


def test_prehook_on_the_accumulation_node_changes_the_gradient(added):
    w = _weight()
    node = _node(w)
    handle = node.register_prehook(lambda g: (g[0] * 0,))
    _Product.apply(X, w).sum().backward()
    assert not w.grad.any()
    handle.remove()
    _Product.apply(X, w).sum().backward()
    assert added == [(4, 4)] and w.grad.any()


def test_tensor_hooks_and_multi_grad_hooks_see_the_gradient(added):
    w, seen = _weight(), []
    handles = [w.register_hook(seen.append), torch.autograd.graph.register_multi_grad_hook((w,), lambda g: seen.append(g[0]))]
    _Product.apply(X, w).sum().backward()
    assert added == [] and len(seen) == 2 and all(g is not None for g in seen)
    for h in handles:
        h.remove()
    w.register_post_accumulate_grad_hook(lambda p: seen.append(p.grad))
    _Product.apply(X, w).sum().backward()
    assert added == [] and len(seen) == 3


def test_weight_used_twice_with_and_without_a_hook(added):
    w = _weight()
    _Product.apply(_Product.apply(X, w), w).sum().backward()
    assert len(added) == 2
    seen, before = [], w.grad.clone()
    y = _Product.apply(_Product.apply(X, w), w)
    y.grad_fn.next_functions[1][0].register_prehook(lambda g: seen.append(g[0]))
    y.sum().backward()
    assert len(added) == 2 and len(seen) == 1
    torch.testing.assert_close(w.grad, before + seen[0])


def test_anomaly_detection_sees_a_nan_weight_gradient(added):
    """Anomaly mode looks at the gradients that functions return."""
    w = _weight()
    x = torch.full((3, 4), float("nan")).bfloat16()
    with pytest.warns(UserWarning), torch.autograd.detect_anomaly():
        y = _Product.apply(x, w)
        with pytest.raises(RuntimeError, match="nan values"):
            y.sum().backward()
    assert added == [] and not w.grad.isnan().any()


def test_gradient_that_is_differentiated_again_is_returned(added):
    w = _weight()
    x = X.clone().requires_grad_()
    _Product.apply(x, w).square().sum().backward(create_graph=True)
    assert added == [] and w.grad.requires_grad


def test_buffer_saved_for_another_backward_is_known_to_have_changed(added):
    w = _weight()
    k = torch.ones((), dtype=torch.bfloat16, requires_grad=True)
    z = (w.grad * k).sum()                  # saves the buffer
    _Product.apply(X, w).sum().backward()
    assert added == [(4, 4)]
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        z.backward()


def test_merged_projection_adds_both_halves_or_fails(added, monkeypatch):
    """The first half is in the buffer already when the second is refused: that must not pass for a whole gradient."""
    w = torch.nn.Parameter(torch.randn(4, 8).bfloat16())
    w.grad, w.flat_grad = torch.zeros_like(w), True
    monkeypatch.setattr(cuda_ops.gemm_tcgen05, "add_supported", lambda a, b, out: True)
    cuda_ops.linear_merged(X, X, w).sum().backward()
    assert added == [(4, 4), (4, 4)] and torch.equal(w.grad[:, :4], w.grad[:, 4:]) and w.grad.any()
    first = gemm.gemm_tn_add
    monkeypatch.setattr(gemm, "gemm_tn_add", lambda a, b, out: len(added) < 3 and first(a, b, out))
    with pytest.raises(_lib.NativeError):
        cuda_ops.linear_merged(X, X, w).sum().backward()
