"""The differentiable operations as C++ autograd functions: what autograd asks of them, and what they refuse."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _attention(mask=None):
    from nitrix_b200.nn import scaled_dot_product_attention

    g = torch.Generator(device="cuda").manual_seed(1)
    leaves = [torch.randn(2, 3, 40, 64, generator=g, device="cuda").bfloat16().requires_grad_(True) for _ in range(3)]
    leaves.append(torch.randn(2, 3, 40, 40, generator=g, device="cuda").bfloat16().requires_grad_(True))
    return leaves, lambda q, k, v, b: scaled_dot_product_attention(q, k, v, bias=b, mask=mask, qk_norm=True)


def _layer_norm():
    from nitrix_b200.nn import layer_norm

    g = torch.Generator(device="cuda").manual_seed(2)
    leaves = [torch.randn(n, generator=g, device="cuda").requires_grad_(True) for n in ((5, 64), (64,), (64,))]
    return leaves, lambda x, w, b: layer_norm(x, w, b)


def _scan():
    from nitrix_b200.nn import selective_scan

    g = torch.Generator(device="cuda").manual_seed(3)
    shapes = ((2, 20, 24), (2, 20, 24), (24, 8), (1, 20, 8), (2, 20, 8), (24,))
    leaves = [torch.rand(s, generator=g, device="cuda").sub(0.6 if s == (24, 8) else 0.0).requires_grad_(True) for s in shapes]
    return leaves, selective_scan


_OPS = {"attention": _attention, "layer_norm": _layer_norm, "selective_scan": _scan}


@pytest.mark.parametrize("op", _OPS)
def test_gradients_of_some_operands_and_on_another_stream_and_through_hooks(op):
    leaves, fn = _OPS[op]()
    want = torch.autograd.grad(fn(*leaves).float().square().sum(), leaves)

    def close(a, b):   # (sums added in any order)
        assert float((a.float() - b.float()).norm()) <= 1e-2 * float(b.float().norm())

    for i, leaf in enumerate(leaves):
        only = [t if j == i else t.detach() for j, t in enumerate(leaves)]
        close(torch.autograd.grad(fn(*only).float().square().sum(), [leaf])[0], want[i])
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(1), t.cpu())[1], lambda t: t.cuda()):
        y = fn(*leaves)
    assert packed
    for a, b in zip(torch.autograd.grad(y.float().square().sum(), leaves), want):
        close(a, b)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = torch.autograd.grad(fn(*leaves).float().square().sum(), leaves)
    torch.cuda.current_stream().wait_stream(side)
    for a, b in zip(got, want):
        close(a, b)
    with torch.no_grad():
        assert not fn(*leaves).requires_grad


@pytest.mark.parametrize("op", _OPS)
def test_what_has_no_rule_is_refused(op):
    leaves, fn = _OPS[op]()
    rest = [t.detach() for t in leaves[1:]]
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda x: fn(x, *rest))(torch.stack([leaves[0].detach()] * 2))
    with pytest.raises(RuntimeError), torch.autograd.forward_ad.dual_level():
        fn(torch.autograd.forward_ad.make_dual(leaves[0], torch.ones_like(leaves[0])), *rest)
    x = leaves[0]
    (gx,) = torch.autograd.grad(fn(x, *rest).float().square().sum(), x, create_graph=True)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(gx.float().sum(), x)
    z = leaves[0] * 1
    y = fn(z, *rest)
    z.add_(1)
    with pytest.raises(RuntimeError, match="inplace"):
        y.float().sum().backward()


@pytest.mark.parametrize("expand", [True, False])
@pytest.mark.parametrize("D,S,T", [(64, 128, 200), (128, 100, 130)])
def test_packed_masks_keep_the_layout_they_were_packed_from(D, S, T, expand):
    # a hook that copies hands the backward an expanded mask with dense strides, while its bits were packed per key alone
    from nitrix_b200.nn import scaled_dot_product_attention

    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v = (torch.randn(3, 4, n, D, generator=g, device="cuda").bfloat16().requires_grad_(True) for n in (S, T, T))
    dout = torch.randn(3, 4, S, D, generator=g, device="cuda").bfloat16()
    mask = torch.rand(3, 1, 1 if expand else S, T, generator=g, device="cuda") > 0.3
    mask[..., 0] = True
    mask = mask.expand(3, 4, S, T) if expand else mask
    want = torch.autograd.grad(scaled_dot_product_attention(q, k, v, mask=mask), (q, k, v), dout)
    restored = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: (restored.append(t.cuda()), restored[-1])[1]):
        out = scaled_dot_product_attention(q, k, v, mask=mask)
    got = torch.autograd.grad(out, (q, k, v), dout)
    assert any(t.shape == mask.shape and t.is_contiguous() for t in restored if t.dtype in (torch.bool, torch.uint8))
    for a, b in zip(got, want):   # (fp32 sums of dq added in any order, then rounded to bf16)
        assert float((a.float() - b.float()).norm()) <= 1e-2 * float(b.float().norm())


@pytest.mark.parametrize("op", _OPS)
def test_forward_mode_is_not_implemented(op):
    # (the class that a Python autograd function without a jvp raises, whichever operand has the tangent)
    leaves, fn = _OPS[op]()
    for i in range(len(leaves)):
        with pytest.raises(NotImplementedError), torch.autograd.forward_ad.dual_level():
            fn(*(torch.autograd.forward_ad.make_dual(t, torch.ones_like(t)) if j == i else t for j, t in enumerate(leaves)))
