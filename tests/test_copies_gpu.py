"""The kernels that bring operands into the layout the attention kernels read: padded copies of a bias and its gradient."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gradient_buffer(shape, layout):
    if layout == "odd_start":        # rows of an odd number of elements that start at an odd one
        *lead, t = shape
        return torch.empty(*lead, t + t % 2 + 1, device="cuda", dtype=torch.bfloat16)[..., 1:t + 1]
    if layout == "key_strided":
        *lead, s, t = shape
        return torch.empty(*lead, t, s, device="cuda", dtype=torch.bfloat16).transpose(-1, -2)
    return torch.empty(shape, device="cuda", dtype=torch.bfloat16)


@pytest.mark.parametrize("layout", ["dense", "odd_start", "key_strided"])
@pytest.mark.parametrize("S,T", [(1, 1), (2, 3), (5, 64), (33, 127), (64, 130), (70, 65), (3, 515)])
def test_padded_copies_of_a_bias_keep_every_element(S, T, layout):
    """A bias whose rows are no multiple of 16 bytes goes through a padded copy, its gradient through another; a bias held
    in rows of 16 bytes needs none.  Same kernels, same operands: the same bits."""
    from nitrix_b200.nn.attention import sdpa_backward, sdpa_forward

    g = torch.Generator(device="cuda").manual_seed(S * 1000 + T)
    B, H, D = 2, 3, 64
    q, dout = (torch.randn(B, H, S, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(B, H, T, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    held = torch.randn(B, H, S, (T + 15) // 16 * 16, generator=g, device="cuda").bfloat16()[..., :T]
    bias = _gradient_buffer((B, H, S, T), layout).copy_(held)
    want, lse = sdpa_forward(q, k, v, held, scale=0.125)
    out, lse2 = sdpa_forward(q, k, v, bias, scale=0.125)
    assert torch.equal(out, want) and torch.equal(lse, lse2)
    # the gradient in this layout, and densely
    grads = []
    for lay in (layout, "dense"):
        bufs = (torch.empty_like(q), torch.empty_like(k), torch.empty_like(v), _gradient_buffer((B, H, S, T), lay))
        grads.append(sdpa_backward(q, k, v, bias, None, out, lse, dout, scale=0.125, want_dbias=True, grads=bufs))
    for name, a, b in zip(("dq", "dk", "dv", "dbias"), *grads):
        assert torch.equal(a, b), name
    p = (q.double() @ k.double().transpose(-1, -2) * 0.125 + held.double()).softmax(-1)
    dp = dout.double() @ v.double().transpose(-1, -2)
    ref = p * (dp - (p * dp).sum(-1, keepdim=True))
    # p and ds are rounded to bf16 (2^-9), out (in delta) too
    assert float((grads[0][3].double() - ref).abs().max()) <= 2e-2 * max(1.0, float(ref.abs().max()))
