"""Backward on the tcgen05 kernels at head dim 64 and 128: lengths around the ring's stages and the tiles' halves, for each kernel
(one kernel, query-major with a full or a shared bias gradient, key-major) and each way a bias is added."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("S,T", [(128, 64), (256, 33), (384, 200), (512, 128), (896, 130), (65, 97), (31, 300)])
@pytest.mark.parametrize("kind", ["plain", "causal", "key_mask", "tile", "tile_odd_scale", "tile_neg", "full_grad", "full_grad_mask",
                                  "shared_grad", "key_grad"])
def test_gradients_against_fp64(D, dtype, S, T, kind):
    from nitrix_b200.nn.attention import sdpa_backward, sdpa_forward

    g = torch.Generator(device="cuda").manual_seed(S * 1000 + T)
    B, H = 2, 2
    q, dout = (torch.randn(B, H, S, D, generator=g, device="cuda").to(dtype) for _ in range(2))
    k, v = (torch.randn(B, H, T, D, generator=g, device="cuda").to(dtype) for _ in range(2))
    scale = {"tile_odd_scale": 0.3, "tile_neg": -0.125}.get(kind, 0.125)
    shape = {"shared_grad": (1, H, S, T), "key_grad": (1, H, 1, T)}.get(kind, (B, H, S, T))
    bias = torch.randn(shape, generator=g, device="cuda").to(dtype) if "tile" in kind or "grad" in kind else None
    mask = None
    if kind == "key_mask":
        mask = (torch.arange(T, device="cuda") < torch.tensor([[1], [(T + 1) // 2]], device="cuda")).reshape(B, 1, 1, T)
    if kind == "full_grad_mask":
        mask = torch.rand(B, 1, S, T, generator=g, device="cuda") < 0.8
        mask[..., 0] = True
    causal, want_dbias = kind == "causal", "grad" in kind
    out, lse = sdpa_forward(q, k, v, bias, mask, scale=scale, causal=causal)
    got = sdpa_backward(q, k, v, bias, mask, out, lse, dout, scale=scale, causal=causal, want_dbias=want_dbias)
    leaves = [t.double().requires_grad_(True) for t in (q, k, v)] + ([bias.double().requires_grad_(True)] if want_dbias else [])
    s = leaves[0] @ leaves[1].transpose(-1, -2) * scale
    if bias is not None:
        s = s + (leaves[3] if want_dbias else bias.double())
    if mask is not None:
        s = s.masked_fill(~mask, -math.inf)
    if causal:
        s = s.masked_fill(torch.ones(S, T, device="cuda", dtype=torch.bool).triu(1), -math.inf)
    want = torch.autograd.grad(s.softmax(-1) @ leaves[2], leaves, dout.double())
    # p, ds, out and the gradients are rounded to 16 bits (2^-9 / 2^-12 relative each)
    tol = 2e-2 if dtype == torch.bfloat16 else 4e-3
    for name, a, b in zip(("dq", "dk", "dv", "dbias"), got, want):
        assert float((a.double() - b).abs().max()) <= tol * max(1.0, float(b.abs().max())), name
