"""Forward on the tcgen05 kernels where two threads share a query row (head dim 64) and where the softmax warps' loop is one of
several: growing logits that move the rows' reference maxima at different keys, every kind of addend and scale, rows of the
output that are only 16-byte aligned."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(q, k, v, bias, mask, causal, scale):
    s = q.double() @ k.double().transpose(-1, -2) * scale
    if bias is not None:
        s = s + bias.double()
    if mask is not None:
        s = s.masked_fill(~mask, -math.inf)
    if causal:
        s = s.masked_fill(torch.ones(s.shape[-2:], device=s.device, dtype=torch.bool).triu(1), -math.inf)
    return s.softmax(-1) @ v.double(), s.logsumexp(-1) / math.log(2.0)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("S,T", [(1, 1), (127, 64), (129, 65), (256, 127), (300, 333), (64, 513)])
@pytest.mark.parametrize("kind", ["plain", "ramp", "causal", "tile", "tile_odd_scale", "tile_neg", "key", "key_neg", "neg",
                                  "mask", "key_mask", "tile_mask_causal"])
def test_forward_against_fp64(D, dtype, S, T, kind):
    from nitrix_b200.nn.attention import sdpa_forward

    g = torch.Generator(device="cuda").manual_seed(S * 1000 + T)
    B, H = 2, 2
    q = torch.randn(B, H, S, D, generator=g, device="cuda").to(dtype)
    k = torch.randn(B, H, T, D, generator=g, device="cuda").to(dtype)
    v = torch.randn(B, H, T, D, generator=g, device="cuda").to(dtype)
    scale = {"tile_odd_scale": 0.3, "tile_neg": -0.125, "key_neg": -0.125, "neg": -0.125}.get(kind, 0.125)
    bias = mask = None
    if kind == "ramp":
        # logits that grow along the keys, by more than the 2^8 lag of the reference maximum per 32 keys, not alike per row
        k = (k.float() * (1 + 0.05 * torch.arange(T, device="cuda"))[:, None]).clamp(-60, 60).to(dtype)
    if kind.startswith("tile"):
        bias = (torch.randn(B, H, S, (T + 7) // 8 * 8, generator=g, device="cuda") * 4).to(dtype)[..., :T]
    if kind.startswith("key") and kind != "key_mask":
        bias = torch.randn(1, H, 1, (T + 7) // 8 * 8, generator=g, device="cuda").to(dtype)[..., :T]
    if kind in ("mask", "tile_mask_causal"):
        mask = torch.rand(B, 1, S, T, generator=g, device="cuda") < 0.8
        mask[..., 0] = True
    if kind == "key_mask":
        mask = (torch.arange(T, device="cuda") < torch.tensor([[1], [(T + 1) // 2]], device="cuda")).reshape(B, 1, 1, T)
    causal = kind in ("causal", "tile_mask_causal")
    want, want_lse = _reference(q, k, v, bias, mask, causal, scale)
    # rows of the output 16-byte aligned only; and the ordinary ones
    narrow = torch.empty(B, H, S, D + 8, device="cuda", dtype=dtype)[..., :D]
    for out in (narrow, None):
        got, lse = sdpa_forward(q, k, v, bias, mask, scale=scale, causal=causal, out=out)
        # p and the output are rounded to 16 bits (2^-9 / 2^-12 each), the sums are fp32
        tol = (2.0 if dtype == torch.bfloat16 else 0.25) * 2.0 ** -7
        assert float((got.double() - want).abs().max()) <= tol * max(1.0, float(want.abs().max()))
        assert float((lse.double() - want_lse).abs().max()) <= 1e-3 * max(1.0, float(want_lse.abs().max()))


@pytest.mark.parametrize("D,tile", [(64, True), (64, False), (128, True), (128, False)])
@pytest.mark.parametrize("B", [289, 384, 385])
def test_many_key_padded_batch_elements_whatever_their_order(B, D, tile):
    # items are dealt by kept length up to the largest batch that a CTA ranks; an element's rows depend on nothing else
    from nitrix_b200.nn.attention import sdpa_forward

    g = torch.Generator(device="cuda").manual_seed(B)
    S, T = 40, 264
    q = torch.randn(B, 1, S, D, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(B, 1, T, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    bias = torch.randn(1, 1, S, T, generator=g, device="cuda").bfloat16() if tile else None
    lengths = torch.randint(1, T + 1, (B, 1), generator=g, device="cuda")
    mask = (torch.arange(T, device="cuda") < lengths).reshape(B, 1, 1, T)
    out, lse = sdpa_forward(q, k, v, bias, mask, scale=0.125)
    for i in range(0, B, 100):
        part = slice(i, i + 100)
        out_i, lse_i = sdpa_forward(q[part], k[part], v[part], bias, mask[part], scale=0.125)
        assert torch.equal(out[part], out_i) and torch.equal(lse[part], lse_i)


@pytest.mark.parametrize("kind", ["mask", "mask_shared", "mask_causal", "mask_key_bias", "mask_neg", "key_mask_neg", "key_bias_neg_mask"])
@pytest.mark.parametrize("S,T", [(300, 700), (130, 385), (257, 90)])
def test_staged_mask_words_over_several_items_per_cta(kind, S, T):
    """Head dim 64 without bias tiles: the ring of mask words wraps within an item and from one to the next, query tiles of
    different (causal) and of no (past the last row) key tiles among them.  Tolerance as above."""
    from nitrix_b200.nn.attention import sdpa_forward

    g = torch.Generator(device="cuda").manual_seed(S * 1000 + T)
    B, H, D = 23, 8, 64
    q = torch.randn(B, H, S, D, generator=g, device="cuda").half()
    k, v = (torch.randn(B, H, T, D, generator=g, device="cuda").half() for _ in range(2))
    scale = -0.125 if "neg" in kind else 0.125
    rows = 1 if kind == "key_mask_neg" else S
    mask = torch.rand(1 if kind == "mask_shared" else B, 1, rows, T, generator=g, device="cuda") < 0.7
    mask[..., 0] = True
    bias = torch.randn(1, H, 1, (T + 7) // 8 * 8, generator=g, device="cuda").half()[..., :T] if "bias" in kind else None
    out, lse = sdpa_forward(q, k, v, bias, mask, scale=scale, causal=kind == "mask_causal")
    for i in range(0, B, 4):
        p = slice(i, i + 4)
        want, want_lse = _reference(q[p], k[p], v[p], bias, mask if kind == "mask_shared" else mask[p], kind == "mask_causal", scale)
        assert float((out[p].double() - want).abs().max()) <= 0.25 * 2.0 ** -7 * max(1.0, float(want.abs().max()))
        assert float((lse[p].double() - want_lse).abs().max()) <= 1e-3 * max(1.0, float(want_lse.abs().max()))
