"""fp32 attention on the tcgen05 kernels (three bf16 planes per operand, six products): forward and every gradient against
a restatement in fp64 on the device, at the sizes where the kernels can go wrong.

Bound: the products left out are below 2^-20 (1e-6) of the one they belong to; the tensor core truncates each of the 24
accumulations of a 64-key step, half an ulp (2^-24) of the sum so far on average, and the accumulators are emptied every
other step: 48 * 2^-24 = 2.9e-6; the scores and dP, 24 accumulations each, add 1.4e-6 on the way in and ex2 2^-22.  So
6e-6 in the 2-norm.
"""
import ctypes as C
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

_BOUND = 6e-6


def _reference(q, k, v, bias, mask, causal, scale, dout):
    q, k, v, dout = (t.double() for t in (q, k, v, dout))
    s = q @ k.transpose(-1, -2) * scale
    if bias is not None:
        s = s + bias.double()
    if mask is not None:
        s = s.masked_fill(~mask, -math.inf)
    if causal:
        s = s.masked_fill(torch.ones(s.shape[-2:], device=s.device, dtype=torch.bool).triu(1), -math.inf)
    p = s.softmax(-1)
    out = p @ v
    ds = p * (dout @ v.transpose(-1, -2) - (out * dout).sum(-1, keepdim=True))
    dbias = None
    if bias is not None:
        dbias = ds
        for a, n in enumerate(bias.shape):
            if n == 1 and ds.shape[a] != 1:
                dbias = dbias.sum(a, keepdim=True)
    return out, ds @ k * scale, ds.transpose(-1, -2) @ q * scale, p.transpose(-1, -2) @ dout, dbias


def _err(a, b):
    return float((a.double() - b).norm() / b.norm())


def _layout(t, kind):
    if kind == "bshd":        # a (B, S, H, D) buffer seen as (B, H, S, D)
        return t.transpose(1, 2).contiguous().transpose(1, 2)
    if kind == "odd":         # rows of D + 1 floats, starting one float in: no 16-byte loads
        b = torch.zeros(t.shape[:-1] + (t.shape[-1] + 1,), device=t.device)
        b[..., 1:] = t
        return b[..., 1:]
    return t


@pytest.mark.parametrize("B,H,S,T,D,causal,bias,mask,layout", [
    (4, 32, 128, 256, 64, False, None, None, "dense"),       # whole tiles, an even number of steps
    (4, 48, 65, 321, 64, False, None, None, "bshd"),         # a second tile of one row; an odd last step of one key
    (2, 64, 300, 130, 64, False, None, None, "odd"),         # second CTA of one query tile; three steps
    (3, 40, 257, 257, 64, True, None, None, "dense"),        # causal over CTAs of two tiles
    (2, 100, 200, 500, 32, False, None, None, "dense"),      # head dim padded to the 64 columns
    (2, 60, 330, 200, 32, True, "full", "key", "bshd"),      # causal with more queries than keys
    (4, 50, 130, 333, 64, False, "full", "full", "dense"),   # ragged bias and mask
    (4, 50, 130, 333, 64, False, "shared", None, "dense"),   # fp32 sums over the batch
    (4, 50, 130, 333, 64, True, "key", "key", "dense"),      # neither has a query axis
    (4, 50, 190, 320, 64, False, "bf16", None, "dense"),     # a 16-bit bias of fp32 operands
    (2, 20, 200, 200, 128, False, "full", "full", "dense"),  # head dim 128 (forward)
    (1, 3, 100, 1111, 128, True, None, None, "odd"),
])
def test_against_fp64(B, H, S, T, D, causal, bias, mask, layout):
    from nitrix_b200 import _cabi
    from nitrix_b200.nn import attention as att

    g = torch.Generator(device="cuda").manual_seed(B * 1000 + S)
    q, k, v, dout = (torch.randn(B, H, n, D, device="cuda", generator=g) for n in (S, T, T, S))
    q, k, v, dout = (_layout(t, layout) for t in (q, k, v, dout))
    shape = {"full": (B, H, S, T), "shared": (1, H, S, T), "key": (1, H, 1, T), "bf16": (B, H, S, T)}
    bias_t = None if bias is None else torch.randn(shape[bias], device="cuda", generator=g)
    if bias == "bf16":
        bias_t = bias_t.bfloat16()
    mask_t = None
    if mask is not None:
        mask_t = torch.rand((B, 1, S if mask == "full" else 1, T), device="cuda", generator=g) > 0.2
        mask_t[..., 0] = True
    scale = 1.0 / math.sqrt(D)
    L = _cabi.lib()
    L.nb200_profile(1)
    out, lse = att.sdpa_forward(q, k, v, bias_t, mask_t, scale=scale, causal=causal)
    grads = att.sdpa_backward(q, k, v, bias_t, mask_t, out, lse, dout, scale=scale, causal=causal, want_dbias=bias is not None)
    torch.cuda.synchronize()
    ran = set(_cabi.kernel_times())
    L.nb200_profile(0)
    assert L.nb200_device_status(0) == 0, _cabi.last_error()
    assert "fwd_fp32_tc_kernel" in ran, ran
    tc_backward = D < 128 and min(S, T) > 64
    assert ("bwd_dkv_fp32_tc_kernel" in ran) == tc_backward, ran
    want = _reference(q, k, v, bias_t, mask_t, causal, scale, dout)
    assert _err(out, want[0]) <= _BOUND
    for name, a, r in zip(("dq", "dk", "dv", "dbias"), grads, want[1:]):
        if r is not None:
            # (a 16-bit dbias is rounded on the way out; the kernels of other paths have the fp32 budget of 1e-4)
            assert _err(a, r) <= (5e-3 if a.dtype != torch.float32 else (_BOUND if tc_backward else 1e-4)), name


@pytest.mark.parametrize("B,H,S,T,D,kind,fwd,bwd", [
    # each line of the two rules from both sides: (forward, backward) on these kernels?
    (3, 8, 128, 128, 64, "none", False, False), (6, 8, 128, 128, 64, "none", False, True), (16, 8, 128, 128, 64, "none", True, True),
    (24, 8, 128, 128, 64, "none", False, True), (24, 8, 128, 128, 64, "key", True, True),
    (12, 8, 192, 192, 32, "none", False, False), (8, 8, 192, 192, 32, "none", False, True), (8, 8, 200, 200, 32, "none", False, True),
    (4, 8, 344, 344, 32, "none", True, True), (4, 8, 512, 100, 32, "none", False, False), (12, 8, 160, 160, 32, "mask", False, False),
    (12, 8, 128, 128, 32, "mask", False, True), (6, 8, 512, 512, 32, "mask", False, True), (4, 8, 768, 768, 32, "mask", True, True),
    (12, 8, 200, 200, 32, "both", True, True), (3, 8, 200, 200, 32, "both", False, False),
    (16, 8, 40, 80, 128, "none", False, False), (8, 8, 40, 80, 128, "none", True, False), (16, 8, 48, 300, 128, "mask", True, False),
])
def test_both_sides_of_the_lines_between_the_fp32_kernels(B, H, S, T, D, kind, fwd, bwd):
    from nitrix_b200 import _cabi
    from nitrix_b200.nn import attention as att

    g = torch.Generator(device="cuda").manual_seed(S + T)
    q, k, v, dout = (torch.randn(B, H, n, D, device="cuda", generator=g) for n in (S, T, T, S))
    bias = torch.randn(B, H, S, T, device="cuda", generator=g) if kind == "both" else None
    mask = None
    if kind != "none":
        mask = torch.rand((B, 1, 1 if kind == "key" else S, T), device="cuda", generator=g) > 0.2
        mask[..., 0] = True
    L = _cabi.lib()
    L.nb200_profile(1)
    out, lse = att.sdpa_forward(q, k, v, bias, mask, scale=D ** -0.5)
    grads = att.sdpa_backward(q, k, v, bias, mask, out, lse, dout, scale=D ** -0.5, want_dbias=bias is not None)
    torch.cuda.synchronize()
    ran = set(_cabi.kernel_times())
    L.nb200_profile(0)
    assert ("fwd_fp32_tc_kernel" in ran) == fwd and ("bwd_dkv_fp32_tc_kernel" in ran) == bwd, ran
    want = _reference(q, k, v, bias, mask, False, D ** -0.5, dout)
    # (the mma.sync kernels have the fp32 budget of 1e-4)
    assert _err(out, want[0]) <= (_BOUND if fwd else 1e-4)
    for a, r in zip(grads, want[1:]):
        if r is not None:
            assert _err(a, r) <= (_BOUND if fwd and bwd else 1e-4)


def test_a_problem_whose_planes_exceed_their_limit_runs_in_ranges():
    # 1100 pairs of S = T = 1024 make 1.2 GiB (forward) and 1.6 GiB (backward) of planes: two ranges each
    from nitrix_b200.nn import attention as att

    g = torch.Generator(device="cuda").manual_seed(6)
    q, k, v, dout = (torch.randn(50, 22, 1024, 64, device="cuda", generator=g) for _ in range(4))
    out, lse = att.sdpa_forward(q, k, v, None, None, scale=0.125)
    grads = att.sdpa_backward(q, k, v, None, None, out, lse, dout, scale=0.125)[:3]
    for b in (0, 30, 49):
        want = _reference(q[b:b + 1], k[b:b + 1], v[b:b + 1], None, None, False, 0.125, dout[b:b + 1])
        for a, r in zip((out, *grads), want):
            assert _err(a[b:b + 1], r) <= _BOUND


@pytest.mark.parametrize("with_bias", [False, True])
def test_large_values_do_not_overflow_before_the_division(with_bias):
    # logits that grow by 5 (2^7.2) from the second step on, less than what moves the reference maximum; the sum of 130
    # probabilities of at most 1 times V stays below the largest fp32
    from nitrix_b200.nn import attention as att

    g = torch.Generator(device="cuda").manual_seed(12)
    q, k = torch.ones(4, 50, 130, 64, device="cuda"), torch.zeros(4, 50, 130, 64, device="cuda")
    v = (1.0 + torch.rand(4, 50, 130, 64, device="cuda", generator=g)) * 1e36
    bias = None
    if with_bias:
        bias = torch.zeros(1, 50, 1, 130, device="cuda")
        bias[..., 64:] = 5.0
    else:
        k[:, :, 64:] = 5.0 / 8.0
    out, lse = att.sdpa_forward(q, k, v, bias, None, scale=0.125)
    s = q.double() @ k.double().transpose(-1, -2) * 0.125 + (0.0 if bias is None else bias.double())
    assert _err(out, s.softmax(-1) @ v.double()) <= _BOUND
    assert float((lse.double() - s.logsumexp(-1) / math.log(2.0)).abs().max()) <= 1e-5


def test_rows_without_a_kept_key_are_nan_and_leave_the_others_alone():
    from nitrix_b200.nn import attention as att

    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(4, 50, 130, 64, device="cuda", generator=g) for _ in range(3))
    k, v = (torch.cat([t, t, t], 2).contiguous() for t in (k, v))
    mask = torch.ones(4, 1, 130, 390, device="cuda", dtype=torch.bool)
    mask[:, :, 5] = False
    out, lse = att.sdpa_forward(q, k, v, None, mask, scale=0.125)
    assert out[:, :, 5].isnan().all() and (lse[:, :, 5] == -math.inf).all()
    keep = [i for i in range(130) if i != 5]
    want = (q.double() @ k.double().transpose(-1, -2) * 0.125).softmax(-1) @ v.double()
    assert _err(out[:, :, keep], want[:, :, keep]) <= _BOUND


def test_bias_of_minus_infinity_drops_keys_and_infinite_operands_stay_in_their_rows():
    from nitrix_b200.nn import attention as att

    g = torch.Generator(device="cuda").manual_seed(5)
    q, dout = (torch.randn(4, 50, 130, 64, device="cuda", generator=g) for _ in range(2))
    k, v = (torch.randn(4, 50, 333, 64, device="cuda", generator=g) for _ in range(2))
    bias = torch.randn(4, 50, 130, 333, device="cuda", generator=g)
    bias[torch.rand(bias.shape, device="cuda", generator=g) < 0.2] = -math.inf
    bias[..., 0] = 0.0
    out, lse = att.sdpa_forward(q, k, v, bias, None, scale=0.125)
    grads = att.sdpa_backward(q, k, v, bias, None, out, lse, dout, scale=0.125, want_dbias=True)
    for a, r in zip((out, *grads), _reference(q, k, v, bias, None, False, 0.125, dout)):
        assert _err(a, r) <= _BOUND
    q[0, 0, 7, 3] = math.inf
    v[1, 0, 5, 2] = math.inf
    got, _ = att.sdpa_forward(q, k, v, None, None, scale=0.125)
    bad = torch.zeros_like(got, dtype=torch.bool)
    bad[0, 0, 7] = True
    bad[1, 0, :, 2] = True
    assert not got[bad].isfinite().any() and got[~bad].isfinite().all()


def test_without_workspace_the_other_kernels_run():
    """The workspace is optional: a C caller that brings none (the query answered 0 bytes before these kernels existed)
    gets the mma.sync kernels, forward and backward."""
    from nitrix_b200 import _cabi
    from nitrix_b200.nn import attention as att

    g = torch.Generator(device="cuda").manual_seed(4)
    q, k, v, dout = (torch.randn(4, 50, 200, 64, device="cuda", generator=g) for _ in range(4))
    want = _reference(q, k, v, None, None, False, 0.125, dout)
    out, lse = torch.empty_like(q), torch.empty(4, 50, 200, device="cuda")
    p = _cabi.new_params()
    att._fill_common(p, q, k, v, out, lse, None, None, 0.125, False, _cabi.KERNEL_AUTO, None)
    L, stream = _cabi.lib(), torch.cuda.current_stream().cuda_stream
    L.nb200_profile(1)
    assert L.nb200_sdpa_fwd(C.byref(p), stream) == _cabi.OK, _cabi.last_error()
    dq, dk, dv = (torch.empty_like(q) for _ in range(3))
    p.dout, p.dq, p.dk, p.dv = (t.data_ptr() for t in (dout, dq, dk, dv))
    p.dout_stride[:] = p.dq_stride[:] = p.dk_stride[:] = p.dv_stride[:] = list(q.stride())
    ws = torch.empty(4 * 50 * 200 * 4 + 256, dtype=torch.uint8, device="cuda")     # delta alone
    p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
    assert L.nb200_sdpa_bwd(C.byref(p), stream) == _cabi.OK, _cabi.last_error()
    torch.cuda.synchronize()
    ran = set(_cabi.kernel_times())
    L.nb200_profile(0)
    assert any("tf32x3" in name for name in ran) and not any("fp32_tc" in name or "split_planes" in name for name in ran), ran
    for a, r in zip((out, dq, dk, dv), want):
        assert _err(a, r) <= 1e-4
