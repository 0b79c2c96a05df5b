"""Selective scan on the GPU against the restated recipe: forward and every gradient, through the C ABI.

The comparison runs the recipe in fp64 on the same (quantised) operands on the device and differentiates it with
autograd, as the reference differentiates its own recipe.  fp32 within 2e-5 of max |reference|; 16-bit within an
output ulp of the storage dtype plus that.  Shapes cover every state-count instantiation (up to 16, 32, 64), lengths
on and off the eight-step chunks, a channel count that does not fill the last CTA, leading batch axes, B and C shared
over the batch, and the optional D.
"""
import pathlib

import numpy as np
import pytest
import torch

from oracle import scan_oracle as S

pytestmark = pytest.mark.gpu


def _operands(lead, length, d, n, dtype, with_d, seed, shared_bc=False):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(lead + (length, d), device="cuda", generator=g)
    delta = torch.rand(lead + (length, d), device="cuda", generator=g) * 0.5 + 0.01
    A = -(torch.rand(d, n, device="cuda", generator=g) * 1.5 + 0.2)
    bc_lead = () if shared_bc else lead
    B = torch.randn(bc_lead + (length, n), device="cuda", generator=g)
    C = torch.randn(bc_lead + (length, n), device="cuda", generator=g)
    D = torch.randn(d, device="cuda", generator=g) if with_d else None
    dy = torch.randn(lead + (length, d), device="cuda", generator=g)
    return [None if t is None else t.to(dtype) for t in (x, delta, A, B, C, D, dy)]


def _run(lead, length, d, n, dtype, with_d=True, seed=0, shared_bc=False):
    from nitrix_b200 import _cabi
    from nitrix_b200.nn import ssm

    x, delta, A, B, C, D, dy = _operands(lead, length, d, n, dtype, with_d, seed, shared_bc)
    leaves = [t.detach().clone().requires_grad_(True) for t in (x, delta, A, B, C) + ((D,) if with_d else ())]
    y = ssm.selective_scan(*leaves[:5], leaves[5] if with_d else None)
    grads = torch.autograd.grad(y, leaves, grad_outputs=dy)
    torch.cuda.synchronize()
    assert _cabi.lib().nb200_device_status(0) == 0, _cabi.last_error()
    ref_leaves = [t.detach().double().requires_grad_(True) for t in (x, delta, A, B, C) + ((D,) if with_d else ())]
    want = S.selective_scan_torch(*ref_leaves[:5], ref_leaves[5] if with_d else None)
    ref_grads = torch.autograd.grad(want, ref_leaves, grad_outputs=dy.double())
    tol = 2e-5 if dtype == torch.float32 else (1.5e-2 if dtype == torch.bfloat16 else 2e-3)
    assert y.dtype == dtype and y.shape == x.shape
    err = float((y.detach().double() - want.detach()).abs().max() / want.detach().abs().max())
    assert err <= tol, ("y", err)
    for name, a, r in zip(("dx", "ddelta", "dA", "dB", "dC", "dD"), grads, ref_grads):
        assert a.dtype == dtype and a.shape == r.shape, name
        err = float((a.double() - r).abs().max() / r.abs().max().clamp_min(1e-6))   # (dA is exactly 0 at length 1)
        assert err <= tol, (name, err)


def test_reference_golden_vector_on_the_gpu():
    from nitrix_b200.nn import ssm

    z = np.load(pathlib.Path(__file__).resolve().parent / "golden" / "selective_scan_float32.npz")
    y = ssm.selective_scan(*(torch.from_numpy(z[k]).cuda() for k in ("x", "delta", "A", "B", "C", "D")))
    np.testing.assert_allclose(y.cpu().numpy(), z["out"], atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("length,d,n", [(1, 8, 4), (8, 64, 16), (37, 100, 16), (64, 200, 3), (129, 96, 32),
                                        (50, 70, 64), (256, 256, 16)])
def test_forward_and_gradients(length, d, n, dtype):
    _run((2,), length, d, n, dtype)


def test_without_the_skip_term_and_with_leading_axes():
    _run((2, 3), 40, 48, 8, torch.float32, with_d=False)
    _run((), 33, 130, 16, torch.float32, with_d=True)


def test_projections_shared_over_the_batch_get_summed_gradients():
    _run((3,), 29, 72, 16, torch.float32, shared_bc=True)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("batch,length,d,n", [(8, 17, 1184, 16), (9, 40, 1061, 8), (8, 25, 1177, 5), (37, 9, 256, 12),
                                              (8, 450, 1030, 16), (8, 450, 1030, 33)])
def test_ragged_channels_and_states_and_several_chunks_per_cta(batch, length, d, n, dtype):
    # channel counts that are no multiple of four (scalar loads) and states that are none, up to 8, 16 and 64; CTAs of the
    # gradients with more than one chunk
    _run((batch,), length, d, n, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("batch,length,d,n,pairs", [(5, 40, 200, 16, 400), (5, 40, 200, 16, 399), (5, 40, 200, 16, 199), (3, 33, 250, 5, 64),
                                                    (3, 17, 333, 33, 130), (2, 9, 30, 8, 30)])
def test_backward_in_ranges_of_a_smaller_workspace(monkeypatch, batch, length, d, n, pairs, dtype):
    # room for the adjoint states of `pairs` (batch element, channel) pairs: two elements at a time and a last one, one
    # element, groups of 64 channels with a last one cut short, the least
    from nitrix_b200 import _cabi
    from nitrix_b200.nn import ssm

    def small(p, device):
        full, least = (ssm._bytes(getattr(_cabi.lib(), f"nb200_selective_scan_workspace{q}_bytes"), p) for q in ("", "_least"))
        states = 4 * ((length + 7) // 8) * n
        size = full - (batch * d - pairs) * states
        assert least == full - (batch * d - min(d, 64)) * states and least <= size
        ws = torch.empty(size, dtype=torch.uint8, device=device)
        p.workspace, p.workspace_bytes = ws.data_ptr(), size
        return ws

    monkeypatch.setattr(ssm, "_workspace", small)
    _run((batch,), length, d, n, dtype)


def test_a_device_without_room_for_all_adjoint_states_runs_in_ranges(monkeypatch):
    empty, seen = torch.empty, []

    def bounded(*shape, **kw):
        if kw.get("dtype") == torch.uint8:
            seen.append(shape[0])
            if len(seen) == 1:
                raise torch.OutOfMemoryError("no room")
        return empty(*shape, **kw)

    monkeypatch.setattr(torch, "empty", bounded)
    _run((4,), 64, 128, 16, torch.float32)
    assert len(seen) == 2 and seen[1] == seen[0] - 4 * 8 * 16 * (4 * 128 - 64)


@pytest.mark.parametrize("length", [1, 3, 4, 5, 12, 17, 20])
def test_sequences_that_end_inside_a_staged_chunk(length):
    # steps are staged by sixteen and taken by four; groups past the end are left out
    _run((3,), length, 72, 16, torch.float32)


@pytest.mark.parametrize("batch,length,d,n", [(256, 33, 20, 16), (300, 70, 64, 33)])
def test_many_sequences_of_few_channels(batch, length, d, n):
    # several chunks per CTA so that fewer CTAs add to the same sums of dA and dD, the last CTA of a sequence with fewer
    _run((batch,), length, d, n, torch.float32)


@pytest.mark.parametrize("lead,length,d,n,dtype", [
    ((1,), 96, 16, 8, torch.float32),        # four segments of 32 steps, the last empty
    ((2,), 97, 5, 16, torch.float32),        # a segment of one step
    ((1,), 192, 33, 3, torch.bfloat16),      # eight segments, two of them empty
    ((3,), 400, 20, 32, torch.float32),      # eight of 64, the last ragged
    ((1,), 131, 130, 64, torch.float16),
    ((2,), 95, 40, 16, torch.float32),       # just below the line: not split
])
def test_walks_split_in_time(lead, length, d, n, dtype):
    """Few channels: segments of the sequence walked side by side, joined by their decays."""
    _run(lead, length, d, n, dtype, seed=length)


# Nine steps whose decays multiply to 2^exponent lie in one segment of the split walks; the other steps' are 2^-0.003.
_ENDS = {"growth over an empty state": (0.0, 200.0), "growth of a small state": (1e-30, 135.0),
         "decay of a large state": (1e30, -140.0), "growth out of the range": (0.0, 600.0)}


@pytest.mark.parametrize("length,n", [(256, 8), (112, 33)])   # eight segments, four with a short one
@pytest.mark.parametrize("form", _ENDS)
def test_segments_join_at_the_ends_of_the_range(form, length, n):
    """What enters a segment passes its whole decay as it would step by step: forward, and mirrored through dx.  Tolerance:
    an exponent of 97 (140 ln 2) times its rate and its span, rounded to 2^-24 three or four times (2e-5), some 45
    exponentials of 2^-22 and as many products of 2^-24 behind it (1.3e-5): 4e-5 of the largest."""
    from nitrix_b200.nn import selective_scan

    start, exponent = _ENDS[form]
    g = torch.Generator(device="cuda").manual_seed(length)
    lead, d, seg = 2, 20, 32
    A = torch.full((d, n), 1.0 if exponent > 0 else -1.0, device="cuda")
    delta = torch.full((lead, length, d), 2.0 ** -9, device="cuda")
    delta[:, seg + 4:seg + 13] = abs(exponent) / 9 * float(np.log(2.0))
    x = torch.zeros(lead, length, d, device="cuda")
    x[:, :4] = start
    C = torch.rand(lead, length, n, generator=g, device="cuda") + 0.5
    C[:, :length - 16] = 0.0    # (what is read is what has passed the segment)
    B = torch.rand(lead, length, n, generator=g, device="cuda") + 0.5
    if start == 0.0:
        x[:, length - 16:] = 1.0
    want = S.selective_scan_torch(*(t.double() for t in (x, delta, A, B, C)))
    y = selective_scan(x, delta, A, B, C)
    assert float((y.double() - want).abs().max()) <= 4e-5 * float(want.abs().max()), form
    # the adjoint walk is the same recurrence last step first, one step later: dy for x, C for B
    rx, rd, rB, rC = (t.flip(1).contiguous() for t in (x, delta, B, C))
    dx, dx64 = [], []
    for z, to, fn in ((torch.zeros_like(x), dx, selective_scan), (torch.zeros_like(x).double(), dx64, S.selective_scan_torch)):
        z.requires_grad_(True)
        to.append(torch.autograd.grad(fn(z, *(t.to(z.dtype) for t in (rd, A, rC, rB))), z, rx.to(z.dtype))[0])
    assert float(dx64[0].abs().max()) > 0
    assert float((dx[0].double() - dx64[0]).abs().max()) <= 4e-5 * float(dx64[0].abs().max()), form


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("length,n", [(256, 8), (112, 33)])
def test_segments_of_states_without_memory(length, n, dtype):
    """A rate of -inf (an fp16 -exp(A_log) overflows to it): the state is what its own step put in, in every segment."""
    from nitrix_b200.nn import selective_scan

    x, delta, A, B, C, _, dy = _operands((2,), length, 20, n, dtype, False, 5)
    A[::3, 1::2] = -float("inf")
    leaves = [t.detach().clone().requires_grad_(True) for t in (x, B, C)]
    y = selective_scan(leaves[0], delta, A, *leaves[1:])
    grads = torch.autograd.grad(y, leaves, dy)
    ref = [t.detach().double().requires_grad_(True) for t in (x, B, C)]
    want = S.selective_scan_torch(ref[0], delta.double(), A.double(), *ref[1:])
    tol = 2e-5 if dtype == torch.float32 else 2e-3   # as above
    for a, r in zip((y.detach(), *grads), (want.detach(), *torch.autograd.grad(want, ref, dy.double()))):
        assert float((a.double() - r).abs().max()) <= tol * float(r.abs().max())


def test_the_backward_asks_this_module_for_its_scratch_each_time(monkeypatch):
    from nitrix_b200.nn import ssm

    own, calls = ssm._workspace, []
    _run((2,), 40, 24, 8, torch.float32)
    monkeypatch.setattr(ssm, "_workspace", lambda p, device: (calls.append(device), own(p, device))[1])
    _run((2,), 40, 24, 8, torch.float32)
    assert len(calls) == 1
