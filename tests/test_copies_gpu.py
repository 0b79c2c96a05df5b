"""The kernels that bring operands into the layout the attention kernels read and results out of it: padded copies of a bias
and its gradient, packed masks, the last pass over a shared bias' gradient."""
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


@pytest.mark.parametrize("layout", ["dense", "odd_start", "key_strided"])
@pytest.mark.parametrize("S,T", [(4, 30011), (1, 90003), (1500, 65), (1500, 63), (400, 257)])
def test_padded_copies_of_few_long_and_of_many_short_rows(S, T, layout):
    # rows cut into pieces (the last one shorter), whole rows, and rows taken element by element
    test_padded_copies_of_a_bias_keep_every_element(S, T, layout)


def _words(bits):
    """(..., n) booleans -> (..., ceil(n / 32) rounded up to 4) 32-bit words, bit i of word w = element 32 w + i."""
    n = bits.shape[-1]
    words = (-(-n // 32) + 3) // 4 * 4
    full = torch.zeros(*bits.shape[:-1], words * 32, dtype=torch.int64)
    full[..., :n] = bits
    weights = 2 ** torch.arange(32, dtype=torch.int64)
    w = (full.reshape(*bits.shape[:-1], words, 32) * weights).sum(-1)
    return torch.where(w >= 2 ** 31, w - 2 ** 32, w).to(torch.int32)


@pytest.mark.parametrize("layout", ["dense", "rows_of_8", "odd_start", "key_strided"])
@pytest.mark.parametrize("S,T", [(2, 1), (63, 16), (64, 256), (65, 264), (130, 272), (257, 511), (100, 31)])
def test_packed_mask_bits(S, T, layout):
    """Row-major and transposed words against a packing on the CPU, for every way the kernel reads the mask."""
    from nitrix_b200.nn.attention import pack_mask

    B, H, D = 2, 3, 64
    g = torch.Generator().manual_seed(S * 1000 + T)
    values = torch.randint(0, 4, (B, H, S, T), generator=g, dtype=torch.uint8) * 85      # 0, 85, 170, 255
    if layout == "dense":
        mask = values.cuda()
    elif layout == "rows_of_8":
        mask = torch.empty(B, H, S, (T + 7) // 8 * 8, dtype=torch.uint8, device="cuda")[..., :T].copy_(values)
    elif layout == "odd_start":
        mask = torch.empty(B, H, S, T + 1, dtype=torch.uint8, device="cuda")[..., 1:].copy_(values)
    else:
        mask = values.transpose(-1, -2).contiguous().cuda().transpose(-1, -2)
    q = torch.empty(B, H, S, D, device="cuda", dtype=torch.bfloat16)
    k = torch.empty(B, H, T, D, device="cuda", dtype=torch.bfloat16)
    blob = pack_mask(q, k, k, mask).blob.cpu()
    rows, cols = _words(values != 0), _words((values != 0).transpose(-1, -2))
    at = (rows.numel() * 4 + 255) // 256 * 256
    assert torch.equal(blob[:rows.numel() * 4].view(torch.int32).reshape(rows.shape), rows)
    assert torch.equal(blob[at:at + cols.numel() * 4].view(torch.int32).reshape(cols.shape), cols)


@pytest.mark.parametrize("layout", ["dense", "rows_of_8", "odd_start", "key_strided"])
@pytest.mark.parametrize("S,T", [(64, 32), (65, 24), (9, 8), (130, 7), (200, 33), (9, 100)])
def test_packed_mask_bits_of_narrow_masks_and_of_warps_without_rows(S, T, layout):
    test_packed_mask_bits(S, T, layout)


@pytest.mark.parametrize("T", [1, 31, 256, 257, 1000, 8200])
def test_packed_key_mask_bits_and_kept_lengths(T):
    from nitrix_b200.nn.attention import pack_mask

    B, H, S, D = 5, 2, 3, 64
    keep = torch.rand(B, 1, 1, T, generator=torch.Generator().manual_seed(T)) < 0.5
    keep[0] = False                                   # no kept key: length 0
    keep[1] = True
    keep[2, ..., T // 2:] = False
    q = torch.empty(B, H, S, D, device="cuda", dtype=torch.bfloat16)
    k = torch.empty(B, H, T, D, device="cuda", dtype=torch.bfloat16)
    blob = pack_mask(q, k, k, keep.cuda()).blob.cpu()
    rows = _words(keep)
    at = (rows.numel() * 4 + 255) // 256 * 256
    assert torch.equal(blob[:rows.numel() * 4].view(torch.int32).reshape(rows.shape), rows)
    lengths = torch.where(keep, torch.arange(1, T + 1), 0).amax(-1).flatten().to(torch.int32)
    assert torch.equal(blob[at:at + 4 * B].view(torch.int32), lengths)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("S,T", [(16, 16), (31, 127), (33, 129), (64, 128), (40, 257), (300, 19), (20, 15)])
def test_gradient_of_a_shared_bias_leaves_in_any_layout(S, T, dtype):
    """Two heads add to the same sums, in either order the same bits: the tiled last pass against the strided one."""
    from nitrix_b200.nn.attention import sdpa_backward, sdpa_forward

    g = torch.Generator(device="cuda").manual_seed(S * 1000 + T)
    q, dout = (torch.randn(1, 2, S, 64, generator=g, device="cuda").to(dtype) for _ in range(2))
    k, v = (torch.randn(1, 2, T, 64, generator=g, device="cuda").to(dtype) for _ in range(2))
    bias = torch.randn(1, 1, S, T, generator=g, device="cuda").to(dtype)
    out, lse = sdpa_forward(q, k, v, bias, scale=0.125)
    got = []
    for buf in (torch.empty_like(bias), torch.empty(1, 1, S, T + 3, device="cuda", dtype=dtype)[..., 1:T + 1],
                torch.empty(1, 1, T, S, device="cuda", dtype=dtype).transpose(-1, -2)):
        bufs = (torch.empty_like(q), torch.empty_like(k), torch.empty_like(v), buf)
        got.append(sdpa_backward(q, k, v, bias, None, out, lse, dout, scale=0.125, want_dbias=True, grads=bufs)[3])
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    p = (q.double() @ k.double().transpose(-1, -2) * 0.125 + bias.double()).softmax(-1)
    dp = dout.double() @ v.double().transpose(-1, -2)
    ref = (p * (dp - (p * dp).sum(-1, keepdim=True))).sum(1, keepdim=True)
    tol = 1e-4 if dtype == torch.float32 else 2e-2
    assert float((got[0].double() - ref).abs().max()) <= tol * max(1.0, float(ref.abs().max()))
