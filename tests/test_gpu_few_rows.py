"""Products of 2 to 8 activation rows (w4_rows_kernel, and the integer kernel where that takes less).

Bound of the products, per output, with A = sum |x| |w|: activations, codes and their products are exact; a 32-element block's
sum is six accumulating instructions, of which the two with the large pieces may truncate at 2^-23 of at most A and the
others at 2^-8 of that; adding the K / 32 blocks, the eight sums of the warps and the bias takes one fp32 rounding each
(2^-24 A): below (2 * 2 * 1.1 + K / 32 + 10) * 2^-24 * A.  The integer kernel rounds every element to a multiple of 2^-22 of its block's
maximum, half of that at most: 2^-23 * sum over blocks of max |x| sum |w| more."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch

    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: GPU tests need a B200")
    return torch


@pytest.fixture(scope="module")
def tb(torch):
    import torchburn_b200 as tb

    return tb


def int4(torch, n, k, g, seed):
    """(packed, scales, the weights in float64), on the GPU."""
    gen = torch.Generator("cuda").manual_seed(seed)
    w = torch.randn(n, k // g, g, device="cuda", generator=gen) * 0.02
    s = (w.abs().amax(-1) / 7).clamp_min(1e-8)
    c = (w / s[..., None]).round_().clamp_(-8, 7)
    q = c.add(8).to(torch.uint8).reshape(n, k)
    return (q[:, 0::2] | (q[:, 1::2] << 4)).contiguous(), s.contiguous(), (c.double() * s.double()[..., None]).reshape(n, k)


INTEGER = [(5, 16 * 148, 256, 32, 0), (5, 14 * 16 * 148 + 5, 256, 32, 0), (8, 33000, 512, 64, 0), (5, 96, 20480, 64, 0), (3, 700, 8192, 64, 0), (8, 8960, 1536, 32, 1),
           (2, 18944, 896, 32, 1), (5, 18944, 1536, 32, 0), (6, 13824, 1024, 128, 1), (4, 24576, 1024, 32, 1)]


@pytest.mark.parametrize("m,n,k,g,pair", [
    (2, 1, 32, 32, 0), (8, 7, 32, 32, 1), (3, 17, 96, 32, 0),             # one block of K, one ragged tile
    (8, 16 * 148 + 1, 288, 32, 0), (5, 16 * 148, 288, 32, 0),             # a tile per CTA, one more; a stage and an eighth
    (4, 8 * 148 * 2 + 3, 512, 64, 1), (8, 14330, 896, 64, 0),             # unaligned rows of scales, copied in eights
    (7, 4864, 896, 128, 1), (8, 1000, 1920, 128, 0),                      # and in fours; K that is no whole stage
    (5, 14 * 16 * 148 + 5, 288, 32, 0), (8, 33000, 768, 64, 0),           # more tiles than a pass holds, and as many
    (6, 6144, 4096, 32, 0), (8, 4096, 14336, 32, 0), (8, 14336, 4096, 32, 1),
    (8, 8960, 1504, 32, 1), (5, 2400, 8192, 32, 0), (7, 5000, 512, 32, 0), (2, 8288, 1024, 32, 1),   # beside the integer kernel's sizes
    *INTEGER])
def test_products_of_few_rows_match_float64(torch, tb, m, n, k, g, pair):
    p, s, w = int4(torch, n, k, g, m + n + k)
    p2, s2, w2 = int4(torch, n, k, g, m + n + k + 1)
    gen = torch.Generator("cuda").manual_seed(m)
    x = torch.randn(m, k, device="cuda", generator=gen) * 10 ** (6 * torch.rand(m, 1, device="cuda", generator=gen) - 3)
    b = torch.randn(n, device="cuda", generator=gen)
    tol = (4.4 + k / 32 + 10) * 2.0 ** -24
    st = torch.cuda.current_stream().cuda_stream

    def run():
        if not pair:
            return tb.w4a32_grouped_linear(x, p, s, b, g)
        y = torch.empty(m, n, device="cuda")
        assert tb.lib().tb_swiglu_gemv_w4a32(x.data_ptr(), p.data_ptr(), s.data_ptr(), b.data_ptr(), p2.data_ptr(), s2.data_ptr(), None, y.data_ptr(),
                                             m, n, k, g, st) == 0, tb.last_error()
        return y
    y = run()
    try:
        tb.lib().tb_set_gemv_tuning(3, 0, 0)
        integer = torch.equal(run(), y)
    finally:
        tb.lib().tb_set_gemv_tuning(1, 0, 0)
    if n > 17:   # (one narrow case is the CUDA-core kernel's in either mode, too few outputs differ in others)
        assert integer == ((m, n, k, g, pair) in INTEGER)
    top = x.double().abs().reshape(m, k // 32, 32).amax(-1, keepdim=True).expand(m, k // 32, 32).reshape(m, k)

    def more(w):
        return 2.0 ** -23 * (top @ w.abs().T) if integer else 0.0
    gate, bound = x.double() @ w.T + b, (x.double().abs() @ w.abs().T + b.abs()) * tol + more(w)
    if pair:
        up, sig = x.double() @ w2.T, torch.sigmoid(gate)
        # silu' <= 1.1, |silu(g)| <= |g|; four roundings of the epilogue
        bound = 1.1 * bound * up.abs() + gate.abs() * ((x.double().abs() @ w2.abs().T) * tol + more(w2)) + 4 * 2.0 ** -23 * (gate * sig * up).abs() + bound * 1e-6
        gate = gate * sig * up
    assert bool(((y.double() - gate).abs() <= bound + 1e-30).all()), float(((y.double() - gate).abs() / bound).max())
    assert torch.equal(run(), y)   # equal calls give equal bits
    assert tb.lib().tb_device_fault_flag() == 0


@pytest.mark.parametrize("k", [512, 896])   # the integer kernel, the streaming one
def test_few_rows_keep_infinities_to_their_row(torch, tb, k):
    """A row with an infinity or a NaN leaves the other rows as they are."""
    p, s, _ = int4(torch, 300, k, 32, 1)
    x = torch.randn(6, k, device="cuda")
    want = tb.w4a32_grouped_linear(x, p, s, None, 32)
    x[2, 7], x[4, 100] = float("inf"), float("nan")
    got = tb.w4a32_grouped_linear(x, p, s, None, 32)
    keep = [0, 1, 3, 5]
    assert torch.equal(got[keep], want[keep])
    assert bool(torch.isnan(got[4]).all()) and not bool(torch.isfinite(got[2]).any())


@pytest.mark.parametrize("pair", [0, 1])
@pytest.mark.parametrize("m,n,k,g", [(2, 700, 896, 32), (3, 6000, 1024, 64), (4, 4097, 640, 128), (5, 96, 4096, 32), (8, 5003, 4096, 32), (8, 600, 7168, 32), (6, 9600, 288, 32)])
def test_the_integer_kernel_stays_selectable(torch, tb, m, n, k, g, pair):
    """tb_set_gemv_tuning(3, ...) takes these products to the integer kernel: other bits than the default's, within the bound of
    its arithmetic (the streaming kernel's for the sums, and half a step of 2^-22 of a block's maximum for each of its elements)."""
    a, b = int4(torch, n, k, g, 1), int4(torch, n, k, g, 2)
    x = torch.randn(m, k, device="cuda", generator=torch.Generator("cuda").manual_seed(m + k))
    st = torch.cuda.current_stream().cuda_stream

    def run():
        y = torch.full((m, n), float("nan"), device="cuda")
        rc = tb.lib().tb_swiglu_gemv_w4a32(x.data_ptr(), a[0].data_ptr(), a[1].data_ptr(), None, b[0].data_ptr(), b[1].data_ptr(), None, y.data_ptr(), m, n, k, g, st) if pair else \
            tb.lib().tb_gemm_w4a32_grouped(x.data_ptr(), a[0].data_ptr(), a[1].data_ptr(), None, y.data_ptr(), m, n, k, g, st)
        assert rc == 0, tb.last_error()
        return y
    streamed = run()
    try:
        tb.lib().tb_set_gemv_tuning(3, 0, 0)
        integer = run()
    finally:
        tb.lib().tb_set_gemv_tuning(1, 0, 0)
    assert not torch.equal(integer, streamed)
    top = x.double().abs().reshape(m, k // 32, 32).amax(-1, keepdim=True).expand(m, k // 32, 32).reshape(m, k)

    def sums(w):
        d = (4.4 + k / 32 + 10) * 2.0 ** -24 * (x.double().abs() @ w.abs().T)
        return x.double() @ w.T, d + 2.0 ** -23 * (top @ w.abs().T)
    (want, d), (up, du) = sums(a[2]), sums(b[2])
    if pair:
        silu = torch.nn.functional.silu(want)
        d = 1.1 * d * (up.abs() + du) + silu.abs() * du + 4 * 2.0 ** -23 * (silu * up).abs()
        want = silu * up
    for y in (streamed, integer):
        assert bool(((y.double() - want).abs() <= d + 1e-30).all())
    assert tb.lib().tb_device_fault_flag() == 0


@pytest.mark.parametrize("m,k", [(5, 288), (8, 4608)])
def test_rows_at_both_ends_of_fp32(torch, tb, m, k):
    """Zeros, numbers of 1e-35 and 1e33 beside ordinary rows, a denormal."""
    n, g = 96, 32
    p, s, w = int4(torch, n, k, g, 5)
    x = torch.randn(m, k, device="cuda", generator=torch.Generator("cuda").manual_seed(6))
    x[0] = 0
    x[1] *= 1e-35
    x[2] *= 1e33
    x[3] = 0
    x[3, k - 50] = 2.5e-39
    got, want = tb.w4a32_grouped_linear(x, p, s, None, g), x.double() @ w.T
    bound = (4.4 + k / 32 + 10) * 2.0 ** -24 * (x.double().abs() @ w.abs().T)
    assert not got[0].any()
    for i in (1, 2, 4, m - 1):
        # a piece below the smallest normal number may come out as zero: k of them, 2^-126 each, times codes of up to 8 and a scale
        assert bool(((got[i].double() - want[i]).abs() <= bound[i] + k * 2.0 ** -126 * 8 * float(s.max())).all()), i
    assert float((got[3].double() - want[3]).abs().max()) < 2e-39   # denormal sums may come out as zeros


@pytest.mark.parametrize("rows", [2, 3, 5, 8])
@pytest.mark.parametrize("hidden,heads,kv,dim,inter", [(896, 14, 7, 64, 640), (4608, 72, 36, 64, 256)])
def test_the_norm_in_front_of_few_rows(torch, tb, rows, hidden, heads, kv, dim, inter):
    """A decoder of one layer at position 0, where attention gives every head its key head's value, against float64.  The pre-pass takes the norm
    of a row in one block of the grid and, beyond 4096, in several.  1e-5: the layers' fp32 sums of random terms, a few 1e-7 each."""
    def norm(i):
        return torch.randn(hidden, device="cuda", generator=torch.Generator("cuda").manual_seed(i)) * 0.1 + 1
    vocab, q = 300, heads * dim
    qkv, o = int4(torch, q + 2 * kv * dim, hidden, 32, 1), int4(torch, hidden, q, 32, 2)
    gate, up, down, head = int4(torch, inter, hidden, 32, 3), int4(torch, inter, hidden, 32, 4), int4(torch, hidden, inter, 32, 5), int4(torch, vocab, hidden, 32, 6)
    embed = torch.randn(vocab, hidden, device="cuda", generator=torch.Generator("cuda").manual_seed(7))
    n1, n2, n3 = norm(8), norm(9), norm(10)
    dec = tb.B200QwenDecoder(embed, [[n1, *qkv[:2], *o[:2], n2, *gate[:2], *up[:2], *down[:2], None]], n3, *head[:2], 1, hidden, inter, heads, kv, dim, 32,
                             1e-6, 16, 10000.0, max_batch=8)
    ids = [(37 * i + 5) % vocab for i in range(rows)]
    got = torch.as_tensor(dec.step_batch(ids, [0] * rows)).cuda().double()

    def rms(x, w):
        return x / (x.square().mean(-1, keepdim=True) + 1e-6).sqrt() * w.double()
    x = embed[ids].double()
    v = (rms(x, n1) @ qkv[2].T)[:, q + kv * dim:].view(rows, kv, 1, dim).expand(rows, kv, heads // kv, dim).reshape(rows, q)
    x = x + v @ o[2].T
    h = rms(x, n2)
    x = x + (torch.nn.functional.silu(h @ gate[2].T) * (h @ up[2].T)) @ down[2].T
    want = rms(x, n3) @ head[2].T
    assert float((got - want).norm() / want.norm()) < 1e-5
