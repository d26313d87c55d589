"""Products of one row at narrow K: K around what a CTA stages in one go (1024 with four warps, 2048 with eight) and around 32-element
blocks, rows around the choices of the launch, single matrices and gate/up pairs.

Bound per output, with A = sum |x| |w|: a 32-element block of x is rounded to multiples of 2^-22 of its maximum, half of
that an element, and sums take one fp32 rounding per block and a few at the end: below (K / 32 + 10) * 2^-24 A plus
2^-23 * sum over blocks of max |x| sum |w|."""
import pytest

from test_gpu_portions import int4, tb, torch  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,g", [(32, 32), (96, 32), (896, 32), (896, 128), (992, 32), (1024, 64), (1056, 32), (2016, 32)])
@pytest.mark.parametrize("n,pair", [(1, 0), (17, 1), (2367, 1), (2368, 1), (4864, 1), (4736, 0), (9472, 1)])
def test_products_of_one_row(torch, tb, k, g, n, pair):  # noqa: F811
    p, s, w = int4(torch, n, k, g, n + k)
    p2, s2, w2 = int4(torch, n, k, g, n + k + 1)
    x = torch.randn(1, k, device="cuda", generator=torch.Generator("cuda").manual_seed(k)) * 3
    y = torch.empty(1, n, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    top = x.double().abs().reshape(1, k // 32, 32).amax(-1, keepdim=True).expand(1, k // 32, 32).reshape(1, k)

    def bound(m):
        return (x.double().abs() @ m.abs().T) * (k / 32 + 10) * 2.0 ** -24 + (top @ m.abs().T) * 2.0 ** -23
    want, tol = x.double() @ w.T, bound(w)
    if pair:
        rc = tb.lib().tb_swiglu_gemv_w4a32(x.data_ptr(), p.data_ptr(), s.data_ptr(), None, p2.data_ptr(), s2.data_ptr(), None, y.data_ptr(), 1, n, k, g, st)
        up, sig = x.double() @ w2.T, torch.sigmoid(want)
        # silu' <= 1.1, |silu(g)| <= |g|; four roundings of the epilogue
        tol = 1.1 * tol * up.abs() + want.abs() * bound(w2) + 4 * 2.0 ** -23 * (want * sig * up).abs() + tol * 1e-6
        want = want * sig * up
    else:
        rc = tb.lib().tb_gemm_w4a32_grouped(x.data_ptr(), p.data_ptr(), s.data_ptr(), None, y.data_ptr(), 1, n, k, g, st)
    assert rc == 0, tb.last_error()
    assert bool(((y.double() - want).abs() <= tol + 1e-30).all()), float(((y.double() - want).abs() / tol).max())
