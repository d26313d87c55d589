"""Gate/up pairs on the tcgen05 kernel whose CTAs take ranges of K that begin and end inside a tile: the last CTA of a tile adds
the parts of both matrices before the SwiGLU.

Per sum |error| <= d = (52 + K / g) 2^-24 A with A = sum |x| |w| + |bias| (as for single products, and one rounding for each of up to
eight parts).  silu has a slope of at most 1.1, so |error| <= 1.1 dg (|up| + du) + |silu| du + 8 roundings of the result."""
import pytest

from test_gpu_portions import int4, tb, torch  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,g", [
    (16, 14336, 4096, 32), (17, 1501, 4096, 32), (33, 130, 20480, 64), (40, 2050, 1280, 128), (100, 14336, 4096, 32), (129, 3000, 4096, 64), (200, 6146, 2048, 128),
    (333, 700, 14336, 32), (512, 1152, 8192, 64), (20, 1, 16384, 32)])
def test_pairs_in_ranges(torch, tb, m, n, k, g):  # noqa: F811
    a, b = int4(torch, n, k, g, m + n), int4(torch, n, k, g, k)
    gen = torch.Generator("cuda").manual_seed(m)
    x = torch.randn(m, k, device="cuda", generator=gen)
    bias = torch.randn(2, (n + 3) // 4 * 4, device="cuda", generator=gen)
    st = torch.cuda.current_stream().cuda_stream
    for b0, b1 in ((None, None), (bias[0, :n], bias[1, :n])):
        ptr = [None if t is None else t.data_ptr() for t in (b0, b1)]
        add = [0.0 if t is None else t.double() for t in (b0, b1)]
        sums = [x.double() @ w[2].T + v for w, v in zip((a, b), add)]
        d = [(52 + k // g) * 2.0 ** -24 * (x.double().abs() @ w[2].abs().T + abs(v)) for w, v in zip((a, b), add)]
        want = torch.nn.functional.silu(sums[0]) * sums[1]
        bound = 1.1 * d[0] * (sums[1].abs() + d[1]) + torch.nn.functional.silu(sums[0]).abs() * d[1] + 2.0 ** -21 * want.abs()
        first = None
        for _ in range(3):
            out = torch.full((m, n), float("nan"), device="cuda")
            assert tb.lib().tb_swiglu_gemv_w4a32(x.data_ptr(), a[0].data_ptr(), a[1].data_ptr(), ptr[0], b[0].data_ptr(), b[1].data_ptr(), ptr[1],
                                                 out.data_ptr(), m, n, k, g, st) == 0, tb.last_error()
            assert bool(((out.double() - want).abs() <= bound).all())
            assert first is None or torch.equal(out, first)
            first = out
    assert tb.lib().tb_device_fault_flag() == 0
