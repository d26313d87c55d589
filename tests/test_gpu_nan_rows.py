"""A NaN or an infinity in an activation row reaches every output of that row and no other row, whichever kernel takes the product:
one, two, three and twelve rows on CUDA cores, streamed, on integer matrix instructions and through the step kernel."""
import numpy as np
import pytest

from test_gpu_portions import int4, tb, torch  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu


def product(torch, tb, x, a, b, g, step=False):  # noqa: F811
    (m, k), n = x.shape, a[0].shape[0]
    y = torch.zeros(m, n, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    if step:
        rc = tb.lib().tb_debug_step_gemv(x.data_ptr(), a[0].data_ptr(), a[1].data_ptr(), None, b and b[0].data_ptr(), b and b[1].data_ptr(), y.data_ptr(), n, k, g, st)
    elif b:
        rc = tb.lib().tb_swiglu_gemv_w4a32(x.data_ptr(), a[0].data_ptr(), a[1].data_ptr(), None, b[0].data_ptr(), b[1].data_ptr(), None, y.data_ptr(), m, n, k, g, st)
    else:
        rc = tb.lib().tb_gemm_w4a32_grouped(x.data_ptr(), a[0].data_ptr(), a[1].data_ptr(), None, y.data_ptr(), m, n, k, g, st)
    assert rc == 0, tb.last_error()
    return y


@pytest.mark.parametrize("pair", [0, 1])
@pytest.mark.parametrize("m,k,step", [(1, 96, 0), (1, 896, 0), (1, 1184, 0), (1, 2080, 0), (1, 4096, 0), (1, 8192, 0), (1, 2048, 1), (2, 896, 0), (2, 2048, 0), (2, 4096, 0),
                                      (3, 896, 0), (5, 896, 0), (12, 896, 0), (12, 1024, 0)])
@pytest.mark.parametrize("value", ["nan", "inf", "-inf"])
def test_products(torch, tb, m, k, step, pair, value):  # noqa: F811
    n, g = 96, 32
    a, b = int4(torch, n, k, g, 1), int4(torch, n, k, g, 2) if pair else None
    x = torch.randn(m, k, device="cuda", generator=torch.Generator("cuda").manual_seed(k + m))
    want = product(torch, tb, x, a, b, g, step)
    bad = m - 1
    for at in (0, 13, 31, k - 32, k - 1):
        y = x.clone()
        y[bad, at] = float(value)
        got = product(torch, tb, y, a, b, g, step)
        assert torch.equal(got[:bad], want[:bad])
        if pair and value != "nan":
            continue   # silu of -inf is 0: what an infinity gives depends on the codes it meets
        assert not bool(torch.isfinite(got[bad]).any()) if value != "nan" else bool(torch.isnan(got[bad]).all()), at
    assert tb.lib().tb_device_fault_flag() == 0


@pytest.mark.parametrize("hidden,fused", [(64, None), (896, None), (2048, None), (2048, True)])
def test_norm_in_front_of_a_product(torch, tb, hidden, fused):  # noqa: F811
    """A token whose embedding holds a NaN: logits of NaN, not the zeros of a row of zeros; the sequences beside it are as without it."""
    gen = torch.Generator("cuda").manual_seed(hidden)
    heads, dim, inter, vocab = hidden // 64, 64, 256, 96
    kv = max(1, heads // 2)
    ones = torch.ones(hidden, device="cuda")
    q = int4(torch, (heads + 2 * kv) * dim, hidden, 32, 1)[:2]
    o = int4(torch, hidden, heads * dim, 32, 2)[:2]
    gate, up, down = int4(torch, inter, hidden, 32, 3)[:2], int4(torch, inter, hidden, 32, 4)[:2], int4(torch, hidden, inter, 32, 5)[:2]
    layer = [ones, *q, *o, ones, *gate, *up, *down, None]
    embed = torch.randn(vocab, hidden, device="cuda", generator=gen) * 0.02
    embed[7, hidden - 3] = float("nan")
    dec = tb.B200QwenDecoder(embed, [layer], ones, *int4(torch, vocab, hidden, 32, 6)[:2], 1, hidden, inter, heads, kv, dim, 32, 1e-6, 64, 10000.0, max_batch=3, fused_step=fused)
    assert np.isfinite(dec.step(5, 0)).all()
    assert np.isnan(dec.step(7, 1)).all()
    dec.reset_kv_cache()
    for ids in ([5, 7], [5, 7, 9]):
        rows = np.asarray(dec.step_batch(ids, [0] * len(ids)))
        assert np.isnan(rows[1]).all() and np.isfinite(rows[[i for i in range(len(ids)) if i != 1]]).all()
    assert tb.lib().tb_device_fault_flag() == 0
