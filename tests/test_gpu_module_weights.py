"""The fused calls on modules whose weights change between calls: each call multiplies with what the module then holds.

Tolerance: three products, each of whose sums carries at most (K / 32 + 52) roundings of 2^-24 of its terms' absolute sum, about
four times its root mean square here: 2e-5 of the largest output is above that for K <= 256."""
import pytest

from test_gpu_portions import int4, tb, torch  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu

HIDDEN, INTER, G = 128, 256, 32


def module(tb, torch, n, k, seed, where):  # noqa: F811
    p, s, _ = int4(torch, n, k, G, seed)
    m = tb.QuantizedLinear(k, n, bias=True, group_size=G).requires_grad_(False)
    m.qweight.copy_(p)
    m.scales.copy_(s)
    m.bias.copy_(torch.randn(n))
    return m.to(where)


def dense(torch, m):  # noqa: F811
    q, s = m.qweight.cuda(), m.scales.cuda().double()
    codes = torch.stack([q & 15, q >> 4], -1).reshape(q.shape[0], -1).double() - 8
    return codes * s.repeat_interleave(codes.shape[1] // s.shape[1], 1), m.bias.cuda().double()


def expect(torch, x, mods):  # noqa: F811
    (g, gb), (u, ub), (d, db) = (dense(torch, m) for m in mods)
    x = x.cuda().double()
    return (torch.nn.functional.silu(x @ g.T + gb) * (x @ u.T + ub)) @ d.T + db


def same(got, want):
    return float((got.cuda().double() - want).abs().max() / want.abs().max()) < 2e-5


CHANGES = {
    "bias in place": lambda m, o: m.bias.copy_(o.bias),
    "bias through data": lambda m, o: m.bias.data.copy_(o.bias.data),
    "codes through data": lambda m, o: m.qweight.data.copy_(o.qweight),
    "scales through data": lambda m, o: m.scales.data.mul_(2),
    "codes in place": lambda m, o: m.qweight.copy_(o.qweight),
    "other tensors": lambda m, o: (setattr(m, "qweight", o.qweight.clone()), setattr(m, "scales", o.scales.clone())),
    "bias replaced": lambda m, o: setattr(m, "bias", o.bias),
    "bias storage replaced": lambda m, o: setattr(m.bias, "data", m.bias.data * 0),
}


@pytest.mark.parametrize("rows", [1, 3, 20])
@pytest.mark.parametrize("which", [0, 2])
@pytest.mark.parametrize("change", list(CHANGES))
def test_a_change_between_calls_is_seen(torch, tb, change, which, rows):  # noqa: F811
    mods = [module(tb, torch, n, k, i, "cuda") for i, (n, k) in enumerate(((INTER, HIDDEN), (INTER, HIDDEN), (HIDDEN, INTER)))]
    x = torch.randn(rows, HIDDEN, device="cuda")
    assert same(tb.fused_swiglu_mlp(x, *mods), expect(torch, x, mods))
    other = module(tb, torch, mods[which].out_features, mods[which].in_features, 9, "cuda")
    CHANGES[change](mods[which], other)
    want = expect(torch, x, mods)
    assert same(tb.fused_swiglu_mlp(x, *mods), want)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        y = tb.fused_swiglu_mlp(x, *mods)
    side.synchronize()
    assert same(y, want)


@pytest.mark.parametrize("change", ["bias in place", "codes in place", "other tensors", "bias replaced"])
def test_modules_on_the_host(torch, tb, change):  # noqa: F811
    """Copied to the device, and again when a tensor has been written to or replaced."""
    mods = [module(tb, torch, n, k, i, "cpu") for i, (n, k) in enumerate(((INTER, HIDDEN), (INTER, HIDDEN), (HIDDEN, INTER)))]
    x = torch.randn(3, HIDDEN)
    assert same(tb.fused_swiglu_mlp(x, *mods), expect(torch, x, mods))
    CHANGES[change](mods[0], module(tb, torch, INTER, HIDDEN, 9, "cpu"))
    assert same(tb.fused_swiglu_mlp(x, *mods), expect(torch, x, mods))


@pytest.mark.parametrize("form", ["codes off 16 bytes", "scales off 16 bytes", "strided", "half scales", "host scales"])
def test_weights_that_are_copied(torch, tb, form):  # noqa: F811
    """Weights that the kernels cannot read as they are give what the others give."""
    mods = [module(tb, torch, n, k, i, "cuda") for i, (n, k) in enumerate(((INTER, HIDDEN), (INTER, HIDDEN), (HIDDEN, INTER)))]

    def off(t):
        flat = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:]
        return flat.copy_(t.reshape(-1)).reshape(t.shape)
    m = mods[1]
    if form == "codes off 16 bytes":
        m.qweight = off(m.qweight)
    elif form == "scales off 16 bytes":
        m.scales = off(m.scales)
    elif form == "strided":
        m.qweight, m.scales = torch.stack([m.qweight] * 2, 1)[:, 0], torch.stack([m.scales] * 2, -1)[..., 0]
    elif form == "half scales":
        m.scales = m.scales.half()
    else:
        m.scales = m.scales.cpu()
    x = torch.randn(5, HIDDEN, device="cuda")
    assert same(tb.fused_swiglu_mlp(x, *mods), expect(torch, x, mods))
    m.bias.mul_(3)
    assert same(tb.fused_swiglu_mlp(x, *mods), expect(torch, x, mods))
