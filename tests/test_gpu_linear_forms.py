"""The forms that a call of the INT4 linear may take: operands that need no conversion take a short way through it."""
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


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("shape", [(256,), (1, 256), (3, 256), (2, 3, 256), (2, 1, 1, 256)])
@pytest.mark.parametrize("form", ["plain", "strided", "transposed", "bfloat16", "double", "parameter", "sliced weights"])
def test_every_form_of_a_call_gives_the_same(torch, tb, shape, bias, form):
    """Operands that need no conversion take a short way; it gives what the general way gives for the same numbers."""
    class Other(torch.Tensor):   # takes the general way
        pass
    n, k, g = 70, 256, 32
    p, s, _ = int4(torch, n, k, g, 3)
    x = torch.randn(*shape, device="cuda")
    b = torch.randn(n, device="cuda") if bias else None
    want = tb.w4a32_grouped_linear(x.as_subclass(Other), p, s, b, g).as_subclass(torch.Tensor)
    if form == "strided":
        x = torch.stack([x, -x], -1)[..., 0]
    elif form == "transposed":
        x = x.reshape(-1, k).T.contiguous().T.reshape(shape) if len(shape) == 1 else x.reshape(-1, k).T.contiguous().T.unflatten(0, shape[:-1])
    elif form in ("bfloat16", "double"):
        x = x.to(getattr(torch, form))
        want = tb.w4a32_grouped_linear(x.float().as_subclass(Other), p, s, b, g).as_subclass(torch.Tensor)
    elif form == "parameter":
        x = torch.nn.Parameter(x)
    elif form == "sliced weights":
        p, s = torch.stack([p, p], 1)[:, 0], torch.stack([s, s], -1)[..., 0]
    y = tb.w4a32_grouped_linear(x, p, s, b, g)
    assert y.shape == (*shape[:-1], n) and y.dtype == torch.float32 and not y.requires_grad and torch.equal(y, want)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        y = tb.w4a32_grouped_linear(x, p, s, b, g)
    side.synchronize()
    assert torch.equal(y, want)


def test_refused_calls_stay_refused(torch, tb):
    p, s, _ = int4(torch, 64, 256, 32, 4)
    x, b = torch.randn(2, 256, device="cuda"), torch.randn(63, device="cuda")
    for args in [(x[:, :128].contiguous(), p, s, None, 32), (x, p, s[:, :4].contiguous(), None, 32), (x, p, s, b, 32), (x, p.to(torch.int8), s, None, 32),
                 (x, p.reshape(-1), s, None, 32), (x, p, s, None, 64), (x, p.cpu()[:32], s, None, 32), (x, p, torch.randn(64, 32, device="cuda"), None, 8)]:
        with pytest.raises((tb.TorchBurnB200Error, ValueError)):
            tb.w4a32_grouped_linear(*args)
