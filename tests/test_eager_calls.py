"""The native host side of eager calls (csrc/eager_calls.cpp) against the Python code it stands for: taken where it may be,
left alone everywhere else."""

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from fdk import models, native


def general(monkeypatch):
    for name in ("eager_linear", "eager_quantise", "eager_repack"):
        monkeypatch.setattr(native, name, native._nothing)


def make(dtype=torch.bfloat16, bits=4, kernel="triton", n=192, k=256):
    weight = (torch.randn((n, k), device="cuda") * k**-0.5).to(dtype)
    return models.QuantisedLinear.create(weight, models.QuantisationConfig(bits, 64, kernel=kernel))


def test_built_and_silent_about_tensors_on_the_cpu():
    from fdk import _eager

    native.lib()
    assert native.eager_linear is _eager.linear
    w, lut = torch.randn(64, 128).bfloat16(), torch.linspace(-1, 1, 16).bfloat16()
    assert native.eager_quantise(w, 4, 64, lut, None) is None
    assert native.eager_linear({}, w) is None and native.eager_linear({}, None) is None and native.eager_linear({}) is None
    assert native.eager_repack(w, w, 64, 128, 4, 64) is None


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,bits", [(torch.bfloat16, 4), (torch.float16, 8), (torch.bfloat16, 3), (torch.float16, 1)])
def test_same_results_as_the_python_code(monkeypatch, dtype, bits):
    layer = make(dtype, bits)
    x = torch.randn((5, 256), device="cuda").to(dtype)
    layer(x)  # tiles the weight, fetches the table, allocates the stream's scratch
    got = native.eager_linear(layer.__dict__, x)
    assert got is not None and got.shape == (5, 192) and got.dtype == dtype and not got.requires_grad
    wide = torch.randn((5, 512), device="cuda").to(dtype)
    forms = [x, x[None], x[:, None], wide[:, ::2], wide[:, 8:264], torch.nn.Parameter(x)]
    outs = [layer(f) for f in forms]
    dense = (torch.randn((96, 128), device="cuda")).to(dtype)
    created = [models.QuantisedLinear.create(dense, models.QuantisationConfig(bits, block)) for block in (32, 64)]
    tiled = native.repack(created[1].weight_data, created[1].scale, 96, 128, bits, 64)
    general(monkeypatch)
    assert all(torch.equal(a, layer(f)) for a, f in zip(outs, forms)) and torch.equal(got, layer(x))
    for block, one in zip((32, 64), created):
        other = models.QuantisedLinear.create(dense, models.QuantisationConfig(bits, block))
        assert all(torch.equal(a, b) for a, b in ((one.weight_data, other.weight_data), (one.scale, other.scale), (one.lut, other.lut)))
    assert torch.equal(tiled, native.repack(created[1].weight_data, created[1].scale, 96, 128, bits, 64))


@pytest.mark.gpu
def test_changes_are_seen(monkeypatch):
    layer, x = make(), torch.randn((3, 256), device="cuda").bfloat16()
    before = layer(x)
    layer.weight_data.data = layer.weight_data.data.flip(0).contiguous()
    assert native.eager_linear(layer.__dict__, x) is None  # another weight: not tiled yet
    flipped = layer(x)
    layer.scale.mul_(2)
    assert native.eager_linear(layer.__dict__, x) is None
    doubled = layer(x)
    layer.lut.mul_(0.5)
    assert native.eager_linear(layer.__dict__, x) is None
    halved = layer(x)
    assert not torch.equal(before, flipped) and torch.equal(doubled, 2 * flipped) and torch.equal(halved, flipped)
    layer.kernel = "torch.compile"
    assert native.eager_linear(layer.__dict__, x) is None
    layer.kernel = "triton"
    with torch.cuda.stream(torch.cuda.Stream()):
        assert native.eager_linear(layer.__dict__, x) is None  # no scratch on this stream yet
        assert torch.equal(layer(x), flipped) and native.eager_linear(layer.__dict__, x) is not None
        torch.cuda.current_stream().synchronize()


@pytest.mark.gpu
def test_what_is_left_to_the_python_code():
    layer, x = make(), torch.randn((3, 256), device="cuda").bfloat16()
    layer(x)

    class Watching(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class Sub(torch.Tensor):
        pass

    call = lambda t: native.eager_linear(layer.__dict__, t)  # noqa: E731
    assert call(x) is not None
    for bad in (x[0], x[None], x.float(), x.half(), x[:, :128], x[:0], x.t(), x.cpu(), x.as_subclass(Sub), None, 3):
        assert call(bad) is None
    with Watching():
        assert call(x) is None
    seen = []
    torch.func.vmap(lambda row: (seen.append(call(row)), row)[1])(x[None])
    assert seen == [None]
    with torch.inference_mode():
        assert call(x) is not None and call(x).is_inference()
    w, lut = torch.randn((64, 128), device="cuda").bfloat16(), torch.linspace(-1, 1, 16, device="cuda").bfloat16()
    quantise = native.eager_quantise
    assert quantise(w, 4, 64, lut, None) is not None
    for args in ((w.t(), 4, 64, lut), (w[:, 1:65], 4, 64, lut), (w.float(), 4, 64, lut), (w, 5, 64, lut), (w, 4, 48, lut),
                 (w, 3, 64, lut), (w[:0], 4, 64, lut), (w, 4, 64, lut.half()), (w, 4, 64, lut.clone().requires_grad_())):
        assert quantise(*args, None) is None
    assert native.device_status() == 0


@pytest.mark.parametrize("shape", [(5, 128), (2, 3, 128)])
def test_the_torch_selector_stays_traceable(shape):
    """A graph tracer cannot look into a native function, and layers of the plain-torch selector have no use for it."""
    native.lib()  # binds the native calls
    layer = models.QuantisedLinear.create(torch.randn(64, 128).bfloat16(), models.QuantisationConfig(4, 64, kernel="torch.compile"))
    x = torch.randn(shape).bfloat16()
    torch._dynamo.reset()
    assert torch.equal(torch.compile(layer, backend="eager", fullgraph=True)(x), layer(x))
