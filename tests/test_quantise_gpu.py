"""The quantiser kernel against the sequence of torch operations that defines it, byte for byte."""

import pytest
import torch

from fdk import models, native

pytestmark = pytest.mark.gpu


def by_torch(weight, config, lut):
    """`QuantisedLinear.create` of the same weight without the kernel: in 16 bits, on the same GPU."""
    can, native.can_quantise = native.can_quantise, lambda *a: False
    try:
        return models.QuantisedLinear.create(weight, config, lut=lut)
    finally:
        native.can_quantise = can


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("n,k,block", [(1, 64, 64), (5, 192, 64), (64, 8, 8), (3, 1024, 256), (300, 640, 32), (513, 2048, 128)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_create_bytes_equal_torch(bits, n, k, block, dtype):
    gen = torch.Generator(device="cuda").manual_seed(n + k + bits)
    w = (torch.randn((n, k), generator=gen, device="cuda") * k**-0.5).to(dtype)
    w.view(-1)[:: 97] = 0.0
    w[-1, : block] = 0.0  # a block of zeros: its scale is the lower limit
    short = torch.sort(torch.randn(max(2, 2**bits - 1), generator=gen, device="cuda"))[0].to(dtype)  # one entry short from 2 bits on
    for lut in (None, models.kmeans_like_codebook(bits).to("cuda", dtype) if bits < 8 else None, short, short.flip(0)):
        config = models.QuantisationConfig(bits, block)
        assert native.can_quantise(w, bits, block, short)
        got, want = models.QuantisedLinear.create(w, config, lut=lut), by_torch(w, config, lut)
        assert torch.equal(got.weight_data, want.weight_data)
        assert torch.equal(got.scale.view(torch.int16), want.scale.view(torch.int16))
        assert torch.equal(got.lut.view(torch.int16), want.lut.view(torch.int16))
        assert got.lut.shape == want.lut.shape and got.scale.shape == want.scale.shape


@pytest.mark.parametrize("bits,block", [(3, 64), (4, 128), (4, 32), (8, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_large_matrices_equal_torch(bits, block, dtype):
    """Sizes that look codes up in a table (4 M weights on, from 3 bits on), with every pattern among the weights,
    codebooks in no order among them."""
    n, k = 2101, 2048
    gen = torch.Generator(device="cuda").manual_seed(bits + block)
    w = (torch.randn((n, k), generator=gen, device="cuda") * k**-0.5).to(dtype)
    patterns = torch.arange(65536, device="cuda", dtype=torch.int32).to(torch.int16).view(dtype)
    w.view(-1)[-65536:] = torch.where(patterns.isfinite(), patterns, torch.zeros_like(patterns))
    w[0, :7] = float("nan")
    w[1, :7] = float("inf")
    for lut in (torch.linspace(-1, 1, 2**bits, device="cuda").to(dtype), torch.randn(2**bits, generator=gen, device="cuda").to(dtype)):
        config = models.QuantisationConfig(bits, block)
        got, want = models.QuantisedLinear.create(w, config, lut=lut), by_torch(w, config, lut)
        assert torch.equal(got.weight_data, want.weight_data)
        assert torch.equal(got.scale.isnan(), want.scale.isnan())
        assert torch.equal(got.scale.nan_to_num(), want.scale.nan_to_num())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_every_quotient_class(dtype):
    """All 16-bit patterns as weights (subnormals, infinities and NaN among them), in blocks whose scales
    span the type's range: the reciprocal form of the quotient and the division agree."""
    patterns = torch.arange(65536, device="cuda", dtype=torch.int32).to(torch.int16).view(dtype)
    gen = torch.Generator(device="cuda").manual_seed(0)
    w = torch.cat([patterns.view(-1, 64), patterns[torch.randperm(65536, generator=gen, device="cuda")].view(-1, 64)])
    w = torch.cat([w, torch.where(w.isfinite(), w, torch.zeros_like(w))])
    config = models.QuantisationConfig(8, 64)
    got, want = models.QuantisedLinear.create(w, config), by_torch(w, config, None)
    assert torch.equal(got.weight_data, want.weight_data)
    assert torch.equal(got.scale.isnan(), want.scale.isnan())
    assert torch.equal(got.scale.nan_to_num(), want.scale.nan_to_num())


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_zeros_beside_small_weights(bits, dtype):
    """Zeros need no division, the smallest values beside them do: every share of zeros in octets whose other weights make
    quotients of all sizes, subnormal ones and such as vanish among them; codebooks with a midpoint at zero and beside it."""
    gen = torch.Generator(device="cuda").manual_seed(bits)
    n, k = 520, 1024
    size = 2.0 ** torch.randint(-140 if dtype == torch.bfloat16 else -24, 1, (n, k), generator=gen, device="cuda").float()
    w = (torch.randn((n, k), generator=gen, device="cuda") * size).to(dtype)
    share = torch.linspace(0, 1, n, device="cuda")[:, None]
    w = torch.where(torch.rand((n, k), generator=gen, device="cuda") < share, torch.zeros_like(w), w)
    w[::2, ::3] *= -1  # negative zeros among them
    tiny = torch.linspace(-1, 1, 2**bits, device="cuda") * (2.0**-130 if dtype == torch.bfloat16 else 2.0**-22)
    for lut in (torch.linspace(-1, 1, 2**bits, device="cuda").to(dtype), tiny.to(dtype)):
        config = models.QuantisationConfig(bits, 64)
        got, want = models.QuantisedLinear.create(w, config, lut=lut), by_torch(w, config, lut)
        assert torch.equal(got.weight_data, want.weight_data)
        assert torch.equal(got.scale.view(torch.int16), want.scale.view(torch.int16))


def test_other_weights_keep_the_general_path():
    w = torch.randn((64, 128), device="cuda").bfloat16()
    lut = torch.linspace(-1, 1, 16, device="cuda", dtype=torch.bfloat16)
    assert native.can_quantise(w, 4, 64, lut)
    for bad in (w.t(), w[:, 1:65], w.float(), w.view(2, 32, 128), w[:0]):
        assert not native.can_quantise(bad, 4, 64, lut)
    assert not native.can_quantise(w, 4, 48, lut) and not native.can_quantise(w, 5, 64, lut)
    t = models.QuantisedLinear.create(w.t().contiguous().t(), models.QuantisationConfig(4, 64))
    assert torch.equal(t.weight_data, models.QuantisedLinear.create(w, models.QuantisationConfig(4, 64)).weight_data)
