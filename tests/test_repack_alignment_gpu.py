"""Packed codes at addresses that allow no wide loads: the same bytes and values as from an aligned buffer."""

import pytest
import torch

from fdk import models, native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("offset", [1, 2, 4, 8])
@pytest.mark.parametrize("n,k", [(1, 64), (100, 576)])
def test_unaligned_codes(bits, offset, n, k):
    layer = models.QuantisedLinear.create(torch.randn((n, k), device="cuda").bfloat16(), models.QuantisationConfig(bits, 64))
    codes, scale = layer.weight_data.data, layer.scale.data
    buffer = torch.empty(codes.numel() + 16, device="cuda", dtype=torch.uint8)
    moved = buffer[offset: offset + codes.numel()].view(codes.shape)
    moved.copy_(codes)
    assert buffer.data_ptr() % 16 == 0 and moved.data_ptr() % 16 == offset
    assert torch.equal(native.repack(moved, scale, n, k, bits, 64), native.repack(codes, scale, n, k, bits, 64))
    assert torch.equal(native.dequantise(moved, layer.lut, scale, bits), native.dequantise(codes, layer.lut, scale, bits))
