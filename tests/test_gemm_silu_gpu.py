"""SiLU(gate) * up in the tensor-core GEMM's epilogue against the product followed by the activation kernel."""

import pytest
import torch

from fdk import models, native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("m,n,k", [(17, 64, 192), (33, 192, 64), (200, 640, 1088), (40, 64 * 7, 64 * 60), (300, 128 * 9, 512)])
def test_equals_two_steps(bits, m, n, k):
    """One 64-row tile, odd numbers of them, cut tiles, several batch tiles: the same bits."""
    gen = torch.Generator(device="cuda").manual_seed(m + n + k + bits)
    weight = (torch.randn((n, k), generator=gen, device="cuda") * (4 / k**0.5)).bfloat16()
    layer = models.QuantisedLinear.create(weight, models.QuantisationConfig(bits, 64))
    x = torch.randn((m, k), generator=gen, device="cuda").bfloat16()
    want = torch.empty((m, n // 2), device="cuda", dtype=torch.bfloat16)
    native.silu_mul(layer(x), want, group=32)
    for _ in range(3):
        got = torch.full_like(want, float("nan"))
        layer.forward_silu_pairs(x, got)
        assert torch.equal(got, want)
    assert native.device_status() == 0


def test_refusals():
    layer = models.QuantisedLinear.create(torch.randn((128, 64), device="cuda").bfloat16(), models.QuantisationConfig(4, 64))
    x, out = torch.randn((20, 64), device="cuda").bfloat16(), torch.empty((20, 64), device="cuda", dtype=torch.bfloat16)
    ws = native.workspace(x.device)

    def call(n=128, x_ptr=x.data_ptr(), size=ws.numel(), flags=0):
        return native.lib().fdk_linear_lut_silu(x_ptr, layer.tiled().data_ptr(), layer.lut.data_ptr(), None, out.data_ptr(), 20, n, 64, 4,
                                                ws.data_ptr(), size, flags, native._stream())

    assert call() == 0
    assert call(n=100) == 2 and call(x_ptr=x.data_ptr() + 2) == 3 and call(size=100) == 6 and call(flags=2) == 1
    torch.cuda.synchronize()
