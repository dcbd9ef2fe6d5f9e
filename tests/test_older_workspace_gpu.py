"""Workspaces of the size from before the kernel for batches that share x had sums of its own there: fdk_linear_lut and the
fused entry points then run the GEMV kernel for all of 1 to 16 rows, every width and output."""

import ctypes

import pytest
import torch

import test_fusion_gpu as fusion
import test_kernels_gpu as kernels
import test_skinny_gpu as skinny
import test_tp_push_gpu as push

pytestmark = pytest.mark.gpu

SKINNY_BYTES = 160 * 128 * 16 * 8  # 128 rows x 16 tagged words for each of up to 160 multiprocessors, at the end of a workspace


@pytest.fixture
def native(monkeypatch):
    from fdk import native as nat

    size = ctypes.c_size_t(0)
    nat.check(nat.lib().fdk_workspace_size(ctypes.byref(size)))
    older = torch.empty(size.value - SKINNY_BYTES, dtype=torch.uint8, device="cuda")
    nat.check(nat.lib().fdk_workspace_init(older.data_ptr(), older.numel(), nat._stream()))
    monkeypatch.setattr(nat, "workspace", lambda device: older)
    yield nat
    torch.cuda.synchronize()


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("m", [1, 3, 5, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(64, 64), (200, 64 * 5), (1024, 768), (64 * 2, 64 * 150)])
def test_plain(native, bits, m, n, k):
    kernels.test_linear_lut_matches_oracle(native, bits, m, n, k)
    assert native.device_status() == 0


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("m,n,k", skinny.FUSED_SIZES)
def test_residual_and_norm_outputs(native, bits, m, n, k):
    skinny.test_residual_and_norm_outputs(native, bits, m, n, k)


@pytest.mark.parametrize("bits", [1, 2, 3, 8])
@pytest.mark.parametrize("m,q_heads,kv_heads,k", [(5, 3, 1, 64 * 33), (12, 2, 1, 64 * 9)])
def test_rotary_output(native, bits, m, q_heads, kv_heads, k):
    skinny.test_rotary_output(native, bits, m, q_heads, kv_heads, k)


@pytest.mark.parametrize("bits,m,n,k,tp", [(4, 5, 1024, 640, 3), (4, 16, 1024, 256, 2), (1, 3, 512, 1024, 2), (3, 9, 512, 512, 2), (8, 8, 512, 192, 2)])
def test_push(native, bits, m, n, k, tp):
    push.test_push_then_reduce_equals_plain_path(native, bits, m, n, k, tp)


# both sides of every line between the kernels: columns, weights of a multiprocessor (64, 128 and 300 K on 148 of them), rows
LINES = [(1, 192, 4032), (1, 192, 4096), (1, 2304, 4096), (2, 2432, 4096), (1, 4672, 4096), (2, 4800, 4096), (1, 5504, 8192), (2, 5568, 8192),
         (3, 4672, 4096), (4, 4800, 4096), (4, 320, 4032), (5, 4800, 4096)]


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("m,n,k", LINES)
def test_both_kernels_agree_at_the_lines(native, monkeypatch, bits, m, n, k):
    """Whichever kernel a workspace of today's size leads to, and the one that an older size leads to: sums of the same fp32
    products in another order, so outputs differ where a rounding to bf16 falls the other way, by one of its units."""
    gen = torch.Generator(device="cuda").manual_seed(n + k + bits)
    codes = torch.randint(0, 256, (n, k * bits // 8), generator=gen, dtype=torch.uint8, device="cuda")
    scale = (torch.rand((n, k // 64), generator=gen, device="cuda") * 2 * k**-0.5).bfloat16()
    lut = torch.randn((8, 1) if bits == 3 else (256, 8 // bits), generator=gen, device="cuda").bfloat16()
    x = torch.randn((m, k), generator=gen, device="cuda").bfloat16()
    tiled = native.repack(codes, scale, n, k, bits, 64)
    size = ctypes.c_size_t(0)
    native.check(native.lib().fdk_workspace_size(ctypes.byref(size)))
    today = torch.empty(size.value, dtype=torch.uint8, device="cuda")
    native.check(native.lib().fdk_workspace_init(today.data_ptr(), today.numel(), native._stream()))
    outs = []
    for workspace in (native.workspace(x.device), today):
        monkeypatch.setattr(native, "workspace", lambda device, _w=workspace: _w)
        out = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
        native.linear_lut(x, tiled, lut, out, n, k, bits)
        assert native.device_status() == 0
        outs.append(out.double())
    unit = 2.0**-7 * torch.maximum(*[o.abs() for o in outs])  # of bf16, at most
    error = 2.0**-24 * k**0.5 * 64 * outs[1].abs().max()      # of fp32 sums of k products, with room, where they cancel
    assert bool(((outs[0] - outs[1]).abs() <= unit + error).all())
    assert ((outs[0] - outs[1]).norm() / outs[1].norm()).item() < 2.0**-11  # and few do
