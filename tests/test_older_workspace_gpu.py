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
