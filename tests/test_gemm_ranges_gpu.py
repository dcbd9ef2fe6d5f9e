"""The tensor-core GEMM where its work split can go wrong: batch sizes around the tile and stage limits, tiles
cut by many ranges, short last slabs, several shapes in turn through one workspace."""

import ctypes

import pytest
import torch

from fdk import models, native

pytestmark = pytest.mark.gpu


def problem(m, n, k, bits, dtype):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k + bits)
    w = (torch.randn((n, k), generator=gen, device="cuda") * k**-0.5).to(dtype)
    layer = models.QuantisedLinear.create(w, models.QuantisationConfig(bits, 64))
    x = torch.randn((m, k), generator=gen, device="cuda").to(dtype)
    dense = native.dequantise(layer.weight_data, layer.lut, layer.scale, bits)
    return layer, x, x.double() @ dense.double().t()


def check(y, want, dtype):
    # fp32 sums of exact products, one rounding of the result: half a unit in the last place, uniform
    # over a binade, is 2^-9 / sqrt(3) relative at most (bf16; 2^-12 / sqrt(3) fp16), plus the sums' own 1e-5
    unit = 2.0**-9 if dtype == torch.bfloat16 else 2.0**-12
    assert ((y.double() - want).norm() / want.norm()).item() < unit + 1e-5
    assert bool(y.isfinite().all())


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("m", [17, 64, 65, 128, 129, 192, 193, 256, 257, 700])
def test_batch_limits(m, bits):
    dtype = torch.float16 if m % 2 else torch.bfloat16
    n, k = (1100, 64 * 37) if m < 300 else (333, 64 * 9)  # ragged last tile, short last slab
    layer, x, want = problem(m, n, k, bits, dtype)
    check(layer(x), want, dtype)
    assert native.device_status() == 0


def test_many_ranges_and_shapes_share_a_workspace():
    """Few tiles over long rows: most CTAs hold the middle of a tile.  Every launch leaves the hand-over flags
    clear for the next one, whatever its shape, and results repeat bit for bit."""
    shapes = [(40, 64, 64 * 150, 4), (250, 130, 64 * 260, 8), (24, 5120, 3072, 4), (200, 1024, 64 * 129, 2), (600, 640, 64 * 33, 3)]
    cases = [problem(*s, torch.bfloat16) for s in shapes]
    first = [layer(x) for layer, x, _ in cases]
    for layer_x, y in list(zip(cases, first)) * 3:
        layer, x, want = layer_x
        again = layer(x)
        assert torch.equal(again, y)
        check(again, want, torch.bfloat16)
    assert native.device_status() == 0


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("m,n,k", [(17, 64, 64), (17, 100, 64 * 90), (32, 256, 64 * 320), (33, 256, 64 * 320), (32, 64 * 81, 64 * 48)])
def test_narrow_tiles(m, n, k, bits):
    """Tiles of up to 32 batch rows have a form of the kernel to themselves: one share, several, many, and the first size beyond."""
    check(m, n, k, bits)


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("m,n,k", [(17, 64, 64), (17, 100, 64 * 90), (32, 256, 64 * 320), (33, 256, 64 * 320), (32, 64 * 81, 64 * 48)])
def test_narrow_tiles(m, n, k, bits):
    """Tiles of up to 32 batch rows have a form of the kernel to themselves: one share, several, many, and the first size beyond."""
    dtype = torch.float16 if m == 17 else torch.bfloat16
    layer, x, want = problem(m, n, k, bits, dtype)
    y = layer(x)
    check(y, want, dtype)
    assert torch.equal(y, layer(x)) and native.device_status() == 0


@pytest.mark.parametrize("m,n,k", [(40, 300, 640), (300, 128, 192)])
def test_without_room_for_partial_sums(m, n, k):
    """The scratch built into the library holds none: tiles are not cut."""
    layer, x, want = problem(m, n, k, 4, torch.bfloat16)
    out = torch.full((m, n), float("nan"), device="cuda", dtype=torch.bfloat16)
    status = native.lib().fdk_linear_lut_static(
        x.data_ptr(), layer.tiled().data_ptr(), layer.lut.data_ptr(), layer.lut_bytes(), out.data_ptr(), m, n, k, 4,
        native.DTYPE_BF16, 0, native._stream())
    assert status == 0
    check(out, want, torch.bfloat16)
    word = ctypes.c_int(0)
    assert native.lib().fdk_static_status(ctypes.byref(word)) == 0 and word.value == 0


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 8])
def test_every_run_gives_the_same_bits(bits):
    """A code slot that is refilled before all its reads are done shows as a run that differs, rarely (one in
    thirty at 4 bits without the proxy fence): long ranges per CTA, many of them, the tensor pipe busy."""
    layer, x, want = problem(1000, 22528, 3072, bits, torch.bfloat16)
    first = layer(x)
    check(first, want, torch.bfloat16)
    differ = torch.zeros((), dtype=torch.int64, device="cuda")
    for _ in range(500):
        differ += (layer(x) != first).any()
    assert differ.item() == 0 and native.device_status() == 0


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("k", [64, 128, 320])
def test_long_ranges_of_short_slabs(k, bits):
    """Many tiles of one to five blocks: slabs of several blocks that hold one, segments shorter than the rings."""
    for m in (20, 128, 700):
        layer, x, want = problem(m, 30000, k, bits, torch.bfloat16)
        y = layer(x)
        check(y, want, torch.bfloat16)
        assert all(torch.equal(layer(x), y) for _ in range(5))
    assert native.device_status() == 0


def test_room_for_some_partial_sums_only():
    """A workspace for fewer CTAs than would share the tiles: they are not cut, and nothing is written behind it."""
    m, n, k = 40, 300, 640
    layer, x, want = problem(m, n, k, 4, torch.bfloat16)
    slot, partial = 48 * 128 * 4, 16384 + 160 * 1024 * 8 + 160 * 48 * 4 + 256  # 48: the batch tile
    for slots in (0, 1, 3, 160):
        size = partial + slots * slot
        buffer = torch.full((size + 4096,), 0xA5, device="cuda", dtype=torch.uint8)
        native.check(native.lib().fdk_workspace_init(buffer.data_ptr(), size, native._stream()))
        for _ in range(2):
            out = torch.full((m, n), float("nan"), device="cuda", dtype=torch.bfloat16)
            native.check(native.lib().fdk_linear_lut(
                x.data_ptr(), layer.tiled().data_ptr(), layer.lut.data_ptr(), layer.lut_bytes(), out.data_ptr(), m, n, k, 4,
                native.DTYPE_BF16, buffer.data_ptr(), size, 0, native._stream()))
            check(out, want, torch.bfloat16)
        word = ctypes.c_int(-1)
        native.check(native.lib().fdk_workspace_status(buffer.data_ptr(), ctypes.byref(word)))
        assert word.value == 0 and bool((buffer[size:] == 0xA5).all())
        used = bool((buffer[partial:size] != 0).any())
        assert used == (slots == 160)
