"""The kernel for batches that share x (skinny_lut_kernel.cuh) at the sizes where its split can go wrong: one row tile, an odd
number of them, ragged rows, padded slabs, groups shared by many CTAs, both n-tile counts and their ends."""

import numpy as np
import pytest
import torch

import fdk_oracle as O
from gpu_util import from_bits, oracle_dense, random_problem, to_bits

pytestmark = pytest.mark.gpu

SIZES = [
    (64, 64),        # one block: most warps have nothing to do
    (200, 64 * 5),   # four tiles, the last one ragged; two padded slabs at 2 bits, one at 1 and 3
    (64 * 3, 64 * 7),    # an odd number of tiles
    (64 * 2, 64 * 150),  # one group, shared by many CTAs
    (64 * 301, 64 * 3),  # more groups than CTAs, each of one to three slabs
    (1000, 64 * 33),     # cuts inside and between groups
]


@pytest.fixture(scope="module")
def native():
    from fdk import native as n

    return n


@pytest.mark.parametrize("bits,rows", [(4, (3, 8, 9, 16)), (2, (5, 16)), (3, (1, 9)), (1, (1, 12)), (8, (2, 16))])
@pytest.mark.parametrize("n,k", SIZES)
def test_edges(native, bits, rows, n, k):
    for m in rows:
        codes, lut, scale, x = random_problem(n, k, bits, m, seed=n + k + bits + m)
        tiled = native.repack(torch.from_numpy(codes).cuda(), from_bits(scale), n, k, bits, 64)
        d_x, d_lut = from_bits(x), from_bits(lut)
        outs = []
        for _ in range(3):
            out = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
            native.linear_lut(d_x, tiled, d_lut, out, n, k, bits, pdl=True)
            outs.append(to_bits(out))
        torch.cuda.synchronize()
        want = O.mm_dense(x, oracle_dense(codes, lut, scale, bits, k))
        # one rounding of the output (2^-9 / sqrt(3) to 2^-8 / sqrt(3)) beside the reference's own of each weight
        assert O.rmsen(O.bf16_to_f32(want), O.bf16_to_f32(outs[0])) < 4e-3
        assert all(np.array_equal(o, outs[0]) for o in outs)
    assert native.device_status() == 0


@pytest.mark.parametrize("m,tiles", [(3, 3), (9, 5)])
def test_residual_output_of_an_odd_number_of_tiles(native, m, tiles):
    n, k, bits = 64 * tiles, 64 * 40, 4
    codes, lut, scale, x = random_problem(n, k, bits, m, seed=m)
    tiled = native.repack(torch.from_numpy(codes).cuda(), from_bits(scale), n, k, bits, 64)
    d_x, d_lut = from_bits(x), from_bits(lut)
    y = torch.empty((m, n), dtype=torch.bfloat16, device="cuda")
    native.linear_lut(d_x, tiled, d_lut, y, n, k, bits)
    h0 = torch.randn((m, n), device="cuda").bfloat16()
    h, sumsq = h0.clone(), torch.full((m, tiles), float("nan"), device="cuda")
    native.linear_lut_fused(d_x, tiled, d_lut, None, m, n, k, bits,
                            native.LinearFusion(resid_h=h.data_ptr(), resid_sumsq=sumsq.data_ptr()))
    torch.cuda.synchronize()
    assert torch.equal(h, h0 + y)
    # 64 squares in fp32, another order of the sum
    assert torch.allclose(sumsq, h.float().view(m, tiles, 64).pow(2).sum(-1), rtol=64 * 2.0**-24)
    assert native.device_status() == 0


# batch rows that the kernel serves at every code width and size, one n-tile and two; groups cut between CTAs, an odd number of
# tiles, a ragged last one
FUSED_SIZES = [(5, 64 * 5, 64 * 33), (8, 1000, 64 * 24), (12, 64 * 3, 64 * 21)]


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("m,n,k", FUSED_SIZES)
def test_residual_and_norm_outputs(native, bits, m, n, k):
    """Residual output with the next norm's weight, and sums multiplied by the norm's factor, against the plain product."""
    import test_fusion_gpu as fusion

    fusion.test_residual_output(native, bits, m, n, k)
    fusion.test_deferred_norm(native, bits, m, n, k, "resid")
    fusion.test_deferred_norm(native, bits, m, n // 64 * 64, k, "silu")


@pytest.mark.parametrize("bits", [1, 2, 3, 8])
@pytest.mark.parametrize("m,q_heads,kv_heads,k", [(5, 3, 1, 64 * 33), (12, 2, 1, 64 * 9)])
def test_rotary_output(native, bits, m, q_heads, kv_heads, k):
    n, max_len, at = (q_heads + 2 * kv_heads) * 128, 40, 17
    codes, lut, scale, x = random_problem(n, k, bits, m, seed=bits + m)
    tiled = native.repack(torch.from_numpy(codes).cuda(), from_bits(scale), n, k, bits, 64)
    d_x, d_lut = from_bits(x), from_bits(lut)
    pos, table = torch.tensor(at, device="cuda"), torch.zeros(64, dtype=torch.int32, device="cuda")
    native.rope_table(pos, table, 500000.0)
    qkv = torch.empty((m, n), dtype=torch.bfloat16, device="cuda")
    native.linear_lut(d_x, tiled, d_lut, qkv, n, k, bits)
    outs = []
    for fused in (False, True):
        caches = [torch.full((m, kv_heads, max_len, 128), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
        q = torch.full((m, q_heads * 128), float("nan"), device="cuda", dtype=torch.bfloat16)
        if fused:
            native.linear_lut_fused(d_x, tiled, d_lut, None, m, n, k, bits, native.LinearFusion(
                rope_pos=pos.data_ptr(), rope_table=table.data_ptr(), q_out=q.data_ptr(), k_cache=caches[0].data_ptr(),
                v_cache=caches[1].data_ptr(), q_heads=q_heads, kv_heads=kv_heads, max_len=max_len))
        else:
            native.rope_append(qkv, pos, q, *caches, q_heads, kv_heads, 500000.0, paired=True)
        outs.append((q, *caches))
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(*outs))
    assert native.device_status() == 0


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("n,k", [(64, 64), (200, 64 * 5), (64 * 3, 64 * 150), (1000, 64 * 33)])
def test_fp16_against_64_bits(native, bits, n, k):
    gen = torch.Generator(device="cuda").manual_seed(n + k + bits)
    codes = torch.randint(0, 256, (n, k * bits // 8), generator=gen, dtype=torch.uint8, device="cuda")
    book = torch.randn(2**bits, generator=gen, device="cuda").half()
    shifts = torch.arange(8 - bits, -1, -bits, device="cuda")
    lut = book[:, None].contiguous() if bits == 3 else book[(torch.arange(256, device="cuda")[:, None] >> shifts) & (2**bits - 1)].contiguous()
    scale = (torch.rand((n, k // 64), generator=gen, device="cuda") * 2 * k**-0.5).half()
    tiled = native.repack(codes, scale, n, k, bits, 64)
    values = native.dequantise(codes, lut, torch.ones_like(scale), bits).double()  # the table's, without a rounding
    w = values * scale.double().repeat_interleave(64, dim=1)
    for m in (5, 8, 9, 16):
        x = torch.randn((m, k), generator=gen, device="cuda").half()
        out = torch.full((m, n), float("nan"), dtype=torch.float16, device="cuda")
        native.linear_lut(x, tiled, lut, out, n, k, bits)
        want = x.double() @ w.T
        # one rounding to 11 bits: at most 2^-11 / sqrt(3) of a value's size, root mean square; fp32 sums of 64 to 9600
        # products beside it (their error, sqrt(k) 2^-24, is below a hundredth of that)
        assert ((out.double() - want).pow(2).mean() / want.pow(2).mean()).sqrt().item() < 1.02 * 2.0**-11 / 3**0.5
    assert native.device_status() == 0
