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
