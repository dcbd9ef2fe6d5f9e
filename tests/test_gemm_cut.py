"""The tensor-core GEMM's cut of its unit sequence (csrc/gemm_cut.cuh), compiled for the host: every range begins at
floor(units * rank / ranges).  The places of the cuts order the fp32 partial sums, so results keep their bits only
while the cuts stay where they are."""

import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "fused-dequantisation-kernels_b200" / "csrc"

SOURCE = """
#include "gemm_cut.cuh"
extern "C" int wrong(int units, int ranges) {  // ranks whose range begins elsewhere
  const fdk::TcCut cut = fdk::make_tc_cut(units, ranges);
  int bad = 0;
  for (int rank = 0; rank <= ranges; ++rank) bad += fdk::tc_cut_begin(cut, rank) != (int)((long long)units * rank / ranges);
  return bad;
}
"""


@pytest.fixture(scope="module")
def wrong(tmp_path_factory):
    compiler = shutil.which("g++") or shutil.which("c++")
    if compiler is None:
        pytest.skip("no host compiler")
    folder = tmp_path_factory.mktemp("cut")
    (folder / "cut.cpp").write_text(SOURCE)
    subprocess.run([compiler, "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(folder / "cut.cpp"), "-o", str(folder / "cut.so")], check=True)
    return ctypes.CDLL(str(folder / "cut.so")).wrong


@pytest.mark.parametrize("ranges", [1, 2, 3, 37, 127, 128, 147, 148, 160, 255, 256])
def test_ranges_begin_at_the_floor_of_their_share(wrong, ranges):
    for units in [*range(1, 3 * ranges + 2), *(5120 * ranges + d for d in (-1, 0, 1)), 2**30 - 1, 2**30]:
        assert wrong(units, ranges) == 0


def test_the_kernel_cuts_there():
    kernel = (CSRC / "gemm_lut_tc.cu").read_text()
    assert "tc_cut_begin(p.cut, rank)" in kernel and "make_tc_cut((int)(p.split ? units : tiles), grid)" in kernel
