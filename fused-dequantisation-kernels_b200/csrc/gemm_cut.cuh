// How the tensor-core GEMM cuts its sequence of units into one range per CTA.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define FDK_CUT_FN __host__ __device__ __forceinline__
#else
#define FDK_CUT_FN inline
#endif

namespace fdk {

// Range `rank` begins at floor(units * rank / ranges): the longer ranges, and with them the cuts inside tiles,
// are spread evenly.  The place of the cuts is the order in which a tile's fp32 partial sums are added,
// so it is part of the result's last bits, which bf16 activations carry through a model (the longer ranges first: the
// logits of a 32-sequence step and of a prompt 1.4 % away, relative RMS).  With the longer ranges first some
// widths happen to be cut at their tiles (4 bits, 160 rows of 5120 x 3072 13.5 us against 14.05 here, of
// 22528 x 3072 25.9 against 25.7).  As base * rank + floor(rem * rank / ranges) it needs no 64-bit
// division on the device: rem * rank < 2^16 (up to 256 ranges), for which the high word of the product with
// ceil(2^32 / ranges) is the quotient exactly.
struct TcCut {
  int base, rem;
  uint32_t magic;
};

FDK_CUT_FN int tc_cut_begin(const TcCut& c, int rank) {
#ifdef __CUDA_ARCH__
  const uint32_t extra = __umulhi((uint32_t)(c.rem * rank), c.magic);
#else
  const uint32_t extra = (uint32_t)(((uint64_t)(uint32_t)(c.rem * rank) * c.magic) >> 32);
#endif
  return c.base * rank + (int)extra;
}

inline TcCut make_tc_cut(int units, int ranges) {  // (one range: no remainder, the magic number is not needed)
  return TcCut{units / ranges, units % ranges, (uint32_t)((((uint64_t)1 << 32) + ranges - 1) / ranges)};
}

}  // namespace fdk
