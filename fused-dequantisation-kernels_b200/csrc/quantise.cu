// Quantiser: dense 16-bit weight -> packed codes, block scales, byte table, in one pass; the same
// bytes as the sequence of framework operations it stands for (src/fdk/models.py:63-104):
//   scale  = max(absmax or mean of the block, 1e-12), rounded to the weight's type
//   scaled = round16(round32(w / scale))
//   code   = lower bound of scaled among the codebook's midpoints round16(round16(a + b) / 2)
// Bound by HBM (2 bytes a weight read, bits / 8 written) and, close to it, by instruction issue
// (~25 per weight at 4 bits: quotient, rounding, a search of `bits` steps).  A lane holds
// octets of eight consecutive weights, neighbouring lanes neighbouring octets, so loads and
// stores of a warp are contiguous and a scale block is a group of 2 to 32 lanes; kQuantBatch
// octets per lane are loaded before the first is coded.
// `QuantisedLinear.create` and the tiled copy, 11264 x 3072, 4 bits: 877 us as framework operations (a
// dozen passes, four of them over 32- or 64-bit intermediates), 78 us with this kernel (host-bound).
#include <type_traits>

#include "fdk_common.cuh"

namespace fdk {
namespace {

constexpr int kQuantThreads = 256;
constexpr int kQuantBatch = 4;

// round16(round32(a / s)) as a float.  a * (1 / s) is within 3 units in the last place of the
// rounded quotient (two roundings of half a unit each, on a relative scale of up to two units,
// against the quotient's own half): unless that window holds a rounding boundary of the 16-bit
// type, both round to the same 16-bit value.  Near a boundary, for quotients that are subnormal in
// the 16-bit type (their boundaries lie elsewhere) and for scales whose reciprocal loses
// precision, the quotient is computed by division.
template <bool FP16>
__device__ __forceinline__ float scaled16(float a, float s, float r, bool exact_r) {
  constexpr uint32_t kLow = FP16 ? 0x1FFFu : 0xFFFFu, kTie = FP16 ? 0x1000u : 0x8000u;
  constexpr float kSmall = FP16 ? 6.2e-5f : 1e-30f;
  float q = a * r;
  const bool near = ((__float_as_uint(q) & kLow) - (kTie - 8u)) <= 16u;
  if (near || !exact_r || (fabsf(q) < kSmall && a != 0.0f)) q = __fdiv_rn(a, s);
  return to_float<FP16>(from_float<FP16>(q));
}

// Largest magnitude, NaN if either is (as the framework's amax).
__device__ __forceinline__ float max_nan(float a, float b) { return (a > b || a != a) ? a : b; }

template <int BITS, bool FP16>
__global__ void __launch_bounds__(kQuantThreads)
    quantise_kernel(const uint4* __restrict__ w, const uint16_t* __restrict__ lut, int lut_len,
                    const uint16_t* __restrict__ scale_in, uint8_t* __restrict__ codes, uint16_t* __restrict__ scale,
                    uint16_t* __restrict__ table, long long octets, int group_log2) {
  constexpr int kCodes = 1 << BITS;
  __shared__ float mid[kCodes];  // kCodes - 1 midpoints
  auto entry = [&](int i) { return lut[i < lut_len ? i : lut_len - 1]; };  // a short codebook repeats its last value
  for (int i = threadIdx.x; i < kCodes - 1; i += kQuantThreads) {
    const float sum = to_float<FP16>(from_float<FP16>(to_float<FP16>(entry(i + 1)) + to_float<FP16>(entry(i))));
    mid[i] = to_float<FP16>(from_float<FP16>(sum * 0.5f));
  }
  if (blockIdx.x == 0) {  // the byte table (3 bits: the codebook itself)
    constexpr int kPerByte = BITS == 3 ? 1 : 8 / BITS, kEntries = (BITS == 3 ? 8 : 256) * kPerByte;
    for (int i = threadIdx.x; i < kEntries; i += kQuantThreads) {
      const int e = i / kPerByte, j = i % kPerByte;
      table[i] = entry(BITS == 3 ? e : (e >> (8 - BITS * (j + 1))) & (kCodes - 1));
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int lanes = 1 << group_log2;  // lanes (octets) per scale block
  // whole warps go through the loop: the shuffles below need all lanes of a block
  const long long step = (long long)gridDim.x * kQuantThreads * kQuantBatch;
  for (long long base = (long long)blockIdx.x * kQuantThreads * kQuantBatch + (threadIdx.x - lane); base < octets; base += step) {
    uint4 v[kQuantBatch];
#pragma unroll
    for (int b = 0; b < kQuantBatch; ++b) {
      const long long o = base + lane + b * kQuantThreads;
      v[b] = o < octets ? __ldcs(w + o) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int b = 0; b < kQuantBatch; ++b) {
      const long long o = base + lane + b * kQuantThreads;
      const uint32_t words[4] = {v[b].x, v[b].y, v[b].z, v[b].w};
      float a[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[2 * i] = pair_lo<FP16>(words[i]);
        a[2 * i + 1] = pair_hi<FP16>(words[i]);
      }
      float s;
      if (scale_in != nullptr) {
        s = o < octets ? to_float<FP16>(scale_in[o >> group_log2]) : 1.0f;
      } else {
        s = fabsf(a[0]);
#pragma unroll
        for (int i = 1; i < 8; ++i) s = max_nan(s, fabsf(a[i]));
        for (int d = 1; d < lanes; d <<= 1) s = max_nan(s, __shfl_xor_sync(0xffffffffu, s, d));
        const uint16_t s16 = from_float<FP16>(s != s ? s : fmaxf(s, 1e-12f));
        s = to_float<FP16>(s16);
        if (o < octets && (lane & (lanes - 1)) == 0) scale[o >> group_log2] = s16;
      }
      const float r = __frcp_rn(s);
      const bool exact_r = s < 1e30f && s > 1e-30f;
      uint32_t packed[2] = {0u, 0u};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float x = scaled16<FP16>(a[i], s, r, exact_r);
        // lower bound, halving as a search over 2^BITS - 1 entries does; NaN is above everything
        uint32_t c = 0;
#pragma unroll
        for (int half = kCodes / 2; half > 0; half /= 2)
          if (!(mid[c + half - 1] >= x)) c += half;
        if constexpr (BITS == 8) packed[i / 4] |= c << (8 * (i % 4));
        else if constexpr (BITS == 3) packed[0] |= c << (21 - 3 * i);  // 24-bit stream, first code highest
        else packed[0] |= c << (8 * (i * BITS / 8) + 8 - BITS - i * BITS % 8);  // first code of a byte in its high bits
      }
      if (o < octets) {
        uint8_t* dst = codes + o * BITS;
        if constexpr (BITS == 8) *reinterpret_cast<uint2*>(dst) = make_uint2(packed[0], packed[1]);
        else if constexpr (BITS == 4) *reinterpret_cast<uint32_t*>(dst) = packed[0];
        else if constexpr (BITS == 2) *reinterpret_cast<uint16_t*>(dst) = (uint16_t)packed[0];
        else if constexpr (BITS == 1) *dst = (uint8_t)packed[0];
        else {
          dst[0] = (uint8_t)(packed[0] >> 16);
          dst[1] = (uint8_t)(packed[0] >> 8);
          dst[2] = (uint8_t)packed[0];
        }
      }
    }
  }
}

template <int BITS, bool FP16>
int launch_quantise(const void* w, const void* lut, int lut_len, const void* scale_in, void* codes, void* scale, void* table,
                    long long octets, int group_log2, cudaStream_t stream) {
  DeviceInfo di;
  if (int st = device_info(&di)) return st;
  const long long per_cta = (long long)kQuantThreads * kQuantBatch;
  const long long wanted = (octets + per_cta - 1) / per_cta, most = 8LL * di.sm_count;
  quantise_kernel<BITS, FP16><<<(int)(wanted < most ? wanted : most), kQuantThreads, 0, stream>>>(
      (const uint4*)w, (const uint16_t*)lut, lut_len, (const uint16_t*)scale_in, (uint8_t*)codes, (uint16_t*)scale,
      (uint16_t*)table, octets, group_log2);
  FDK_CUDA(cudaGetLastError());
  return FDK_OK;
}

}  // namespace
}  // namespace fdk

using namespace fdk;

extern "C" int fdk_quantise(const void* w, int n, int k, int bits, int block_size, int dtype, const void* lut, int lut_len,
                            const void* scale_in, void* codes, void* scale, void* table, void* stream) {
  FDK_CHECK_ARG(n > 0 && k > 0, FDK_ERR_BAD_ARG, "n=%d, k=%d must be positive", n, k);
  FDK_CHECK_ARG(bits_supported(bits), FDK_ERR_SHAPE, "bits=%d not in {1,2,3,4,8}", bits);
  int group_log2 = 0;
  while ((8 << group_log2) < block_size && group_log2 < 5) ++group_log2;
  FDK_CHECK_ARG((8 << group_log2) == block_size && k % block_size == 0, FDK_ERR_SHAPE,
                "block_size=%d must be a power of two from 8 to 256 that divides k=%d", block_size, k);
  FDK_CHECK_ARG(w && lut && codes && table && (scale != nullptr) != (scale_in != nullptr), FDK_ERR_BAD_ARG, "null pointer");
  FDK_CHECK_ARG(lut_len >= 1 && lut_len <= (1 << bits), FDK_ERR_BAD_ARG, "codebook of %d entries", lut_len);
  FDK_CHECK_ARG(dtype == FDK_DTYPE_BF16 || dtype == FDK_DTYPE_F16, FDK_ERR_BAD_ARG, "dtype=%d", dtype);
  FDK_CHECK_ARG(((uintptr_t)w & 15) == 0 && ((uintptr_t)codes & 15) == 0 &&
                    (((uintptr_t)lut | (uintptr_t)scale | (uintptr_t)scale_in | (uintptr_t)table) & 1) == 0,
                FDK_ERR_ALIGN, "w and codes must be 16-byte aligned");
  const long long octets = (long long)n * (k / 8);
  const cudaStream_t st = (cudaStream_t)stream;
  auto launch = [&](auto bits_c) {
    constexpr int B = decltype(bits_c)::value;
    return dtype == FDK_DTYPE_F16 ? launch_quantise<B, true>(w, lut, lut_len, scale_in, codes, scale, table, octets, group_log2, st)
                                  : launch_quantise<B, false>(w, lut, lut_len, scale_in, codes, scale, table, octets, group_log2, st);
  };
  switch (bits) {
    case 1: return launch(std::integral_constant<int, 1>{});
    case 2: return launch(std::integral_constant<int, 2>{});
    case 3: return launch(std::integral_constant<int, 3>{});
    case 4: return launch(std::integral_constant<int, 4>{});
    default: return launch(std::integral_constant<int, 8>{});
  }
}
