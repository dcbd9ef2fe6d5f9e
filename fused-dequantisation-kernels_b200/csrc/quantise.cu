// Quantiser: dense 16-bit weight -> packed codes, block scales, byte table, in one pass; the same
// bytes as the sequence of framework operations it stands for (src/fdk/models.py:63-104):
//   scale  = max(absmax or mean of the block, 1e-12), rounded to the weight's type
//   scaled = round16(round32(w / scale))
//   code   = lower bound of scaled among the codebook's midpoints round16(round16(a + b) / 2)
// Bound by instruction issue (2 bytes a weight read and bits / 8 written would take 13 us at 11264 x 3072), so
// everything after the quotient works on pairs of 16-bit values: rounding, the test for quotients that
// need a division, the search (whose first four steps choose among midpoints in registers by mask), packing.  A
// lane holds octets of eight consecutive weights, neighbouring lanes neighbouring octets, so loads and
// stores of a warp are contiguous and a scale block is a group of 2 to 32 lanes; kQuantBatch
// octets per lane are loaded before the first is coded.
// From 3 bits on large matrices look the code of each 16-bit quotient up in a table of 65536 bytes (random bytes meet in
// about 3.4 of 32 banks), so the steps of the search are paid per CTA.  us at 11264 x 3072, with one weight at a time and
// every step of the search in shared memory / in pairs / with the table: 8 bits 152 / 93 / 38, 4 bits 64 / 46 / 34.5, 3 bits
// 56 / 38 / 34, 2 bits 40 / 29, 1 bit 33 / 25.
#include <type_traits>

#include "fdk_common.cuh"

namespace fdk {
namespace {

template <bool TABLE>
constexpr int kQuantThreads = TABLE ? 1024 : 256;
constexpr int kQuantBatch = 4;
constexpr long long kTableOctets = 1 << 19;  // 4 M weights: below, a launch takes little longer than its host call either way

// round16(round32(a / s)) by a * (1 / s).  That product is within 3 units in the last place of the
// rounded quotient (two roundings of half a unit each, on a relative scale of up to two units,
// against the quotient's own half): unless that window holds a rounding boundary of the 16-bit
// type, both round to the same 16-bit value.  Near a boundary, for quotients that are subnormal in
// the 16-bit type (their boundaries lie elsewhere) and for scales whose reciprocal loses
// precision, the quotient is computed by division.
template <bool FP16>
struct Quotient {
  static constexpr uint32_t kTie = FP16 ? 0x1000u : 0x8000u;  // half a unit of the 16-bit type, in units of the fp32
  static constexpr uint32_t kLow = 2 * kTie - 1;
  static constexpr float kSmall = FP16 ? 6.2e-5f : 1e-30f;
  static __device__ __forceinline__ uint16_t exact(float a, float s, float r, bool exact_r) {  // one, whatever it is
    float q = a * r;
    const bool near = ((__float_as_uint(q) & kLow) - (kTie - 8u)) <= 16u;
    if (near || !exact_r || (fabsf(q) < kSmall && a != 0.0f)) q = __fdiv_rn(a, s);
    return from_float<FP16>(q);
  }
};

// Two 16-bit values at a time.
template <bool FP16>
__device__ __forceinline__ uint32_t round_pair(float lo, float hi) {
  uint32_t d;
  if constexpr (FP16) asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  else asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
template <bool FP16>
__device__ __forceinline__ uint32_t max_nan_pair(uint32_t a, uint32_t b) {  // a NaN if either is, as the framework's amax
  uint32_t d;
  if constexpr (FP16) asm("max.NaN.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  else asm("max.NaN.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// 0xFFFF where !(m >= x): m < x, or either is a NaN
template <bool FP16>
__device__ __forceinline__ uint32_t below_pair(uint32_t m, uint32_t x) {
  uint32_t d;
  if constexpr (FP16) {
    d = __hltu2_mask(*reinterpret_cast<const __half2*>(&m), *reinterpret_cast<const __half2*>(&x));
  } else {
    d = __hltu2_mask(*reinterpret_cast<const __nv_bfloat162*>(&m), *reinterpret_cast<const __nv_bfloat162*>(&x));
  }
  return d;
}
__device__ __forceinline__ uint32_t min_u16_pair(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("min.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t add_u16_pair(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("add.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// GROUP: log2 of the octets per scale block where it is 3 or 4 (blocks of 64 and 128), 0: group_log2.
// TABLE: the code of every 16-bit quotient is looked up in a table of bytes, made by the CTA (one per SM) before it
// begins (1.7 us); without it each is searched for.
template <int BITS, bool FP16, int GROUP, bool TABLE>
__global__ void __launch_bounds__(kQuantThreads<TABLE>, TABLE ? 1 : 4)
    quantise_kernel(const uint4* __restrict__ w, const uint16_t* __restrict__ lut, int lut_len,
                    const uint16_t* __restrict__ scale_in, uint8_t* __restrict__ codes, uint16_t* __restrict__ scale,
                    uint16_t* __restrict__ table, long long octets, int group_log2) {
  constexpr int kThreads = kQuantThreads<TABLE>;
  constexpr int kCodes = 1 << BITS;
  constexpr int kTop = BITS < 4 ? BITS : 4;  // steps of the search over midpoints in registers
  extern __shared__ __align__(16) uint8_t code_of[];  // TABLE: a byte per 16-bit pattern
  float* const mid = reinterpret_cast<float*>(code_of + (TABLE ? 65536 : 0));  // kCodes - 1 midpoints
  auto entry = [&](int i) { return lut[i < lut_len ? i : lut_len - 1]; };  // a short codebook repeats its last value
  for (int i = threadIdx.x; i < kCodes - 1; i += kThreads) {
    const float sum = to_float<FP16>(from_float<FP16>(to_float<FP16>(entry(i + 1)) + to_float<FP16>(entry(i))));
    mid[i] = to_float<FP16>(from_float<FP16>(sum * 0.5f));
  }
  if (blockIdx.x == 0) {  // the byte table (3 bits: the codebook itself)
    constexpr int kPerByte = BITS == 3 ? 1 : 8 / BITS, kEntries = (BITS == 3 ? 8 : 256) * kPerByte;
    for (int i = threadIdx.x; i < kEntries; i += kThreads) {
      const int e = i / kPerByte, j = i % kPerByte;
      table[i] = entry(BITS == 3 ? e : (e >> (8 - BITS * (j + 1))) & (kCodes - 1));
    }
  }
  __syncthreads();
  // the search's first steps: midpoint (of 2^kTop - 1) twice in a word
  constexpr int kTopCodes = 1 << kTop, kRest = kCodes / kTopCodes;
  uint32_t top[kTopCodes - 1];
#pragma unroll
  for (int i = 0; i < kTopCodes - 1; ++i) {
    const float m = mid[(i + 1) * kRest - 1];
    top[i] = round_pair<FP16>(m, m);
  }
  // The codes of a pair: lower bounds, halving as a search over 2^BITS - 1 entries does (whatever their order); NaN is
  // above everything
  auto search = [&](uint32_t x, uint32_t (&code)[2]) {
    uint32_t mask[kTop], c = 0;
#pragma unroll
    for (int l = 0; l < kTop; ++l) {
      uint32_t node[kTopCodes / 2];
#pragma unroll
      for (int j = 0; j < (1 << l); ++j) node[j] = top[(2 * j + 1) * (kTopCodes >> (l + 1)) - 1];
#pragma unroll
      for (int k = 0; k < l; ++k)
#pragma unroll
        for (int j = 0; j < (1 << (l - 1 - k)); ++j)
          node[j] = (mask[k] & node[j + (1 << (l - 1 - k))]) | (~mask[k] & node[j]);
      mask[l] = below_pair<FP16>(node[0], x);
      c |= mask[l] & ((uint32_t)(kTopCodes >> (l + 1)) * 0x10001u);
    }
    code[0] = c & 0xFFFFu;
    code[1] = c >> 16;
    if constexpr (kRest > 1) {  // the other steps one by one
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float xf = e ? pair_hi<FP16>(x) : pair_lo<FP16>(x);
        code[e] *= kRest;
#pragma unroll
        for (int half = kRest / 2; half > 0; half /= 2)
          if (!(mid[code[e] + half - 1] >= xf)) code[e] += half;
      }
    }
  };
  if constexpr (TABLE) {
    // four patterns (of one sign) at a time: where the midpoints ascend, two ends with one code have it between them too
    bool ascending = true;
    for (int i = threadIdx.x; i < kCodes - 2; i += kThreads) ascending = ascending && mid[i] <= mid[i + 1];
    ascending = __syncthreads_and(ascending);
#pragma unroll 1
    for (uint32_t w4 = threadIdx.x; w4 < 16384u; w4 += kThreads) {
      const uint32_t p = 4 * w4;
      uint32_t ends[2], inner[2];
      search(p | ((p + 3) << 16), ends);
      inner[0] = inner[1] = ends[0];
      if (!ascending || ends[0] != ends[1]) search((p + 1) | ((p + 2) << 16), inner);
      reinterpret_cast<uint32_t*>(code_of)[w4] = ends[0] | (inner[0] << 8) | (inner[1] << 16) | (ends[1] << 24);
    }
    __syncthreads();
  }
  const int lane = threadIdx.x & 31;
  const int log2 = GROUP != 0 ? GROUP : group_log2, lanes = 1 << log2;  // lanes (octets) per scale block
  // whole warps go through the loop: the shuffles below need all lanes of a block
  const long long step = (long long)gridDim.x * kThreads * kQuantBatch;
  for (long long base = (long long)blockIdx.x * kThreads * kQuantBatch + (threadIdx.x - lane); base < octets; base += step) {
    const int left = (int)min(octets - base, (long long)(kThreads * kQuantBatch));  // octets from here on
    const uint4* const src = w + base;
    uint8_t* const dst = codes + base * BITS;
    const long long first = base >> log2;  // scale block of this warp's first octet
    uint4 v[kQuantBatch];
#pragma unroll
    for (int b = 0; b < kQuantBatch; ++b) {
      const int o = lane + b * kThreads;
      v[b] = o < left ? __ldcs(src + o) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int b = 0; b < kQuantBatch; ++b) {
      const int o = lane + b * kThreads;
      const uint32_t words[4] = {v[b].x, v[b].y, v[b].z, v[b].w};
      float s;
      if (scale_in != nullptr) {
        s = o < left ? to_float<FP16>(scale_in[first + (o >> log2)]) : 1.0f;
      } else {
        constexpr uint32_t kAbs = 0x7FFF7FFFu;
        uint32_t m = max_nan_pair<FP16>(max_nan_pair<FP16>(words[0] & kAbs, words[1] & kAbs),
                                        max_nan_pair<FP16>(words[2] & kAbs, words[3] & kAbs));
        m = max_nan_pair<FP16>(m, (m >> 16) | (m << 16));
#pragma unroll
        for (int d = 1; d < lanes; d <<= 1) m = max_nan_pair<FP16>(m, __shfl_xor_sync(0xffffffffu, m, d));
        s = pair_lo<FP16>(m);
        const uint16_t s16 = from_float<FP16>(s != s ? s : fmaxf(s, 1e-12f));
        s = to_float<FP16>(s16);
        if (o < left && (lane & (lanes - 1)) == 0) scale[first + (o >> log2)] = s16;
      }
      const float r = __frcp_rn(s);
      const bool exact_r = s < 1e30f && s > 1e-30f;
      using Q = Quotient<FP16>;
      uint32_t x[4];
      uint32_t nearest = 0xFFFFFFFFu;  // smallest distance behind the start of the window around a boundary
      float least = 1.0f;              // smallest magnitude
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float q0 = pair_lo<FP16>(words[i]) * r, q1 = pair_hi<FP16>(words[i]) * r;
        x[i] = round_pair<FP16>(q0, q1);
        uint32_t low = __byte_perm(__float_as_uint(q0), __float_as_uint(q1), 0x5410);
        if (FP16) low &= Q::kLow * 0x10001u;
        nearest = min_u16_pair(nearest, add_u16_pair(low, ((0x10000u - (Q::kTie - 8u)) & 0xFFFFu) * 0x10001u));
        least = fminf(least, fminf(fabsf(q0), fabsf(q1)));
      }
      const bool near = (nearest & 0xFFFFu) <= 16u || (nearest >> 16) <= 16u;
      if (near || least < Q::kSmall || !exact_r) {
        // Zeros are exact (pruned or padded weights: at 11264 x 3072, a tenth of them zero, 39 us at 2 bits and 43 at 4 where every
        // octet with one divided, 31 and 37 now): the smallest magnitude beside them counts, whose pattern
        // less one is the least when those of zeros wrap to the top.
        uint32_t rest = 0xFFFFFFFFu;
#pragma unroll
        for (int i = 0; i < 4; ++i) rest = min_u16_pair(rest, add_u16_pair(words[i] & 0x7FFF7FFFu, 0xFFFFFFFFu));
        const uint32_t smallest = min(rest & 0xFFFFu, rest >> 16);
        if (near || !exact_r || (smallest != 0xFFFFu && pair_lo<FP16>(smallest + 1u) * r < Q::kSmall)) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            x[i] = (uint32_t)Q::exact(pair_lo<FP16>(words[i]), s, r, exact_r) | ((uint32_t)Q::exact(pair_hi<FP16>(words[i]), s, r, exact_r) << 16);
        }
      }
      uint32_t packed[2] = {0u, 0u};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t c[2];
        if constexpr (TABLE) {
          c[0] = code_of[x[i] & 0xFFFFu];
          c[1] = code_of[x[i] >> 16];
        } else {
          search(x[i], c);
        }
        if constexpr (BITS == 8) packed[i / 2] += c[0] * (1u << (16 * (i % 2))) + c[1] * (256u << (16 * (i % 2)));
        else if constexpr (BITS == 3) packed[0] += c[0] * (1u << (21 - 6 * i)) + c[1] * (1u << (18 - 6 * i));  // 24-bit stream, first code highest
        else {  // first code of a byte in its high bits
          constexpr int kShift[4] = {8 * (0 * BITS / 4) + 8 - 2 * BITS, 8 * (BITS / 4) + 8 - 2 * BITS - 2 * BITS % 8,
                                     8 * (2 * BITS / 4) + 8 - 2 * BITS - 4 * BITS % 8, 8 * (3 * BITS / 4) + 8 - 2 * BITS - 6 * BITS % 8};
          packed[0] += c[0] * (1u << (kShift[i] + BITS)) + c[1] * (1u << kShift[i]);
        }
      }
      if (o < left) {
        uint8_t* const at = dst + o * BITS;
        if constexpr (BITS == 8) *reinterpret_cast<uint2*>(at) = make_uint2(packed[0], packed[1]);
        else if constexpr (BITS == 4) *reinterpret_cast<uint32_t*>(at) = packed[0];
        else if constexpr (BITS == 2) *reinterpret_cast<uint16_t*>(at) = (uint16_t)packed[0];
        else if constexpr (BITS == 1) *at = (uint8_t)packed[0];
        else {
          at[0] = (uint8_t)(packed[0] >> 16);
          at[1] = (uint8_t)(packed[0] >> 8);
          at[2] = (uint8_t)packed[0];
        }
      }
    }
  }
}

template <int BITS, bool FP16, bool TABLE>
int launch_quantise(const void* w, const void* lut, int lut_len, const void* scale_in, void* codes, void* scale, void* table,
                    long long octets, int group_log2, const DeviceInfo& di, cudaStream_t stream) {
  constexpr int kThreads = kQuantThreads<TABLE>;
  const long long per_cta = (long long)kThreads * kQuantBatch;
  const long long wanted = (octets + per_cta - 1) / per_cta, most = (TABLE ? 1LL : 4LL) * di.sm_count;
  auto launch = [&](auto kernel, std::atomic<bool>(&allowed)[64]) {
    if (TABLE) {
      if (int st = allow_all_smem(kernel, allowed, di)) return st;
    }
    kernel<<<(int)(wanted < most ? wanted : most), kThreads, (TABLE ? 65536 : 0) + (sizeof(float) << BITS), stream>>>(
        (const uint4*)w, (const uint16_t*)lut, lut_len, (const uint16_t*)scale_in, (uint8_t*)codes, (uint16_t*)scale,
        (uint16_t*)table, octets, group_log2);
    FDK_CUDA(cudaGetLastError());
    return FDK_OK;
  };
  static std::atomic<bool> allowed[3][64] = {};
  if (group_log2 == 3) return launch(quantise_kernel<BITS, FP16, 3, TABLE>, allowed[0]);
  if (group_log2 == 4) return launch(quantise_kernel<BITS, FP16, 4, TABLE>, allowed[1]);
  return launch(quantise_kernel<BITS, FP16, 0, TABLE>, allowed[2]);
}

// The table from 3 bits on, for matrices over which its 1.7 us are spread.
template <int BITS, bool FP16>
int choose_quantise(const void* w, const void* lut, int lut_len, const void* scale_in, void* codes, void* scale, void* table,
                    long long octets, int group_log2, cudaStream_t stream) {
  DeviceInfo di;
  if (int st = device_info(&di)) return st;
  if constexpr (BITS >= 3) {
    if (octets >= kTableOctets)
      return launch_quantise<BITS, FP16, true>(w, lut, lut_len, scale_in, codes, scale, table, octets, group_log2, di, stream);
  }
  return launch_quantise<BITS, FP16, false>(w, lut, lut_len, scale_in, codes, scale, table, octets, group_log2, di, stream);
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
    return dtype == FDK_DTYPE_F16 ? choose_quantise<B, true>(w, lut, lut_len, scale_in, codes, scale, table, octets, group_log2, st)
                                  : choose_quantise<B, false>(w, lut, lut_len, scale_in, codes, scale, table, octets, group_log2, st);
  };
  switch (bits) {
    case 1: return launch(std::integral_constant<int, 1>{});
    case 2: return launch(std::integral_constant<int, 2>{});
    case 3: return launch(std::integral_constant<int, 3>{});
    case 4: return launch(std::integral_constant<int, 4>{});
    default: return launch(std::integral_constant<int, 8>{});
  }
}
