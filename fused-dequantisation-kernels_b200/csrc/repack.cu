// Offline repacker between the reference's packed tensors and the tiled buffer,
// plus the bit-exact dequantisers.
#include <type_traits>

#include "fdk_common.cuh"
#include "lut_table.cuh"

namespace fdk {
namespace {

// BYTES source bytes (2, 4, 6, 8 or 16) as little-endian words; `wide`: the address is a multiple of
// BYTES (of 2 for six).
template <int BYTES>
__device__ __forceinline__ void load_piece(const uint8_t* src, bool wide, uint32_t (&w)[4]) {
  if (wide) {
    if constexpr (BYTES == 16) {
      const uint4 q = *reinterpret_cast<const uint4*>(src);
      w[0] = q.x; w[1] = q.y; w[2] = q.z; w[3] = q.w;
    } else if constexpr (BYTES == 8) {
      const uint2 q = *reinterpret_cast<const uint2*>(src);
      w[0] = q.x; w[1] = q.y;
    } else if constexpr (BYTES == 4) {
      w[0] = *reinterpret_cast<const uint32_t*>(src);
    } else {
      const uint16_t* h = reinterpret_cast<const uint16_t*>(src);
      w[0] = h[0];
      if constexpr (BYTES == 6) {
        w[0] |= (uint32_t)h[1] << 16;
        w[1] = h[2];
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < (BYTES + 3) / 4; ++i) w[i] = 0;
#pragma unroll
    for (int i = 0; i < BYTES; ++i) w[i / 4] |= (uint32_t)src[i] << (8 * (i % 4));
  }
}

// Packed codes + scales -> tiled buffer.  Bound by HBM: each warp writes one sub-tile (16 rows) of a
// slab, every lane its own V 16-byte vectors, contiguous across the warp; the lane's source is
// 2 * KSB pieces of 2 * BITS bytes (16 elements of row g and of row g + 8 of each block), and the
// four lanes of a row read 32 contiguous bytes (64 at 8 bits, 96 at 3), whole sectors.  The
// CTA's eight warps take two neighbouring slabs, so that a row's sectors and the scales' (two of
// 32 bytes per slab) are shared through L1.  11264 x 3072 at 4 bits: 62.0 us before (a byte at
// a time), 10.8 us now.
template <int BITS>
__global__ void __launch_bounds__(256)
    repack_kernel(const uint8_t* __restrict__ codes, const uint16_t* __restrict__ scale, uint8_t* __restrict__ tiled,
                  int n, int k, int per_scale, TiledDims d, bool wide) {
  using L = Layout<BITS>;
  constexpr int CB = L::kRowChunk;
  const int lane = threadIdx.x & 31, r = (threadIdx.x >> 5) & 3;
  const int g = lane >> 2, t = lane & 3;
  const size_t row_bytes = (size_t)(k / 8) * BITS;
  const int blocks = k / kBlock, scales = blocks / per_scale;
  const int slabs = d.row_tiles * d.k_slabs;
  for (int slab = blockIdx.x * 2 + (threadIdx.x >> 7); slab < slabs; slab += gridDim.x * 2) {
    const int rt = slab / d.k_slabs, ks = slab - rt * d.k_slabs;
    uint8_t* dst = tiled + (size_t)slab * L::kSlabBytes;
    uint32_t out[L::V * 4];
#pragma unroll
    for (int i = 0; i < L::V * 4; ++i) out[i] = 0;
#pragma unroll
    for (int jb = 0; jb < L::KSB; ++jb) {
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int row = rt * kTileRows + 16 * r + 8 * half + g, blk = ks * L::KSB + jb;
        if (row < n && blk < blocks) {
          uint32_t w[4];
          load_piece<CB>(codes + row * row_bytes + (size_t)blk * (8 * BITS) + t * CB, wide, w);
          if constexpr (BITS == 3) {
            const uint8_t src[6] = {(uint8_t)w[0], (uint8_t)(w[0] >> 8), (uint8_t)(w[0] >> 16), (uint8_t)(w[0] >> 24),
                                    (uint8_t)w[1], (uint8_t)(w[1] >> 8)};
            const uint64_t enc = encode3_pairs(src);
            w[0] = (uint32_t)enc;
            w[1] = (uint32_t)(enc >> 32);
          }
          const int at = (jb * 2 + half) * CB;  // byte offset inside the lane's share, constant
          if constexpr (CB >= 4 && CB % 4 == 0) {
#pragma unroll
            for (int i = 0; i < CB / 4; ++i) out[at / 4 + i] = w[i];
          } else if constexpr (CB == 2) {
            out[at / 4] |= w[0] << (8 * (at % 4));
          } else {  // six bytes, at an even offset
            if (at % 4 == 0) {
              out[at / 4] = w[0];
              out[at / 4 + 1] |= w[1];
            } else {
              out[at / 4] |= w[0] << 16;
              out[at / 4 + 1] = (w[0] >> 16) | (w[1] << 16);
            }
          }
        }
      }
    }
#pragma unroll
    for (int v = 0; v < L::V; ++v)
      *reinterpret_cast<uint4*>(dst + ((r * L::V + v) * 32 + lane) * 16) =
          make_uint4(out[4 * v], out[4 * v + 1], out[4 * v + 2], out[4 * v + 3]);
    // scales: word (jb, g, r) = rows 16 r + g and 16 r + g + 8, one lane each
    if (lane < 8 * L::KSB) {
      const int jb = lane >> 3, gg = lane & 7, blk = ks * L::KSB + jb;
      uint32_t s2 = 0;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int row = rt * kTileRows + 16 * r + 8 * half + gg;
        if (row < n && blk < blocks) s2 |= (uint32_t)scale[(size_t)row * scales + blk / per_scale] << (16 * half);
      }
      *reinterpret_cast<uint32_t*>(dst + L::kCodeBytes + jb * 128 + gg * 16 + r * 4) = s2;
    }
  }
}

// Stands between a repack and the launches after it.  A projection launched with FDK_FLAG_PDL reads the
// tiled buffer before it waits for the kernel before it; were that the repack, its stores need not be
// visible yet (it is over, or the projection would not have started, but only a wait or the plain
// order of a stream makes its stores visible).  This kernel follows the repack in plain order, and whatever
// comes next starts after it.
__global__ void repacked_kernel() {}

template <int BITS>
int launch_repack(const void* codes, const void* scale, void* tiled, int n, int k, int block_size, cudaStream_t stream) {
  const TiledDims d = tiled_dims(n, k, BITS);
  const int pairs = (int)(((long long)d.row_tiles * d.k_slabs + 1) / 2);
  constexpr int CB = Layout<BITS>::kRowChunk, kAlign = CB == 6 ? 2 : CB;
  repack_kernel<BITS><<<pairs < 148 * 32 ? pairs : 148 * 32, 256, 0, stream>>>(
      (const uint8_t*)codes, (const uint16_t*)scale, (uint8_t*)tiled, n, k, block_size / kBlock, d,
      (uintptr_t)codes % kAlign == 0);
  FDK_CUDA(cudaGetLastError());
  repacked_kernel<<<1, 32, 0, stream>>>();
  FDK_CUDA(cudaGetLastError());
  return FDK_OK;
}

__global__ void unpack_kernel(const uint8_t* __restrict__ tiled, uint8_t* __restrict__ codes,
                              uint16_t* __restrict__ scale, int n, int k, int bits, int block_size,
                              TiledDims d) {
  const int blocks = k / kBlock;
  const long long total = (long long)n * blocks * 4;
  const int cb = 2 * bits;
  const int row_bytes = k / 8 * bits;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    int t = (int)(idx & 3);
    long long rest = idx >> 2;
    int blk = (int)(rest % blocks);
    int row = (int)(rest / blocks);
    uint8_t buf[16];
    for (int i = 0; i < cb; ++i) buf[i] = tiled[tiled_code_offset(row, blk, t * cb + i, bits, d)];
    if (bits == 3) {
      uint64_t enc = 0;
      for (int i = 0; i < 6; ++i) enc |= (uint64_t)buf[i] << (8 * i);
      decode3_pairs(enc, buf);
    }
    uint8_t* dst = codes + (size_t)row * row_bytes + (size_t)blk * (8 * bits) + t * cb;
    for (int i = 0; i < cb; ++i) dst[i] = buf[i];
    if (t == 0 && (blk * kBlock) % block_size == 0) {
      scale[(size_t)row * (k / block_size) + (size_t)blk * kBlock / block_size] =
          *reinterpret_cast<const uint16_t*>(tiled + tiled_scale_offset(row, blk, d));
    }
  }
}

// Decodes 8 consecutive elements [k0, k0+8) of one row from `bits * 1` source
// bytes (8 elements always fill whole bytes) and writes one 16-byte vector.
template <bool FP16>
__device__ __forceinline__ void dequant8(const uint8_t* src, const uint16_t* __restrict__ lut, int bits,
                                         float s, uint16_t* dst) {
  uint16_t vals[8];
  if (bits == 3) {
    uint32_t be = ((uint32_t)src[0] << 16) | ((uint32_t)src[1] << 8) | src[2];
#pragma unroll
    for (int j = 0; j < 8; ++j) vals[j] = lut[(be >> (21 - 3 * j)) & 7];
  } else {
    const int e = 8 / bits;  // elements per byte
    for (int b = 0; b < bits; ++b) {
      const uint16_t* row = lut + (size_t)src[b] * e;
      for (int j = 0; j < e; ++j) vals[b * e + j] = row[j];
    }
  }
  uint4 out;
  uint32_t* o = reinterpret_cast<uint32_t*>(&out);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint16_t lo = from_float<FP16>(to_float<FP16>(vals[2 * j]) * s);
    uint16_t hi = from_float<FP16>(to_float<FP16>(vals[2 * j + 1]) * s);
    o[j] = (uint32_t)lo | ((uint32_t)hi << 16);
  }
  *reinterpret_cast<uint4*>(dst) = out;
}

// Packed codes + scales -> dense W.  Bound by the store of W (2 bytes a weight against bits / 8
// read), so everything else has to hide behind it: a thread decodes an OCTET (8 consecutive
// elements, BITS source bytes, one 16-byte store), neighbouring lanes neighbouring octets, so
// that loads and stores of a warp are contiguous; kDequantBatch octets per thread are loaded
// before the first is decoded; the byte table is looked up in shared memory, replicated per lane
// (lut_table.cuh: no bank conflicts), and the scale multiplies two elements per instruction.
// 8192^2, 4 bits, bf16: 86.9 us before (one octet per thread at a time, table read element by
// element from global memory), 35.0 us now = 4.9 TB/s of W and codes.
// Rows are contiguous and whole octets and whole blocks, so octets and scales are counted
// through the matrix: octet o has its codes at BITS * o and its scale at o / (block_size / 8).
constexpr int kDequantThreads = 512;
constexpr int kDequantBatch = 4;

template <int BITS, bool FP16>
__global__ void __launch_bounds__(kDequantThreads)
    dequantise_kernel(const uint8_t* __restrict__ codes, const uint16_t* __restrict__ lut,
                      const uint16_t* __restrict__ scale, uint4* __restrict__ w, long long octets, int block_octets,
                      int block_shift, bool aligned) {
  using T = Table<BITS>;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const uint32_t table = smem_addr(smem_raw);
  fill_table<BITS>(table, [&](int i) { return (uint32_t)lut[2 * i] | ((uint32_t)lut[2 * i + 1] << 16); });
  __syncthreads();
  const uint32_t lane_base = table + T::lane_offset(threadIdx.x & 31);
  constexpr int kWords = BITS == 8 ? 2 : 1;
  const long long step = (long long)gridDim.x * kDequantThreads * kDequantBatch;
  for (long long o0 = (long long)blockIdx.x * kDequantThreads * kDequantBatch + threadIdx.x; o0 < octets; o0 += step) {
    uint32_t c[kDequantBatch][kWords];
    uint32_t sc[kDequantBatch];
#pragma unroll
    for (int u = 0; u < kDequantBatch; ++u) {
      const long long o = o0 + u * kDequantThreads;
      if (o >= octets) break;
      const uint8_t* src = codes + o * BITS;
      if (BITS == 8 && aligned) {
        const uint2 q = __ldcs(reinterpret_cast<const uint2*>(src));
        c[u][0] = q.x;
        c[u][kWords - 1] = q.y;
      } else if (BITS == 4 && aligned) {
        c[u][0] = __ldcs(reinterpret_cast<const uint32_t*>(src));
      } else if (BITS == 2 && aligned) {
        c[u][0] = __ldcs(reinterpret_cast<const uint16_t*>(src));
      } else {
#pragma unroll
        for (int i = 0; i < kWords; ++i) c[u][i] = 0;
#pragma unroll
        for (int i = 0; i < BITS; ++i) c[u][i / 4] |= (uint32_t)src[i] << (8 * (i % 4));
      }
      sc[u] = scale[block_shift >= 0 ? o >> block_shift : o / block_octets];
    }
#pragma unroll
    for (int u = 0; u < kDequantBatch; ++u) {
      const long long o = o0 + u * kDequantThreads;
      if (o >= octets) break;
      uint4 v;
      const uint32_t x = c[u][0];
      if constexpr (BITS == 4) {
        v = make_uint4(lut32(entry_addr<4, 0>(x, lane_base)), lut32(entry_addr<4, 1>(x, lane_base)),
                       lut32(entry_addr<4, 2>(x, lane_base)), lut32(entry_addr<4, 3>(x, lane_base)));
      } else if constexpr (BITS == 8) {
        auto pair = [&](auto first, uint32_t word) {
          constexpr int J = decltype(first)::value;
          return prmt<0x7610>(lut32(entry_addr<8, J>(word, lane_base)), lut32(entry_addr<8, J + 1>(word, lane_base)));
        };
        const uint32_t y = c[u][kWords - 1];
        v = make_uint4(pair(std::integral_constant<int, 0>{}, x), pair(std::integral_constant<int, 2>{}, x),
                       pair(std::integral_constant<int, 0>{}, y), pair(std::integral_constant<int, 2>{}, y));
      } else if constexpr (BITS == 2) {
        const uint2 lo = lut64(entry_addr<2, 0>(x, lane_base)), hi = lut64(entry_addr<2, 1>(x, lane_base));
        v = make_uint4(lo.x, lo.y, hi.x, hi.y);
      } else if constexpr (BITS == 1) {
        v = lut128(entry_addr<1, 0>(x, lane_base));
      } else {  // 3 bits: four pairs of codes in 24 bits, the first in the high bits of the first byte
        const uint32_t be = prmt<0x4012>(x, 0u);
        v = make_uint4(lut32(lane_base + (be >> 18) * T::kStride), lut32(lane_base + ((be >> 12) & 63u) * T::kStride),
                       lut32(lane_base + ((be >> 6) & 63u) * T::kStride), lut32(lane_base + (be & 63u) * T::kStride));
      }
      const uint32_t s2 = sc[u] | (sc[u] << 16);
      __stcs(w + o, make_uint4(mul_pair<FP16>(v.x, s2), mul_pair<FP16>(v.y, s2), mul_pair<FP16>(v.z, s2), mul_pair<FP16>(v.w, s2)));
    }
  }
}

template <int BITS, bool FP16>
int launch_dequantise(const void* codes, const void* lut, const void* scale, void* w, long long octets, int block_octets,
                      cudaStream_t stream) {
  DeviceInfo di;
  if (int st = device_info(&di)) return st;
  int shift = -1;
  if ((block_octets & (block_octets - 1)) == 0)
    for (shift = 0; (1 << shift) < block_octets; ++shift) {}
  constexpr int kAlign = BITS == 8 ? 8 : BITS == 4 ? 4 : BITS == 2 ? 2 : 1;
  // three CTAs of 512 threads per SM; each fills its table once
  const long long per_cta = kDequantThreads * kDequantBatch;
  const long long wanted = (octets + per_cta - 1) / per_cta, most = 3LL * di.sm_count;
  dequantise_kernel<BITS, FP16><<<(int)(wanted < most ? wanted : most), kDequantThreads, Table<BITS>::kBytes, stream>>>(
      (const uint8_t*)codes, (const uint16_t*)lut, (const uint16_t*)scale, (uint4*)w, octets, block_octets, shift,
      (uintptr_t)codes % kAlign == 0);
  FDK_CUDA(cudaGetLastError());
  return FDK_OK;
}

template <bool FP16>
__global__ void dequantise_tiled_kernel(const uint8_t* __restrict__ tiled, const uint16_t* __restrict__ lut,
                                        uint16_t* __restrict__ w, int n, int k, int bits, TiledDims d) {
  // one thread per 16 consecutive elements (the unit the tiled layout keeps together)
  const long long total = (long long)n * (k / 16);
  const int cb = 2 * bits;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    int h = (int)(idx % (k / 16));
    int row = (int)(idx / (k / 16));
    int blk = h >> 2, t = h & 3;
    uint8_t buf[16];
    for (int i = 0; i < cb; ++i) buf[i] = tiled[tiled_code_offset(row, blk, t * cb + i, bits, d)];
    if (bits == 3) {
      uint64_t enc = 0;
      for (int i = 0; i < 6; ++i) enc |= (uint64_t)buf[i] << (8 * i);
      decode3_pairs(enc, buf);
    }
    float s = to_float<FP16>(*reinterpret_cast<const uint16_t*>(tiled + tiled_scale_offset(row, blk, d)));
    uint16_t* dst = w + (size_t)row * k + (size_t)h * 16;
    dequant8<FP16>(buf, lut, bits, s, dst);
    dequant8<FP16>(buf + bits, lut, bits, s, dst + 8);
  }
}

int grid_for(long long total, int threads) {
  long long g = (total + threads - 1) / threads;
  if (g > 148LL * 32) g = 148LL * 32;
  if (g < 1) g = 1;
  return (int)g;
}

int check_shape(int n, int k, int bits, int block_size) {
  FDK_CHECK_ARG(n > 0 && k > 0, FDK_ERR_BAD_ARG, "n=%d, k=%d must be positive", n, k);
  FDK_CHECK_ARG(bits_supported(bits), FDK_ERR_SHAPE, "bits=%d not in {1,2,3,4,8}", bits);
  FDK_CHECK_ARG(k % kBlock == 0, FDK_ERR_SHAPE, "k=%d must be a multiple of 64", k);
  FDK_CHECK_ARG(block_size > 0 && block_size % kBlock == 0 && k % block_size == 0, FDK_ERR_SHAPE,
                "block_size=%d must be a multiple of 64 that divides k=%d", block_size, k);
  return FDK_OK;
}

}  // namespace
}  // namespace fdk

using namespace fdk;

extern "C" int fdk_tiled_size(int n, int k, int bits, size_t* bytes_host) {
  FDK_CHECK_ARG(bytes_host != nullptr, FDK_ERR_BAD_ARG, "bytes_host is null");
  if (int st = check_shape(n, k, bits, kBlock)) return st;
  *bytes_host = tiled_bytes(n, k, bits);
  return FDK_OK;
}

extern "C" int fdk_repack(const void* codes, const void* scale, int n, int k, int bits, int block_size,
                          void* tiled, void* stream) {
  if (int st = check_shape(n, k, bits, block_size)) return st;
  FDK_CHECK_ARG(codes && scale && tiled, FDK_ERR_BAD_ARG, "null pointer");
  FDK_CHECK_ARG(((uintptr_t)tiled & 15) == 0 && ((uintptr_t)scale & 1) == 0, FDK_ERR_ALIGN,
                "tiled must be 16-byte aligned, scale 2-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  switch (bits) {
    case 1: return launch_repack<1>(codes, scale, tiled, n, k, block_size, st);
    case 2: return launch_repack<2>(codes, scale, tiled, n, k, block_size, st);
    case 3: return launch_repack<3>(codes, scale, tiled, n, k, block_size, st);
    case 4: return launch_repack<4>(codes, scale, tiled, n, k, block_size, st);
    default: return launch_repack<8>(codes, scale, tiled, n, k, block_size, st);
  }
}

extern "C" int fdk_unpack(const void* tiled, int n, int k, int bits, int block_size, void* codes,
                          void* scale, void* stream) {
  if (int st = check_shape(n, k, bits, block_size)) return st;
  FDK_CHECK_ARG(codes && scale && tiled, FDK_ERR_BAD_ARG, "null pointer");
  TiledDims d = tiled_dims(n, k, bits);
  long long total = (long long)n * (k / kBlock) * 4;
  unpack_kernel<<<grid_for(total, 256), 256, 0, (cudaStream_t)stream>>>(
      (const uint8_t*)tiled, (uint8_t*)codes, (uint16_t*)scale, n, k, bits, block_size, d);
  FDK_CUDA(cudaGetLastError());
  return FDK_OK;
}

extern "C" int fdk_dequantise(const void* codes, const void* lut, const void* scale, int n, int k,
                              int bits, int block_size, int dtype, void* w_out, void* stream) {
  FDK_CHECK_ARG(n > 0 && k > 0, FDK_ERR_BAD_ARG, "n=%d, k=%d must be positive", n, k);
  FDK_CHECK_ARG(bits_supported(bits), FDK_ERR_SHAPE, "bits=%d not in {1,2,3,4,8}", bits);
  FDK_CHECK_ARG(k % 8 == 0 && block_size > 0 && k % block_size == 0 && block_size % 8 == 0, FDK_ERR_SHAPE,
                "k=%d must be a multiple of 8 and of block_size=%d (itself a multiple of 8)", k, block_size);
  FDK_CHECK_ARG(codes && lut && scale && w_out, FDK_ERR_BAD_ARG, "null pointer");
  FDK_CHECK_ARG(dtype == FDK_DTYPE_BF16 || dtype == FDK_DTYPE_F16, FDK_ERR_BAD_ARG, "dtype=%d", dtype);
  FDK_CHECK_ARG(((uintptr_t)w_out & 15) == 0, FDK_ERR_ALIGN, "w_out must be 16-byte aligned");
  const long long octets = (long long)n * (k / 8);
  const bool fp16 = dtype == FDK_DTYPE_F16;
  auto launch = [&](auto bits_c) {
    constexpr int B = decltype(bits_c)::value;
    return fp16 ? launch_dequantise<B, true>(codes, lut, scale, w_out, octets, block_size / 8, (cudaStream_t)stream)
                : launch_dequantise<B, false>(codes, lut, scale, w_out, octets, block_size / 8, (cudaStream_t)stream);
  };
  switch (bits) {
    case 1: return launch(std::integral_constant<int, 1>{});
    case 2: return launch(std::integral_constant<int, 2>{});
    case 3: return launch(std::integral_constant<int, 3>{});
    case 4: return launch(std::integral_constant<int, 4>{});
    default: return launch(std::integral_constant<int, 8>{});
  }
}

extern "C" int fdk_dequantise_tiled(const void* tiled, const void* lut, int n, int k, int bits, int dtype,
                                    void* w_out, void* stream) {
  if (int st = check_shape(n, k, bits, kBlock)) return st;
  FDK_CHECK_ARG(tiled && lut && w_out, FDK_ERR_BAD_ARG, "null pointer");
  FDK_CHECK_ARG(dtype == FDK_DTYPE_BF16 || dtype == FDK_DTYPE_F16, FDK_ERR_BAD_ARG, "dtype=%d", dtype);
  FDK_CHECK_ARG(((uintptr_t)w_out & 15) == 0, FDK_ERR_ALIGN, "w_out must be 16-byte aligned");
  TiledDims d = tiled_dims(n, k, bits);
  long long total = (long long)n * (k / 16);
  int grid = grid_for(total, 256);
  if (dtype == FDK_DTYPE_F16) {
    dequantise_tiled_kernel<true><<<grid, 256, 0, (cudaStream_t)stream>>>(
        (const uint8_t*)tiled, (const uint16_t*)lut, (uint16_t*)w_out, n, k, bits, d);
  } else {
    dequantise_tiled_kernel<false><<<grid, 256, 0, (cudaStream_t)stream>>>(
        (const uint8_t*)tiled, (const uint16_t*)lut, (uint16_t*)w_out, n, k, bits, d);
  }
  FDK_CUDA(cudaGetLastError());
  return FDK_OK;
}
