// Fused dequantise + skinny GEMM for small batches: out[m, n] = x[m, k] . W[n, k]^T, m up to 16, W as tiled
// low-bit codes + block scales + a lookup table (fdk_layout.cuh).
//
// The arithmetic is that of linear_lut_kernel.cuh (codes from global memory straight into registers, table
// lookups in shared memory, mma.sync per 64-block in fp32, the block scale on the fp32 block sum); the split of the
// work is made for batches that share x, and for few warps with many registers each:
//   * A CTA (one per SM) works on GROUPS of 128 rows: two 64-row tiles.  Its warps are two row tiles x four or six
//     phases of K; the slabs of a group form one sequence, all groups form one sequence, of which each CTA
//     owns a contiguous range (stream-K), its phases taking slab columns in turn.
//   * The two warps of a phase share x: each copies half of a 64-column block of it into a ring in shared memory
//     (cp.async, three blocks ahead), so x is read from L2 once per 128 rows and its latency does not show.
//   * With 157 to 255 registers (at 3 bits and one n-tile 168, and spills) the lookups of one sub-tile run beside the MMAs of another, and every code vector is
//     replaced by the next slab's as soon as it has been used.  8192^2, 16 rows, 4 bits, eight warps: 16.2 us at 128
//     registers, 14.0 with all; one n-tile, 8 rows: 12.8 us with eight warps, 12.0 with twelve of 168 registers.
//   * At the end of a group the warps deposit their sums; each (tile, pair of sub-tiles, n-tile) is added up by one
//     warp and finished by it.  A group that is cut by the end of a range belongs to the CTA with its first slabs; the
//     others publish their sums as words {sum, tag, sum, tag}, which the owner polls (bounded).  Fixed orders
//     throughout: results repeat bit for bit.
// What bounds it: the shared-memory pipe (64 lookups, 16 wavefronts of x per n-tile pair and 17 of codes per 4096
// weights, of ~185 cycles at 16 rows) and the issue of ~350 instructions.  Before (linear_lut_kernel.cuh, where every
// warp reads x from L2 for itself) and now, us per launch in a graph: 8192^2, 16 rows 17.1 -> 14.0 at 4 bits, 25.1 -> 14.9
// at 3, 17.0 -> 13.9 at 2, 18.7 -> 13.9 at 1, 25.1 -> 19.7 at 8; 3072^2, 16 rows, 4 bits 9.0 -> 6.1.
#pragma once
#include <atomic>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "linear_lut_params.cuh"
#include "tp_exchange.cuh"

namespace fdk {
namespace skinny {
namespace {

// Warps of a CTA: registers count more than warps where there are two n-tiles.
template <int NB>
constexpr int kWarps = NB == 1 ? 12 : 8;
constexpr int kTiles = 2;
constexpr int kRing = 4;   // x blocks of a phase in shared memory
constexpr int kAhead = 3;  // slabs of a warp that L2 is asked for ahead of the one being loaded
constexpr uint32_t kSpinLimit = 1u << 20;

// Shared memory below everything else (bytes from its start): the norm factors of the batch rows, the position and
// the cos/sin table of the rotary output, the halves of the residual output's sums of squares.
constexpr uint32_t kHeadInv = 0, kHeadPos = 64, kHeadRope = 128, kHeadSq = 384, kHeadBytes = 640;

// The lookup table starts at this address of the shared window, so that the address of an entry is the code
// byte in bits 8..15 of the lane's offset (one PRMT), the start of the table an immediate of the load.
constexpr uint32_t kTableWindow = 2048;

__device__ __forceinline__ uint32_t tab32(uint32_t at) {
  uint32_t v;
  asm("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(at), "n"(kTableWindow));
  return v;
}
__device__ __forceinline__ uint2 tab64(uint32_t at) {
  uint2 v;
  asm("ld.shared.v2.u32 {%0,%1}, [%2+%3];" : "=r"(v.x), "=r"(v.y) : "r"(at), "n"(kTableWindow));
  return v;
}
__device__ __forceinline__ uint4 tab128(uint32_t at) {
  uint4 v;
  asm("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4+%5];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at), "n"(kTableWindow));
  return v;
}

// A fragments of one sub-tile for the four MMA k-steps of 64-block JB, from the lane's code vectors of it:
//   a[s][0] = row g,   elements 4s, 4s+1      a[s][1] = row g+8, elements 4s, 4s+1
//   a[s][2] = row g,   elements 4s+2, 4s+3    a[s][3] = row g+8, elements 4s+2, 4s+3
// (elements counted inside the lane's 16-element share of the block; x is read with the same numbering).
template <int BITS, int JB>
__device__ __forceinline__ void build_fragments(const uint4 (&code)[Layout<BITS>::V], uint32_t lane_off, uint32_t (&a)[4][4]) {
  if constexpr (BITS == 4) {
    auto four = [&](uint32_t w, int s, int row) {
      a[s][row] = tab32(entry_addr<4, 0, true>(w, lane_off));
      a[s][row + 2] = tab32(entry_addr<4, 1, true>(w, lane_off));
      a[s + 1][row] = tab32(entry_addr<4, 2, true>(w, lane_off));
      a[s + 1][row + 2] = tab32(entry_addr<4, 3, true>(w, lane_off));
    };
    four(code[0].x, 0, 0);
    four(code[0].z, 0, 1);
    four(code[0].y, 2, 0);
    four(code[0].w, 2, 1);
  } else if constexpr (BITS == 2) {
    auto row_of = [&](uint32_t w, int row) {
      const uint2 q0 = tab64(entry_addr<2, 0, true>(w, lane_off)), q1 = tab64(entry_addr<2, 1, true>(w, lane_off));
      const uint2 q2 = tab64(entry_addr<2, 2, true>(w, lane_off)), q3 = tab64(entry_addr<2, 3, true>(w, lane_off));
      a[0][row] = q0.x; a[0][row + 2] = q0.y; a[1][row] = q1.x; a[1][row + 2] = q1.y;
      a[2][row] = q2.x; a[2][row + 2] = q2.y; a[3][row] = q3.x; a[3][row + 2] = q3.y;
    };
    row_of(word_of<2 * JB>(code[0]), 0);
    row_of(word_of<2 * JB + 1>(code[0]), 1);
  } else if constexpr (BITS == 1) {
    const uint32_t w = word_of<JB>(code[0]);  // bytes 0, 1: row g; bytes 2, 3: row g + 8
    auto half_row = [&](const uint4& q, int s, int row) {
      a[s][row] = q.x; a[s][row + 2] = q.y; a[s + 1][row] = q.z; a[s + 1][row + 2] = q.w;
    };
    half_row(tab128(entry_addr<1, 0, true>(w, lane_off)), 0, 0);
    half_row(tab128(entry_addr<1, 1, true>(w, lane_off)), 2, 0);
    half_row(tab128(entry_addr<1, 2, true>(w, lane_off)), 0, 1);
    half_row(tab128(entry_addr<1, 3, true>(w, lane_off)), 2, 1);
  } else if constexpr (BITS == 8) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
#pragma unroll
      for (int row = 0; row < 2; ++row) {
        const uint32_t w = word_at(code[row], s);
        a[s][row] = prmt<0x7610>(tab32(entry_addr<8, 0, true>(w, lane_off)), tab32(entry_addr<8, 1, true>(w, lane_off)));
        a[s][row + 2] = prmt<0x7610>(tab32(entry_addr<8, 2, true>(w, lane_off)), tab32(entry_addr<8, 3, true>(w, lane_off)));
      }
    }
  } else {  // 3 bits: 96-bit little-endian group per block, pair field f at bits [6 f, 6 f + 6)
    uint32_t w[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) w[i] = word_at(code[(3 * JB + i) / 4], (3 * JB + i) % 4);
#pragma unroll
    for (int f = 0; f < 16; ++f) {
      const int o = 6 * f, wi = o >> 5, sh = o & 31;
      // the field moved to bits 7..12: times 128, the table stride
      const uint32_t v = sh + 6 > 32 ? __funnelshift_r(w[wi], w[wi + 1 < 3 ? wi + 1 : 2], sh - 7)
                                     : (sh >= 7 ? w[wi] >> (sh - 7) : w[wi] << (7 - sh));
      a[(f & 7) >> 1][(f & 1) * 2 + (f >> 3)] = tab32((v & 0x1F80u) | lane_off);
    }
  }
}

__device__ __forceinline__ uint4 ld_relaxed_v4(const uint4* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_v4(uint4* p, uint4 v) {
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// What is done with the finished sums of a tile (a value of the launch: it is looked at once per group).
enum Epilogue { kStore, kSilu, kPush, kResidual, kRotary };

// kFused: with the norm factors of the decode fusions and the rotary and tensor-parallel outputs.  kResid: with the norm
// factors and the residual output.  The plain kernel carries none of their code (0.3 us of 6 to 12), and they not
// each other's: in one, the registers of the residual output cost the others up to 15 % (3 bits, one n-tile, 28672 x
// 4096 with SiLU 29.8 us, 25.2 apart).
enum Form { kLean, kFused, kResid };
template <int BITS, int NB, bool FP16, Form FORM>
__global__ void __launch_bounds__(32 * kWarps<NB>, 1)
    skinny_lut_kernel(const __grid_constant__ LinearParams p, const __grid_constant__ InlineLut<BITS> inl) {
  constexpr bool FUSED = FORM != kLean;
  using L = Layout<BITS>;
  constexpr bool WIDE = BITS != 3;
  using Tab = Table<BITS, WIDE>;
  constexpr int kThreads = 32 * kWarps<NB>, kPhases = kWarps<NB> / kTiles;
  constexpr int kSlot = NB * 1024;         // bytes of an x block: 8 NB rows of 128 bytes
  constexpr int kFetch = 4;                // CTAs whose sums are fetched together
  constexpr int kUnits = 2 * NB;           // a tile's sums: sub-tiles (q, q + 2) x eight batch rows, unit q * NB + nb
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const uint32_t raw = smem_addr(smem_raw);
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);  // uniform for the compiler
  const int g = lane >> 2, t = lane & 3;
  const int tile = warp & (kTiles - 1), phase = warp / kTiles;
  const uint32_t table_addr = raw + p.table_off;
  const Epilogue epi = FORM == kResid ? kResidual : FORM == kFused ? (Epilogue)p.epilogue : p.silu ? kSilu : kStore;
  const uint32_t ring = raw + p.xres_off + phase * (kRing * kSlot);

  // waits go to CTAs of lower block index, which the GPU starts first
  const int cta = (int)gridDim.x - 1 - (int)blockIdx.x;
  const int c0 = cta_begin(p, cta), c1 = c0 + p.base + (cta < p.rem ? 1 : 0);
  const int row_tiles = (p.n + kTileRows - 1) / kTileRows;
  // A group's tiles are row tile `group` and row tile `group + groups`, so that the slabs of a warp's tiles lie one
  // behind the other in memory, in the order in which it takes them.  (The last group may have one tile
  // only: the other tile's warp then works on the matrix's last slab again and again, for nothing.)
  const int groups = (row_tiles + kTiles - 1) / kTiles;
  const int slab0 = tile * groups * p.k_slabs, slab_end = row_tiles * p.k_slabs - 1;
  auto slab_at = [&](int item) { return p.tiled + (size_t)(uint32_t)min(slab0 + item, slab_end) * L::kSlabBytes; };
  int it = c0 + phase;

  // codes first: they do not depend on the kernel before
  uint4 code[kSubTiles][L::V], sc[L::KSB];
  if (it < c1) {
    const uint8_t* const slab = slab_at(it);
#pragma unroll
    for (int r = 0; r < kSubTiles; ++r)
#pragma unroll
      for (int v = 0; v < L::V; ++v) code[r][v] = ldg_stream(slab + lane * 16 + (r * L::V + v) * 512);
#pragma unroll
    for (int jb = 0; jb < L::KSB; ++jb) sc[jb] = ldg_stream(slab + L::kCodeBytes + g * 16 + jb * 128);
#pragma unroll 1
    for (int d = 1; d <= kAhead; ++d)
      if (lane == 0 && it + d * kPhases < c1) prefetch_slab<BITS>(slab_at(it + d * kPhases));
  }
  {
    const bool from_params = p.lut == nullptr;
    auto word = [&](int i) { return from_params ? inl.w[i] : __ldg(reinterpret_cast<const uint32_t*>(p.lut) + i); };
    if constexpr (BITS == 4 || BITS == 2 || BITS == 1) fill_table_unrolled<BITS, WIDE, kThreads>(table_addr, word, (int)threadIdx.x);
    else fill_table<BITS, WIDE>(table_addr, kThreads, word, (int)threadIdx.x);
  }
  // batch rows that there are none of: zeros
  for (int i = threadIdx.x; i < kPhases * kRing * NB * 8 * 8; i += kThreads) {
    const int row = (i >> 3) % (8 * NB);
    if (row >= p.m) asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(raw + p.xres_off + i * 16), "r"(0u) : "memory");
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (table_addr != kTableWindow) {  // the host planned for another window address (uniform exit)
    if (threadIdx.x == 0) atomicOr(p.counters + kStatusWord, kStatusSmemLayout);
    return;
  }

  // x: slab and column of the block to be copied next, and its slot.  The copies run on behind the last block
  // that is needed (the columns start again from 0 at the end of a row).
  const int first = div_k(p, c0), last = div_k(p, c1 - 1);
  const int k_pad = p.k_slabs * L::kSlabK;
  int xs = (it - first * p.k_slabs) * L::kSlabK;
  while (xs >= k_pad) xs -= k_pad;
  int xcol = xs;
  uint32_t xslot = 0;
  // lane's chunks: row 4 tile + lane / 8 (+ 8 i), 16-byte column lane % 8
  const int xrow = tile * 4 + (lane >> 3);
  const uint16_t* const xsrc = p.x + (size_t)xrow * p.k + (lane & 7) * 8;
  const uint32_t xdst = ring + xrow * 128 + (((lane & 7) ^ (xrow & 7)) << 4);
  auto copy_x = [&] {
#pragma unroll
    for (int i = 0; i < NB; ++i)
      if (xrow + 8 * i < p.m)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(xdst + xslot + i * 1024), "l"(xsrc + (size_t)(8 * i) * p.k + xcol)
                     : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
    xslot = (xslot + kSlot) & (kRing * kSlot - 1);
    if (L::KSB > 1) xcol += kBlock;
    if (L::KSB == 1 || (xcol & (L::kSlabK - 1)) == 0 || xcol >= p.k) {  // (padded blocks are left out)
      xs += kPhases * L::kSlabK;
      while (xs >= k_pad) xs -= k_pad;
      xcol = xs;
    }
  };
#pragma unroll
  for (int d = 0; d < kRing - 1; ++d) copy_x();
  const int uses_first = ld_relaxed_s32(p.counters + first), uses_last = ld_relaxed_s32(p.counters + last);
  uint32_t push_seq = 0;
  if (FORM == kFused && epi == kPush) push_seq = (uint32_t)ld_relaxed_s32(reinterpret_cast<const int*>(p.seq));  // reduces completed so far
  if constexpr (FUSED) {
    // what only the epilogues read: the deferred RMSNorm's factors (the row's sums of squares added in a fixed order; 1
    // without it), the position and its cos/sin table
    float* const inv = reinterpret_cast<float*>(smem_raw + kHeadInv);
#pragma unroll 1
    for (int b = warp; b < 8 * NB; b += kWarps<NB>) {
      float sum = 0.f;
      if (p.scale_ss != nullptr && b < p.m) {
#pragma unroll 1
        for (int j0 = lane; j0 < p.scale_tiles; j0 += 128) {
          float part[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) part[u] = j0 + 32 * u < p.scale_tiles ? __ldcg(p.scale_ss + (size_t)b * p.scale_tiles + j0 + 32 * u) : 0.f;
          sum += (part[0] + part[1]) + (part[2] + part[3]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      }
      if (lane == 0) inv[b] = p.scale_ss != nullptr && b < p.m ? rsqrtf(sum / (float)p.k + p.scale_eps) : 1.f;
    }
    if (FORM == kFused && epi == kRotary && warp == kWarps<NB> - 1) {
      uint32_t* const table = reinterpret_cast<uint32_t*>(smem_raw + kHeadRope);
      table[lane] = __ldcg(p.rope_table + lane);
      table[lane + 32] = __ldcg(p.rope_table + lane + 32);
      if (lane == 0) *reinterpret_cast<long long*>(smem_raw + kHeadPos) = *reinterpret_cast<const volatile long long*>(p.rope_pos);
    }
  }
  __syncthreads();  // the table and the zero rows are in place
  uint32_t lane_off = Tab::lane_offset(lane);
  asm volatile("" : "+r"(lane_off)::"memory");  // lookups, plain functions of it, stay behind the barrier

  float tot[kSubTiles][NB][4];
#pragma unroll
  for (int r = 0; r < kSubTiles; ++r)
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int i = 0; i < 4; ++i) tot[r][nb][i] = 0.f;
  bool timed_out = false;
  int cur = first;

  auto deposit_at = [&](int of_warp, int unit, int half) {
    const uint32_t slot = (uint32_t)((of_warp * kUnits + unit) * 2 + half);
    return raw + p.slots_off + slot * 512 + lane * 16;
  };
  // What the residual output reads for a unit, asked for together and ahead of the sums: h is read and written, so loads
  // left beside the stores wait for them one by one (eight trips to L2 at two rows and more: 3 rows of 3072^2, 4 bits
  // 8.5 us, 6.0 this way).
  struct Residual {
    uint16_t h[FORM == kResid ? 2 : 1][4], w[FORM == kResid ? 2 : 1][2];
  };
  auto fetch_residual = [&](int rt, int q, int nb, Residual& r) {
    if constexpr (FORM == kResid) {
      const int row0 = rt * kTileRows + 16 * q + g;
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int b = 8 * nb + 2 * t + (i & 1), row = row0 + 32 * h + 8 * (i >> 1);
          r.h[h][i] = b < p.m && row < p.n ? __ldcg(p.resid_h + (size_t)b * p.n + row) : (uint16_t)0;
          if ((i & 1) == 0) r.w[h][i >> 1] = p.resid_w != nullptr && row < p.n ? __ldg(p.resid_w + row) : (uint16_t)0;
        }
    }
  };
  // The end of the sub-tiles q and q + 2 of row tile rt, batch rows 8 nb .. 8 nb + 7: sum[h][i] is row
  // 16 q + 32 h + g + 8 (i / 2) of the tile, batch row 8 nb + 2 t + i % 2.
  auto finish = [&](int rt, int q, int nb, const float (&sum)[2][4], const Residual& res) {
    auto rnd = [](float v) { return to_float<FP16>(from_float<FP16>(v)); };
    const int row0 = rt * kTileRows + 16 * q + g;  // row of sum[0][0]
    const bool live = rt < row_tiles;
    if constexpr (FORM == kResid) {
      // y rounded as if stored, added to the residual stream; sums of squares over the lanes of a batch row
      float sq[2] = {0.f, 0.f};
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int b = 8 * nb + 2 * t + (i & 1), row = row0 + 32 * h + 8 * (i >> 1);
          if (live && b < p.m && row < p.n) {
            const size_t at = (size_t)b * p.n + row;
            const uint16_t hnew = from_float<FP16>(to_float<FP16>(res.h[h][i]) + rnd(sum[h][i]));
            p.resid_h[at] = hnew;
            const float hf = to_float<FP16>(hnew);
            sq[i & 1] = fmaf(hf, hf, sq[i & 1]);
            if (p.resid_w != nullptr)  // the next RMSNorm's weight folded in: x of the next projection
              p.resid_x[at] = from_float<FP16>(hf * to_float<FP16>(res.w[h][i >> 1]));
          }
        }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) sq[j] += __shfl_xor_sync(0xffffffffu, sq[j], o);
        if (g == 0) reinterpret_cast<float*>(smem_raw + kHeadSq)[(tile * 2 + q) * 8 * NB + 8 * nb + 2 * t + j] = sq[j];
      }
    } else if (FORM == kFused && epi == kPush) {
      // four consecutive rows (four lanes) as two words {two outputs, tag}, into every rank's exchange buffer
      const uint32_t ptag = push_seq + 1u;
      const size_t base = (size_t)((push_seq & 1u) * p.tp + p.rank) * p.stage_slot;
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t v = from_float<FP16>(sum[h][i]);
          const uint32_t pair = v | (__shfl_down_sync(0xffffffffu, v, 4) << 16);
          const uint32_t next = __shfl_down_sync(0xffffffffu, pair, 8);
          const int b = 8 * nb + 2 * t + (i & 1);
          if (live && b < p.m && (g & 3) == 0) {
            const size_t off = (base + (size_t)b * p.n + row0 + 32 * h + 8 * (i >> 1)) / 2;
#pragma unroll 1
            for (int j = 0; j < p.tp; ++j)
              asm volatile("st.relaxed.sys.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p.peer_stage[j] + off), "r"(pair), "r"(ptag),
                           "r"(next), "r"(ptag)
                           : "memory");
          }
        }
    } else if (live) {
      const long long pos = FORM == kFused ? *reinterpret_cast<const long long*>(smem_raw + kHeadPos) : 0;
      const bool in_cache = FORM == kFused && epi == kRotary && pos >= 0 && pos < p.max_len;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int b = 8 * nb + 2 * t + (i & 1), lrow = 16 * q + g + 8 * (i >> 1);  // of 32: the partner is 32 rows on
        if (b >= p.m) continue;
        if (epi == kStore) {
          uint16_t* const dst = p.out + (size_t)b * p.n + rt * kTileRows + lrow;
          if (rt * kTileRows + lrow < p.n) dst[0] = from_float<FP16>(sum[0][i]);
          if (rt * kTileRows + lrow + 32 < p.n) dst[32] = from_float<FP16>(sum[1][i]);
        } else if (FORM == kLean || epi == kSilu) {  // rows come as 32 gate + 32 up
          const float gate = rnd(sum[0][i]), up = rnd(sum[1][i]);
          p.out[(size_t)b * (p.n / 2) + rt * (kTileRows / 2) + lrow] = from_float<FP16>(rnd(gate / (1.f + __expf(-gate))) * up);
        } else {  // rotary: tile rt is half th of head rt / 2; dimensions 32 th + lrow and 64 further on
          const int head = rt >> 1, th = rt & 1;
          const float x0 = rnd(sum[0][i]), x1 = rnd(sum[1][i]);
          if (head < p.q_heads + p.kv_heads) {
            const uint32_t cs = reinterpret_cast<const uint32_t*>(smem_raw + kHeadRope)[32 * th + lrow];
            const float co = pair_lo<FP16>(cs), si = pair_hi<FP16>(cs);
            const uint16_t o0 = from_float<FP16>(rnd(x0 * co) + rnd(-x1 * si)), o1 = from_float<FP16>(rnd(x1 * co) + rnd(x0 * si));
            uint16_t* dst = nullptr;
            if (head < p.q_heads) dst = p.q_out + ((size_t)b * p.q_heads + head) * 128;
            else if (in_cache) dst = p.k_cache + (((size_t)b * p.kv_heads + (head - p.q_heads)) * p.max_len + pos) * 128;
            if (dst != nullptr) {
              dst[32 * th + lrow] = o0;
              dst[32 * th + lrow + 64] = o1;
            }
          } else if (in_cache) {  // v: rows in their own order
            uint16_t* const dst = p.v_cache + (((size_t)b * p.kv_heads + (head - p.q_heads - p.kv_heads)) * p.max_len + pos) * 128;
            dst[64 * th + lrow] = from_float<FP16>(x0);
            dst[64 * th + lrow + 32] = from_float<FP16>(x1);
          }
        }
      }
    }
  };
  // Finishes groups cur .. target - 1: every warp deposits its sums, the owner of a unit adds the phases
  // in order, and writes the outputs, publishes the sums (a group that starts in another CTA), or adds the
  // sums of the CTAs that hold the rest of the group.
  auto flush_until = [&](int target) {
#pragma unroll 1
    while (cur < target) {
      const int lo = cur * p.k_slabs, hi = lo + p.k_slabs;
      const bool owner = c0 <= lo, full = owner && c1 >= hi;
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float(&v)[4] = tot[q + 2 * h][nb];
            asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(deposit_at(warp, q * NB + nb, h)), "f"(v[0]), "f"(v[1]),
                         "f"(v[2]), "f"(v[3])
                         : "memory");
            v[0] = v[1] = v[2] = v[3] = 0.f;
          }
      Residual res;
      if (FORM == kResid && owner && phase < kUnits) fetch_residual(cur + tile * groups, phase / NB, phase % NB, res);
      __syncthreads();
      const int uses = cur == first ? uses_first : uses_last;  // only those two can be split
      const uint32_t tag = ((uint32_t)(uses + 1) << 12) | (uint32_t)cur;
      if (phase < kUnits) {
        const int unit = phase, q = unit / NB, nb = unit % NB;
        float sum[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int ph = 0; ph < kPhases; ++ph) {
            float4 d;
            asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];"
                         : "=f"(d.x), "=f"(d.y), "=f"(d.z), "=f"(d.w)
                         : "r"(deposit_at(ph * kTiles + tile, unit, h))
                         : "memory");
            s.x += d.x; s.y += d.y; s.z += d.z; s.w += d.w;
          }
          sum[h][0] = s.x; sum[h][1] = s.y; sum[h][2] = s.z; sum[h][3] = s.w;
        }
        // words {sum, tag, sum, tag}: four per lane, unit and tile
        auto words = [&](int of_cta) {
          return reinterpret_cast<uint4*>(p.partial) + ((size_t)of_cta * (kTiles * kUnits) + tile * kUnits + unit) * 128 + lane;
        };
        if (!owner) {
          uint4* const mine = words(cta);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            st_relaxed_v4(mine + j * 32, make_uint4(__float_as_uint(sum[j >> 1][2 * (j & 1)]), tag,
                                                    __float_as_uint(sum[j >> 1][2 * (j & 1) + 1]), tag));
        } else {
          if (!full) {
            int end = cta + 1;  // the CTAs up to the one with the group's last slab
            while (cta_begin(p, end) < hi) ++end;
#pragma unroll 1
            for (int cb = cta + 1; cb < end; cb += kFetch) {  // in CTA order, some at a time
              uint4 v[kFetch][4];
              for (uint32_t spin = 0;; ++spin) {
                bool fresh = true;
#pragma unroll
                for (int o = 0; o < kFetch; ++o)
#pragma unroll
                  for (int j = 0; j < 4; ++j) {
                    v[o][j] = cb + o < end ? ld_relaxed_v4(words(cb + o) + j * 32) : make_uint4(0u, tag, 0u, tag);
                    fresh = fresh && v[o][j].y == tag && v[o][j].w == tag;
                  }
                if (__all_sync(0xffffffffu, fresh)) break;
                if (spin > kSpinLimit) {
                  timed_out = true;
                  break;
                }
              }
#pragma unroll
              for (int o = 0; o < kFetch; ++o)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  sum[j >> 1][2 * (j & 1)] += __uint_as_float(v[o][j].x);
                  sum[j >> 1][2 * (j & 1) + 1] += __uint_as_float(v[o][j].z);
                }
            }
          }
          if constexpr (FUSED) {
            const float* const inv = reinterpret_cast<const float*>(smem_raw + kHeadInv) + 8 * nb + 2 * t;
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int i = 0; i < 4; ++i) sum[h][i] *= inv[i & 1];
          }
          finish(cur + tile * groups, q, nb, sum, res);
        }
      }
      __syncthreads();  // the deposits have been read; everybody is done with the foreign sums
      if (!full && owner && threadIdx.x == 0) p.counters[cur] = (uses + 1) & 0x7FFFF;
      if (FORM == kResid && owner && threadIdx.x < kTiles * 8 * NB) {
        const int of_tile = threadIdx.x / (8 * NB), b = threadIdx.x % (8 * NB), rt = cur + of_tile * groups;
        const float* const sq = reinterpret_cast<const float*>(smem_raw + kHeadSq) + of_tile * 2 * 8 * NB + b;
        if (b < p.m && rt < row_tiles) p.resid_ss[(size_t)b * row_tiles + rt] = sq[0] + sq[8 * NB];
      }
      ++cur;
    }
  };

  // lane's share of x rows g (+ 8 nb): 16-byte chunks 2 t and 2 t + 1, swizzled by the row
  const uint32_t x_lo = g * 128 + (((2 * t) ^ g) << 4), x_hi = g * 128 + (((2 * t + 1) ^ g) << 4);
  uint32_t slot = 0;
  int seg_end = (first + 1) * p.k_slabs;
#pragma unroll 1
  for (; it < c1; it += kPhases) {
    while (it >= seg_end) {
      flush_until(cur + 1);
      seg_end += p.k_slabs;
    }
    const uint8_t* const next = slab_at(min(it + kPhases, c1 - 1)) + lane * 16;  // (at the end a slab that L2 has anyway)
    const uint8_t* const next_sc = next + (L::kCodeBytes + g * 16 - lane * 16);
    if (it + (kAhead + 1) * kPhases < c1) {
      if (lane == 0) prefetch_slab<BITS>(slab_at(it + (kAhead + 1) * kPhases));
    }
    const int col0 = (it - (seg_end - p.k_slabs)) * L::kSlabK;
    // Each code vector is replaced by the next slab's as soon as it has been used: vector v of a sub-tile is last
    // used by block ((v + 1) * 16 - 1) / (4 * BITS).
    auto refill = [&](auto jbc, auto rc) {
      constexpr int R = decltype(rc)::value;
#pragma unroll
      for (int v = 0; v < L::V; ++v)
        if (((v + 1) * 16 - 1) / (4 * BITS) == decltype(jbc)::value) code[R][v] = ldg_stream(next + (R * L::V + v) * 512);
    };
    auto block = [&](auto jbc) {
      constexpr int JB = decltype(jbc)::value;
      const bool live = L::KSB == 1 || col0 + JB * kBlock < p.k;  // a padded block holds zero codes and scales
      if (!live) {
        sc[JB] = ldg_stream(next_sc + JB * 128);
        refill(jbc, std::integral_constant<int, 0>{});
        refill(jbc, std::integral_constant<int, 1>{});
        refill(jbc, std::integral_constant<int, 2>{});
        refill(jbc, std::integral_constant<int, 3>{});
        return;
      }
      float scale[kSubTiles][2];
      {
        const uint32_t w[4] = {sc[JB].x, sc[JB].y, sc[JB].z, sc[JB].w};
#pragma unroll
        for (int r = 0; r < kSubTiles; ++r) {
          scale[r][0] = pair_lo<FP16>(w[r]);
          scale[r][1] = pair_hi<FP16>(w[r]);
        }
      }
      sc[JB] = ldg_stream(next_sc + JB * 128);
      asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 2) : "memory");
      asm volatile("bar.sync %0, %1;" ::"r"(1 + phase), "n"(32 * kTiles) : "memory");  // both halves are there
      copy_x();
      const uint32_t at = ring + slot;
      slot = (slot + kSlot) & (kRing * kSlot - 1);
      uint32_t x[NB][8];
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        const uint4 l4 = ring128(at + nb * 1024 + x_lo), h4 = ring128(at + nb * 1024 + x_hi);
        x[nb][0] = l4.x; x[nb][1] = l4.y; x[nb][2] = l4.z; x[nb][3] = l4.w;
        x[nb][4] = h4.x; x[nb][5] = h4.y; x[nb][6] = h4.z; x[nb][7] = h4.w;
      }
      auto sub_tile = [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        uint32_t a[4][4];
        build_fragments<BITS, JB>(code[R], lane_off, a);
        refill(jbc, rc);
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          float acc[4];
          const float zero[4] = {0.f, 0.f, 0.f, 0.f};
          mma16816<FP16>(acc, a[0], x[nb][0], x[nb][1], zero);
#pragma unroll
          for (int st = 1; st < 4; ++st) mma16816<FP16>(acc, a[st], x[nb][2 * st], x[nb][2 * st + 1], acc);
          tot[R][nb][0] = fmaf(acc[0], scale[R][0], tot[R][nb][0]);
          tot[R][nb][1] = fmaf(acc[1], scale[R][0], tot[R][nb][1]);
          tot[R][nb][2] = fmaf(acc[2], scale[R][1], tot[R][nb][2]);
          tot[R][nb][3] = fmaf(acc[3], scale[R][1], tot[R][nb][3]);
        }
      };
      sub_tile(std::integral_constant<int, 0>{});
      sub_tile(std::integral_constant<int, 1>{});
      sub_tile(std::integral_constant<int, 2>{});
      sub_tile(std::integral_constant<int, 3>{});
    };
    block(std::integral_constant<int, 0>{});
    if constexpr (L::KSB > 1) block(std::integral_constant<int, 1>{});
    if constexpr (L::KSB > 2) {
      block(std::integral_constant<int, 2>{});
      block(std::integral_constant<int, 3>{});
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");  // the copies behind the last block
  flush_until(last + 1);
  if (timed_out && lane == 0) atomicOr(p.counters + kStatusWord, kStatusTimeout);
}

// ---- host side ----------------------------------------------------------------------------------------------

template <int BITS, int NB, bool FP16, Form FORM>
int launch_kernel(LinearParams p, const InlineLut<BITS>& inl, int sm_count, unsigned flags, cudaStream_t stream) {
  constexpr int kThreads = 32 * kWarps<NB>, kPhases = kWarps<NB> / kTiles;
  uint32_t base = 0;
  if (int st = dynamic_smem_base(&base)) return st;
  DeviceInfo di;
  if (int st = device_info(&di)) return st;
  FDK_CHECK_ARG(base + kHeadBytes <= kTableWindow, FDK_ERR_CUDA, "dynamic shared memory starts at %u of the window", base);
  uint32_t at = kTableWindow - base;
  p.table_off = at;
  at += Table<BITS, BITS != 3>::kBytes;
  p.slots_off = at;  // deposits
  at += kThreads * 2 * NB * 2 * 16;
  p.xres_off = at;  // x ring
  at += kPhases * kRing * NB * 1024;
  FDK_CHECK_ARG(at <= (uint32_t)di.max_smem_optin, FDK_ERR_CUDA, "%u bytes of shared memory exceed %d", at, di.max_smem_optin);
  p.epilogue = p.tp > 0 ? kPush : p.silu ? kSilu : p.resid_h != nullptr ? kResidual : p.rope_pos != nullptr ? kRotary : kStore;
  const int groups = (p.total / p.k_slabs + kTiles - 1) / kTiles;
  p.total = groups * p.k_slabs;
  // One CTA per SM, fewer where so many would share a group that fetching their sums (about 0.2 us a CTA) costs
  // more than they save (a slab takes a warp about 0.9 us): total / (grid phases) 0.9 + grid / groups 0.2 is least at
  // the root below (256 x 20480, 3 rows: 20.2 us with 148 CTAs).  Not fewer than groups: with as many none is shared
  // (256^2, one row at 1 bit, two groups of one slab: 4.8 us in one CTA, 3.2 in two).
  const double best = std::sqrt((double)p.total * groups * (0.9 / 0.2) / kPhases);
  int grid = p.total < sm_count ? p.total : sm_count;
  if (best < grid) grid = best < groups ? (groups < grid ? groups : grid) : (int)best;
  p.base = p.total / grid;
  p.rem = p.total % grid;
  auto kernel = skinny_lut_kernel<BITS, NB, FP16, FORM>;
  static std::atomic<bool> allowed[64] = {};
  if (int st = allow_all_smem(kernel, allowed, di)) return st;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = at;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (flags & FDK_FLAG_PDL) ? 1 : 0;
  FDK_CUDA(cudaLaunchKernelEx(&cfg, kernel, p, inl));
  return FDK_OK;
}

template <int BITS, int NB, bool FP16>
int launch(const LinearParams& p, const InlineLut<BITS>& inl, int sm_count, unsigned flags, cudaStream_t stream) {
  const bool fused = p.tp > 0 || p.rope_pos != nullptr || p.scale_ss != nullptr;
  if constexpr (!FP16) {  // (the decode fusions take bf16)
    if (p.resid_h != nullptr) return launch_kernel<BITS, NB, FP16, kResid>(p, inl, sm_count, flags, stream);
  }
  return fused ? launch_kernel<BITS, NB, FP16, kFused>(p, inl, sm_count, flags, stream)
               : launch_kernel<BITS, NB, FP16, kLean>(p, inl, sm_count, flags, stream);
}

}  // namespace
}  // namespace skinny

template <int BITS>
int launch_skinny_bits(LinearParams p, const void* lut_host, int sm_count, int dtype, unsigned flags, cudaStream_t stream) {
  InlineLut<BITS> inl;
  if (lut_host != nullptr) {
    memcpy(inl.w, lut_host, sizeof(inl.w));
    p.lut = nullptr;
  } else {
    memset(inl.w, 0, sizeof(inl.w));
  }
  if (dtype == FDK_DTYPE_F16) {
    return p.m > 8 ? skinny::launch<BITS, 2, true>(p, inl, sm_count, flags, stream) : skinny::launch<BITS, 1, true>(p, inl, sm_count, flags, stream);
  }
  return p.m > 8 ? skinny::launch<BITS, 2, false>(p, inl, sm_count, flags, stream) : skinny::launch<BITS, 1, false>(p, inl, sm_count, flags, stream);
}

}  // namespace fdk
