// Fused dequantise + GEMM for batches of 17 and more rows, on the fifth-generation tensor
// cores:  out[m, n] = x[m, k] . W[n, k]^T  with W = bf16(table value * block scale), the
// reference's dense W (src/fdk/kernels.py:23-24) bit for bit (fp16(...) for fp16 inputs), built
// block by block in tensor memory and never written to HBM.
//
// Persistent, one CTA per SM.  The product is cut into tiles of 128 weight rows (MMA M) by up to
// 192 batch rows (MMA N); the slabs of all tiles form one sequence, of which each CTA owns a
// contiguous range, so every SM has the same work whatever the sizes.  A tile that is cut by a
// range boundary belongs to the CTA with its first slabs; the others park their fp32 sums in the
// workspace, under flags that hold the number of the launch: a flag that an earlier launch left, whatever
// became of that launch, is never taken for one of this.  24 warps, specialised:
//   warps 0..15  dequantise, in four sets of four warps; set s takes the 64-column blocks
//                s, s + 4, ...: code bytes from shared memory -> replicated table lookup ->
//                times the block scale -> tcgen05.st into the stage's A tile in TENSOR memory;
//   warps 16..19 epilogue of a tile, while the next one is being computed (the last tile of
//                a CTA, when the dequantising warps have nothing left to do, is shared with them);
//   warps 20, 21 code slabs by cp.async.bulk, into a ring of their own;
//   warp 22      x by tiled TMA loads (tensor map, 128-byte swizzle, no multicast);
//   warp 23      allocates tensor memory; one thread issues tcgen05.mma (A from tensor memory,
//                x from shared memory) and tcgen05.commit hands the stage back.
// What bounds it: up to about 128 batch rows the dequantising warps (a block of 128 x 64 weights takes
// ~750 warp instructions, ~190 cycles of four schedulers, and ~170 shared-memory wavefronts) and the
// latency of the single threads that issue copies and MMAs (a barrier read queues behind the lookups:
// 110 to 190 cycles); above, the tensor pipe (2 N cycles a block).  A in tensor memory keeps both
// the store of the tile and the MMA's reads of it out of shared memory, and its MMAs of
// small N are faster (a block at N = 32 takes 68 cycles, 161 with A in shared memory).  Before (A in
// shared memory, eight dequantising warps, a tile per CTA) and now, 4 bits, public call: 48 rows of
// 11264 x 3072, four in a graph, 92.4 -> 51.0 us; 2048 rows of 28672 x 4096 792 -> 403 to 428 us, by the clock
// (1.12 to 1.19 PFLOP/s).  Tried and not kept: groups of four blocks per copy, barrier and stage (18.4 us at
// 32 rows of 8192^2 against 16.7, kernel alone: a set then waits for a whole group, and the larger
// stages leave fewer of them).
// Every wait is bounded; one that runs out sets a status bit, and the kernel still lets copies and MMAs on
// their way arrive, frees its tensor memory and returns.  Under programmatic launch the bounds count this kernel's own time only: a
// role waits for the kernel before (griddepcontrol.wait, which has no bound) ahead of its first bounded
// wait that x, and so that kernel, can hold up.
#include <cuda.h>

#include <cmath>
#include <cstring>

#include "fdk_common.cuh"
#include "gemm_cut.cuh"
#include "lut_table.cuh"

namespace fdk {
namespace {

constexpr int kTcDequantWarps = 16;
constexpr int kTcEpilogueWarps = 4;
constexpr int kTcCodeWarps = 2;
constexpr int kTcWarps = kTcDequantWarps + kTcEpilogueWarps + kTcCodeWarps + 2;
constexpr int kTcXWarp = kTcWarps - 2, kTcMmaWarp = kTcWarps - 1, kTcFirstCodeWarp = kTcXWarp - kTcCodeWarps;
constexpr int kTcThreads = 32 * kTcWarps;
constexpr int kTcTileRows = 128;
// Batch rows of a tile (MMA N, at most 256).  With 192 two accumulators and four A stages fit tensor memory,
// so a tile's epilogue overlaps the next tile; with 256 it does not: 4 bits, kernel alone, 1000 rows of
// 5120 x 3072 35.9 us against 30.8, 256 of 3072^2 20.9 / 13.6, 2048 of 28672 x 4096 366 / 352.  128: 31.4, 13.6, 388.
constexpr int kTcMaxBatch = 192;
constexpr int kTcMaxStages = 8;
constexpr int kTcMaxCodeSlots = 16;
constexpr int kTcTmemColumns = 512;
constexpr int kTcAccumulators = 2;
static_assert(kTcFlagsPerRank == (kTcMaxBatch / 16) * 4, "a flag per 16 batch columns x 32 weight rows");
// Launches counted in the workspace: every CTA adds one at its end, rank 0 also what is missing to 2^16, so that
// the count above the low 16 bits moves on when the last CTA has added.
constexpr int kTcLaunchShift = 16;
// rows of the lookup table 256 bytes apart: a lookup address is one PRMT.  8 bits: no room beside
// 128 batch rows and four slabs
template <int BITS>
constexpr bool kTcWideTable = BITS == 1 || BITS == 2 || BITS == 4;
constexpr int kTcStatusTimeout = 1;
constexpr int kTcStatusSmemLayout = 2;

struct TcParams {
  const uint8_t* tiled;
  const void* lut;        // device byte table, or null when it travels in the parameters
  uint16_t* out;
  int* status;            // device-side error bits
  int m, n, n_tile;       // batch rows, weight rows, batch rows of a tile (multiple of 16)
  int m_tiles, tiles;     // batch tiles; all tiles (the batch tile varies fastest)
  int row_tiles;          // 64-row tiles of the tiled buffer
  int k_blocks, k_slabs;  // k / 64; slabs per 64-row tile
  int stages_log2, code_slots;
  int split;              // ranges may cut tiles
  TcCut cut;              // the CTAs' ranges of units (of whole tiles where they are not cut)
  float* partial;         // [rank][n_tile][128] fp32 sums of a CTA that does not own its first tile
  int* flags;             // [rank][column sixteenth][row quarter] the launch that published
  unsigned long long* launches;  // launches on this workspace with cut tiles
  uint32_t smem_base, table_addr, bar_addr;
  uint32_t b_addr[kTcMaxStages], c_addr[kTcMaxCodeSlots];
};

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(map), "r"(c0), "r"(c1), "r"(bar)
      : "memory");
}
// One thread of a converged warp.  The warps that issue copies and MMAs run their loops with all
// lanes and only issue under this predicate: addresses and descriptors, which those instructions
// take from uniform registers, then stay there (in a branch on the lane number each MMA
// cost ~160 cycles of register moves: 8192^2, 32 rows: 30.5 us).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Shared-memory matrix descriptor but for the address (its bits 4..17 go to bits 0..13): K-major,
// 128-byte swizzle (2 in bits 61..63), 8-row groups 1024 bytes apart (bits 32..45, in 16-byte units; the
// leading offset, bits 16..29, is unused with a swizzle), descriptor version 1 (bit 46).
constexpr uint64_t kDescBase = ((uint64_t)2 << 61) | ((uint64_t)1 << 46) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 16);

// D[tensor memory] (+)= A[tensor memory: one lane per row, two 16-bit elements per column] . B[shared]^T
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_store16(uint32_t addr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"r"(v[0]),
      "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
      "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tmem_load16(uint32_t addr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(addr)
      : "memory");
}

__device__ __forceinline__ void tmem_load8(uint32_t addr, uint32_t (&v)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
      : "r"(addr)
      : "memory");
}

__device__ __forceinline__ uint32_t ring32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint2 ring64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
  return v;
}

// A lane's tile row and the code words of it.  The tiled buffer gives the 16 elements [16 t, 16 t + 16)
// of rows 16 r + g and 16 r + g + 8 to lane 4 g + t; here lane 4 g + t collects the whole block of
// ONE row, because a tensor-memory lane is a row of A (16 r + 8 half + g of a 64-row tile).  Fetching piece c
// (16 elements) from all lanes at once would meet in a few banks, the rows being 64 and 512 bytes
// apart, so lane l fetches piece c ^ x(l) in round c (x spreads what the bank bits of the row do
// not) and the pieces are put in order by conditional swaps.
template <int BITS>
struct RowCodes {
  static constexpr int kWords = BITS == 8 ? 4 : (BITS == 4 || BITS == 3) ? 2 : 1;  // words per piece
  uint32_t w[4][kWords];

  // slab: the 64-row slab of the lane's row; r: its 16-row sub-tile, half: row 8..15 of it; jb: block of the slab
  __device__ __forceinline__ void load(uint32_t slab, int jb, int g, int r, int half, int x) {
    using L = Layout<BITS>;
    const uint32_t at = slab + (r * L::V * 32 + 4 * g) * 16;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const uint32_t lane_at = at + (uint32_t)((c ^ x) * 16);
      if constexpr (BITS == 4) {
        const uint2 q = ring64(lane_at + half * 8);
        w[c][0] = q.x; w[c][1] = q.y;
      } else if constexpr (BITS == 8) {
        const uint4 q = ring128(lane_at + half * 512);
        w[c][0] = q.x; w[c][1] = q.y; w[c][2] = q.z; w[c][3] = q.w;
      } else if constexpr (BITS == 2) {
        w[c][0] = ring32(lane_at + jb * 8 + half * 4);
      } else if constexpr (BITS == 1) {
        w[c][0] = ring32(lane_at + jb * 4) >> (16 * half);
      } else {  // 3 bits: 12 bytes per block and lane, six of each row, in three 16-byte vectors
        const int w0 = 3 * jb + half, w1 = w0 + 1;
        const uint32_t a = ring32(lane_at + (w0 >> 2) * 512 + (w0 & 3) * 4), b = ring32(lane_at + (w1 >> 2) * 512 + (w1 & 3) * 4);
        w[c][0] = __funnelshift_r(a, b, 16 * half);
        w[c][1] = b >> (16 * half);
      }
    }
#pragma unroll
    for (int i = 0; i < kWords; ++i) {
      swap_if(x & 1, w[0][i], w[1][i]);
      swap_if(x & 1, w[2][i], w[3][i]);
      swap_if(x & 2, w[0][i], w[2][i]);
      swap_if(x & 2, w[1][i], w[3][i]);
    }
  }
  // Which piece lane 4 g + t of a warp fetches first.
  __device__ static __forceinline__ int first_piece(int g, int t) {
    if constexpr (BITS == 4) return ((g >> 1) & 1) | (t & 2);
    else if constexpr (BITS == 8) return t;
    else return g >> 1;
  }
  __device__ static __forceinline__ void swap_if(int cond, uint32_t& a, uint32_t& b) {
    const uint32_t lo = cond ? b : a, hi = cond ? a : b;
    a = lo;
    b = hi;
  }

  // The 16 elements (eight pairs) of piece C, in element order, times the scale pair.
  template <int C, bool FP16, bool WIDE>
  __device__ __forceinline__ void decode(uint32_t lane_base, uint32_t s2, uint32_t (&v)[16], int at) const {
    const uint32_t(&q)[kWords] = w[C];
    if constexpr (BITS == 4) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        v[at + 4 * i] = lut32(entry_addr<4, 0, WIDE>(q[i], lane_base));
        v[at + 4 * i + 1] = lut32(entry_addr<4, 1, WIDE>(q[i], lane_base));
        v[at + 4 * i + 2] = lut32(entry_addr<4, 2, WIDE>(q[i], lane_base));
        v[at + 4 * i + 3] = lut32(entry_addr<4, 3, WIDE>(q[i], lane_base));
      }
    } else if constexpr (BITS == 8) {  // sixteen single lookups, merged in pairs
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[at + 2 * i] = prmt<0x7610>(lut32(entry_addr<8, 0, WIDE>(q[i], lane_base)), lut32(entry_addr<8, 1, WIDE>(q[i], lane_base)));
        v[at + 2 * i + 1] = prmt<0x7610>(lut32(entry_addr<8, 2, WIDE>(q[i], lane_base)), lut32(entry_addr<8, 3, WIDE>(q[i], lane_base)));
      }
    } else if constexpr (BITS == 2) {  // one byte = four elements = one 8-byte entry
      const uint2 a = lut64(entry_addr<2, 0, WIDE>(q[0], lane_base)), b = lut64(entry_addr<2, 1, WIDE>(q[0], lane_base));
      const uint2 c = lut64(entry_addr<2, 2, WIDE>(q[0], lane_base)), d = lut64(entry_addr<2, 3, WIDE>(q[0], lane_base));
      v[at] = a.x; v[at + 1] = a.y; v[at + 2] = b.x; v[at + 3] = b.y;
      v[at + 4] = c.x; v[at + 5] = c.y; v[at + 6] = d.x; v[at + 7] = d.y;
    } else if constexpr (BITS == 1) {  // one byte = eight elements = one 16-byte entry
      const uint4 a = lut128(entry_addr<1, 0, WIDE>(q[0], lane_base)), b = lut128(entry_addr<1, 1, WIDE>(q[0], lane_base));
      v[at] = a.x; v[at + 1] = a.y; v[at + 2] = a.z; v[at + 3] = a.w;
      v[at + 4] = b.x; v[at + 5] = b.y; v[at + 6] = b.z; v[at + 7] = b.w;
    } else {  // 3 bits: eight 6-bit pair fields of a 48-bit group, each moved to bits 7..12 (times 128)
      static_assert(BITS != 3 || Table<3>::kStride == 128, "field extraction assumes 128-byte table rows");
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int o = 6 * i;
        const uint32_t f = o + 6 <= 32 ? (o >= 7 ? q[0] >> (o - 7) : q[0] << (7 - o))
                           : o < 32    ? __funnelshift_r(q[0], q[1], o - 7)
                           : o - 32 >= 7 ? q[1] >> (o - 39) : q[1] << (39 - o);
        v[at + i] = lut32(lane_base + (f & (63u << 7)));
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) v[at + i] = mul_pair<FP16>(v[at + i], s2);
  }
};

// 16-row sub-tile of a 64-row tile that lane 4 g + t of an even or odd quarter collects.  PAIRS: sub-tiles apart by two,
// so that in a weight of alternating 32 gate rows and their 32 up rows both factors of an output are in one warp,
// two lanes apart (the plain product keeps 32 consecutive rows together: its stores are 1 % of 2048 x 28672 faster for it).
template <bool PAIRS>
__device__ __forceinline__ int sub_tile_of(int quarter, int t) {
  return PAIRS ? (quarter & 1) + 2 * (t >> 1) : 2 * (quarter & 1) + (t >> 1);
}

// Unit range of CTA `rank`: units are (tile, slab) pairs, a tile's slabs consecutive.
__device__ __forceinline__ int range_begin(const TcParams& p, int rank) {
  const int begin = tc_cut_begin(p.cut, rank);
  return p.split ? begin : p.k_slabs * begin;
}

// Position in the unit sequence.  Stepped, not divided out: the warps that issue copies and MMAs
// are single threads whose latency per block (two integer divisions cost ~300 cycles) was the
// pace of the whole kernel: 8192^2, 32 rows: 33.7 us.
struct Cursor {
  int ks, mt, nt;
  __device__ __forceinline__ Cursor(const TcParams& p, int unit) {
    const int tile = unit / p.k_slabs;
    ks = unit - tile * p.k_slabs;
    nt = tile / p.m_tiles;
    mt = tile - nt * p.m_tiles;
  }
  __device__ __forceinline__ bool next(const TcParams& p) {  // true at the first slab of a tile
    if (++ks < p.k_slabs) return false;
    ks = 0;
    if (++mt == p.m_tiles) {
      mt = 0;
      ++nt;
    }
    return true;
  }
};

// kTcSilu: out[m, n / 2] = silu(gate) * up of a weight whose rows alternate 32 gate rows and their 32 up rows, with the
// roundings of the plain product followed by silu_mul_kernel.  kTcNarrow: the plain product with batch tiles of at most
// 32 columns, whose owners fetch shares eight columns at a time: an instantiation of its own, because in the others that
// code made the compiler spill (80 registers) and large products up to 2 % slower (1000 rows of 22528 x 3072 111.4 us, 109.1
// without; 300 rows 39.9, 38.7).
enum TcForm { kTcPlain, kTcSilu, kTcNarrow };
constexpr int kTcNarrowColumns = 32;

template <int BITS, bool FP16, TcForm FORM>
__global__ void __launch_bounds__(kTcThreads, 1)
    gemm_lut_tc_kernel(const __grid_constant__ TcParams p, const __grid_constant__ InlineLut<BITS> inl,
                       const __grid_constant__ CUtensorMap x_map) {
  constexpr bool SILU = FORM == kTcSilu;
  using L = Layout<BITS>;
  constexpr bool WIDE = kTcWideTable<BITS>;
  using T = Table<BITS, WIDE>;
  constexpr int KSB = L::KSB;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t raw = smem_addr(smem_raw);
  if (raw != p.smem_base) {
    if (threadIdx.x == 0) atomicOr(p.status, kTcStatusSmemLayout);
    return;
  }
  // x, the workspace and out are only touched after griddepcontrol.wait; codes and table are not
  // written by the kernel before
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);  // uniform for the compiler
  const int S = 1 << p.stages_log2;
  const uint32_t full = p.bar_addr, empty = full + 8 * kTcMaxStages,
                 c_full = empty + 8 * kTcMaxStages, c_empty = c_full + 8 * kTcMaxCodeSlots,
                 acc_full = c_empty + 8 * kTcMaxCodeSlots, acc_empty = acc_full + 16, acc_last = acc_empty + 16, tmem_slot = acc_last + 8,
                 launch_slot = tmem_slot + 4;
  // Waits go to CTAs of lower block index, which the GPU starts first: rank r's successors in
  // the unit sequence are the blocks before it.
  const int rank = (int)gridDim.x - 1 - (int)blockIdx.x;
  const int u0 = range_begin(p, rank), u1 = range_begin(p, rank + 1);
  bool timed_out = false;

  // Start-up, everything at once: the code producers set up their own barriers and request the first codes, the x
  // producer sets up the others, the MMA warp allocates tensor memory, and all other warps fill the table.
  // (One after another, with a CTA-wide barrier ahead of the copies and one behind the table: the first codes were
  // there 2.6 us after the start of the CTA.)
  const size_t tile_bytes = (size_t)p.k_slabs * L::kSlabBytes;  // one 64-row tile
  // two producer warps, a slab each in turn: wait, expectation and two copies take one of them ~300 cycles
  auto request_codes = [&](const Cursor& c, int slot) {
    const uint8_t* src = p.tiled + 2 * c.nt * tile_bytes + (size_t)c.ks * L::kSlabBytes;
    const bool second = 2 * c.nt + 1 < p.row_tiles;
    const uint32_t bar = c_full + 8 * slot, dst = p.c_addr[slot];
    if (elect_one()) {
      mbar_expect(bar, (uint32_t)L::kSlabBytes * (second ? 2 : 1));
      bulk_copy(dst, src, L::kSlabBytes, bar);
      if (second) bulk_copy(dst + (uint32_t)L::kSlabBytes, src + tile_bytes, L::kSlabBytes, bar);
    }
  };
  const bool code_producer = warp >= kTcFirstCodeWarp && warp < kTcXWarp;
  Cursor c(p, code_producer ? u0 + warp - kTcFirstCodeWarp : u0);  // the producers' position
  auto init_fence = [] {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
  };
  if (code_producer) {
    const int first = warp - kTcFirstCodeWarp;
    const int mine = first + kTcCodeWarps * lane;
    if (mine < p.code_slots) {
      mbar_init(c_full + 8 * mine, 1);
      mbar_init(c_empty + 8 * mine, KSB == 1 ? 4 : kTcDequantWarps);  // one set, or all
    }
    init_fence();
    for (int slot = first; slot < p.code_slots; slot += kTcCodeWarps) {  // the first use of every slot
      if (u0 + slot < u1) request_codes(c, slot);
      for (int i = 0; i < kTcCodeWarps; ++i) c.next(p);
    }
  } else if (warp == kTcXWarp) {
    if (lane == 0) asm volatile("prefetch.tensormap [%0];" ::"l"(&x_map) : "memory");
    if (lane < S) {
      mbar_init(full + 8 * lane, 5);  // x has arrived, and the four warps of a set have stored A
      mbar_init(empty + 8 * lane, 1);
    }
    if (lane < kTcAccumulators) {
      mbar_init(acc_full + 8 * lane, 1);
      mbar_init(acc_empty + 8 * lane, kTcEpilogueWarps);
    }
    if (lane == 31) mbar_init(acc_last, 2);  // the last MMAs, and the launch number in shared memory
    init_fence();
  } else {
    if (warp == kTcMmaWarp) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"((uint32_t)kTcTmemColumns)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    constexpr int kFillThreads = kTcThreads - 32 * (kTcCodeWarps + 1);
    const int tid = warp == kTcMmaWarp ? kFillThreads - 32 + lane : threadIdx.x;
    auto fill = [&](auto word) {
      if constexpr (BITS == 4 || BITS == 2 || BITS == 1) fill_table_unrolled<BITS, WIDE, kFillThreads>(p.table_addr, word, tid);
      else fill_table<BITS, WIDE>(p.table_addr, kFillThreads, word, tid);
    };
    if (p.lut == nullptr) fill([&](int i) { return inl.w[i]; });
    else fill([&](int i) { return __ldg(reinterpret_cast<const uint32_t*>(p.lut) + i); });
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // All of tensor memory is allocated, so it starts at address 0; a constant keeps the MMAs' operands
  // in uniform registers.
  constexpr uint32_t tmem_base = 0;
  const uint32_t acc_base = tmem_base + 32 * S;  // A stages of 32 columns, then the accumulators
  auto blocks_of = [&](int ks) { return KSB == 1 ? 1 : min(KSB, p.k_blocks - ks * KSB); };

  // ---- epilogue of one tile segment [begin, end) of slabs, by `parts` warps per 32-row quarter ----
  auto epilogue = [&](int tile, int begin, int end, uint32_t acc, int part, auto parts_c, int launch) {
    constexpr int parts = decltype(parts_c)::value;
    const int nt = tile / p.m_tiles, mt = tile - nt * p.m_tiles;
    const int quarter = warp & 3;
    const int row = nt * kTcTileRows + (SILU ? 64 * (quarter >> 1) + 16 * sub_tile_of<SILU>(quarter, lane & 3) + 8 * (lane & 1) + (lane >> 2)
                                             : 32 * quarter + 8 * (lane & 3) + (lane >> 2));
    const size_t slot = (size_t)p.n_tile * kTcTileRows;
    const uint32_t taddr = acc + ((uint32_t)(quarter * 32) << 16);
    const int tile_end = (tile + 1) * p.k_slabs;
    int last_rank = rank;  // ranks rank + 1 .. last_rank hold the rest of the tile
    if (begin == 0 && end < p.k_slabs)
      while (range_begin(p, last_rank + 1) < tile_end) ++last_rank;
    // flag of 16 columns of 32 rows: one warp publishes them
    auto flag = [&](int of_rank, int c0) { return p.flags + of_rank * kTcFlagsPerRank + (c0 >> 4) * 4 + quarter; };
    auto await_shares = [&](int c0) {
      for (int o = rank + 1 + lane; o <= last_rank; o += 32) {  // a lane per share
        int* const f = flag(o, c0);
        unsigned long long t0 = 0;
        for (uint32_t spin = 0;; ++spin) {
          int set;
          asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(set) : "l"(f) : "memory");
          if (set == launch) break;
          if ((spin & 255u) == 255u) {
            unsigned long long now;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            if (t0 == 0) t0 = now;
            else if (now - t0 > 2000000000ull) { timed_out = true; break; }
          }
        }
      }
      timed_out = __any_sync(0xffffffffu, timed_out);
      __syncwarp();  // the lanes' reads below come after every polling lane's acquire (a vote orders no memory)
    };
    // Several shares of a tile of few columns: eight columns at a time, so that every warp has some and the loads of four
    // shares are in flight (32 rows: 5120 x 3072 8.97 us -> 8.58, 256 x 20480 11.2 -> 9.7; with one share, or with so many
    // columns that the warps go round twice, 16 at a time are better: 48 rows of 11264 x 3072 11.8 against 12.6).  Two
    // warps then wait for one flag.
    if (FORM == kTcNarrow && parts > 1 && last_rank > rank + 1) {
      static_assert(parts == 1 || kTcNarrowColumns <= 8 * parts, "eight columns a warp");
      if (const int c0 = 8 * part; c0 < p.n_tile) {
        uint32_t acc8[8];
        tmem_load8(taddr + (uint32_t)c0, acc8);
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(acc8[j]);
        await_shares(c0);
        for (int o = rank + 1; o <= last_rank; o += 4) {  // in rank order
          const float* theirs = p.partial + o * slot + (size_t)c0 * kTcTileRows + 32 * quarter + lane;
          float t[4][8];
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int j = 0; j < 8; ++j) t[q][j] = o + q <= last_rank ? __ldcg(theirs + q * slot + j * kTcTileRows) : 0.f;
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] += t[q][j];
        }
        const int b0 = mt * p.n_tile + c0;
        if (row < p.n) {
          uint16_t* dst = p.out + (size_t)b0 * p.n + row;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (b0 + j < p.m) dst[(size_t)j * p.n] = from_float<FP16>(v[j]);
        }
      }
      return;
    }
    for (int c0 = 16 * part; c0 < p.n_tile; c0 += 16 * parts) {
      uint32_t acc16[16];
      tmem_load16(taddr + (uint32_t)c0, acc16);
      const size_t at = (size_t)c0 * kTcTileRows + 32 * quarter + lane;
      if (begin != 0) {
        float* mine = p.partial + rank * slot + at;
#pragma unroll
        for (int j = 0; j < 16; ++j) __stcg(mine + j * kTcTileRows, __uint_as_float(acc16[j]));
      } else {
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(acc16[j]);
        if (last_rank > rank) {
          await_shares(c0);
          // in rank order; two shares' loads are in flight at a time
          for (int o = rank + 1; o <= last_rank; o += 2) {
            const float* theirs = p.partial + o * slot + at;
            float t[32];
#pragma unroll
            for (int j = 0; j < 16; ++j) t[j] = __ldcg(theirs + j * kTcTileRows);
            if (o < last_rank) {
#pragma unroll
              for (int j = 0; j < 16; ++j) t[16 + j] = __ldcg(theirs + slot + j * kTcTileRows);
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] += t[j];
            if (o < last_rank) {
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] += t[16 + j];
            }
          }
        }
        if constexpr (SILU) {
          const int b0 = mt * p.n_tile + c0;
          // a gate lane takes the even columns and the up lane two lanes on the odd ones; each sends the other its factor
          auto rnd = [](float x) { return to_float<FP16>(from_float<FP16>(x)); };
          const bool is_up = (lane & 2) != 0;
          const int width = p.n / 2;
          float gate[8], up[8], act[8];
          bool exact = false;  // some quotient has to be a division (silu_quotient)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float own = rnd(is_up ? v[2 * j + 1] : v[2 * j]);
            const float other = __shfl_xor_sync(0xffffffffu, rnd(is_up ? v[2 * j] : v[2 * j + 1]), 2);
            gate[j] = is_up ? other : own;
            up[j] = is_up ? own : other;
            exact = silu_quotient(gate[j], act[j]) || exact;
          }
          if (exact) {
#pragma unroll
            for (int j = 0; j < 8; ++j) act[j] = gate[j] / (1.f + __expf(-gate[j]));
          }
          uint16_t* dst = p.out + (size_t)(b0 + is_up) * width + (nt * 2 + (quarter >> 1)) * 32 + 16 * (quarter & 1) + 8 * (lane & 1) + (lane >> 2);
          if (row < p.n) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (b0 + 2 * j + is_up < p.m) dst[(size_t)(2 * j) * width] = from_float<FP16>(rnd(act[j]) * up[j]);
          }
        } else if (row < p.n) {
          const int b0 = mt * p.n_tile + c0;
          uint16_t* dst = p.out + (size_t)b0 * p.n + row;
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (b0 + j < p.m) dst[(size_t)j * p.n] = from_float<FP16>(v[j]);
        }
      }
    }
    if (begin != 0) {  // publish: no barrier, every warp vouches for its own columns
      __syncwarp();
      __threadfence();
      const int c0 = 16 * (part + lane * parts);
      if (c0 < p.n_tile) asm volatile("st.relaxed.gpu.global.s32 [%0], %1;" ::"l"(flag(rank, c0)), "r"(launch) : "memory");
    }
  };
  constexpr int kSets = kTcDequantWarps / 4;
  // the CTA's last tile segment
  const int last_tile = u1 > u0 ? (u1 - 1) / p.k_slabs : 0;
  const int last_begin = max(u0 - last_tile * p.k_slabs, 0), last_end = u1 - last_tile * p.k_slabs;
  const int segments = u1 > u0 ? last_tile - u0 / p.k_slabs + 1 : 0;
  auto last_epilogue = [&](int part) {
    if (!mbar_wait(acc_last, 0)) timed_out = true;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    epilogue(last_tile, last_begin, last_end, acc_base + (segments - 1) % kTcAccumulators * p.n_tile, part,
             std::integral_constant<int, kSets + 1>{}, (int)ring32(launch_slot));
  };

  if (segments == 0) {
    // more CTAs than units
  } else if (code_producer) {
    // ---------------- code producer ----------------
    const int first = warp - kTcFirstCodeWarp;
    int slot = first, phase = 1;  // the first round is on its way
    asm volatile("griddepcontrol.wait;" ::: "memory");  // from here on a slot is freed by way of x
    for (int u = u0 + first + p.code_slots; u < u1; u += kTcCodeWarps) {
      if (!mbar_wait(c_empty + 8 * slot, phase ^ 1)) { timed_out = true; break; }
      request_codes(c, slot);
      for (int i = 0; i < kTcCodeWarps; ++i) c.next(p);
      if ((slot += kTcCodeWarps) >= p.code_slots) {
        slot -= p.code_slots;
        phase ^= 1;
      }
    }
  } else if (warp == kTcXWarp) {
    // ---------------- x producer ----------------
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int i = 0;
    for (int u = u0; u < u1 && !timed_out; ++u, c.next(p)) {
      const int nb = blocks_of(c.ks);
      for (int jb = 0; jb < nb; ++jb, ++i) {
        const int s = i & (S - 1);
        const uint32_t dst = p.b_addr[s], bar = full + 8 * s;
        if (!mbar_wait(empty + 8 * s, ((i >> p.stages_log2) & 1) ^ 1)) { timed_out = true; break; }
        if (elect_one()) {
          mbar_expect(bar, (uint32_t)p.n_tile * 128);
          tma_load_2d(dst, &x_map, (c.ks * KSB + jb) * kBlock, c.mt * p.n_tile, bar);
        }
      }
    }
  } else if (warp == kTcMmaWarp) {
    // ---------------- MMA issuer ----------------
    asm volatile("griddepcontrol.wait;" ::: "memory");  // a stage is full once x is in it
    // instruction descriptor: fp32 accumulate, A and B both bf16 (format 1) or both fp16
    // (format 0), both K-major, N = n_tile, M = 128
    constexpr uint32_t kFormat = FP16 ? 0u : 1u;
    const uint32_t idesc = (1u << 4) | (kFormat << 7) | (kFormat << 10) | ((uint32_t)(p.n_tile >> 3) << 17) | ((128u >> 4) << 24);
    int i = 0, ks = u0 % p.k_slabs;
    for (int seg = 0, u = u0; seg < segments && !timed_out; ++seg) {
      const int a = seg % kTcAccumulators;
      const uint32_t acc = acc_base + a * p.n_tile;
      if (!mbar_wait(acc_empty + 8 * a, ((seg / kTcAccumulators) & 1) ^ 1)) { timed_out = true; break; }
      uint32_t accumulate = 0;
      for (bool more = true; more && !timed_out;) {
        const int nb = blocks_of(ks);
        if (++ks == p.k_slabs) { ks = 0; more = false; }
        if (++u == u1) more = false;
        for (int jb = 0; jb < nb; ++jb, ++i) {
          const int s = i & (S - 1);
          const uint32_t parity = (i >> p.stages_log2) & 1;
          const uint64_t b_desc = kDescBase | (p.b_addr[s] >> 4);
          if (!mbar_wait(full + 8 * s, parity)) { timed_out = true; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          // four K = 16 slices of the 64-column block: 8 columns of A, 32 bytes of x (2 in the
          // descriptor's 16-byte units) apart
          if (elect_one()) {
            umma_f16_ts(acc, tmem_base + 32 * s, b_desc, idesc, accumulate);
            umma_f16_ts(acc, tmem_base + 32 * s + 8, b_desc + 2, idesc, 1);
            umma_f16_ts(acc, tmem_base + 32 * s + 16, b_desc + 4, idesc, 1);
            umma_f16_ts(acc, tmem_base + 32 * s + 24, b_desc + 6, idesc, 1);
            umma_commit(empty + 8 * s);  // the stage may be refilled once these MMAs have read it
          }
          accumulate = 1;
        }
      }
      // the last segment has a barrier of its own, for the dequantising warps too, which have
      // not followed acc_full's phases
      if (elect_one()) umma_commit(seg + 1 < segments ? acc_full + 8 * a : acc_last);
    }
  } else if (warp >= kTcDequantWarps) {
    // ---------------- epilogue ----------------
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int launch = 0;  // the same in every CTA: it moves on once all have read it
    if (p.split) {
      unsigned long long count;
      asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(count) : "l"(p.launches) : "memory");
      launch = (int)(count >> kTcLaunchShift) + 1;
    }
    if (warp == kTcDequantWarps && lane == 0) {  // for the warps that share the last epilogue
      asm volatile("st.shared.u32 [%0], %1;" ::"r"(launch_slot), "r"(launch) : "memory");
      mbar_arrive(acc_last);
    }
    int u = u0;
    for (int seg = 0; seg + 1 < segments; ++seg) {
      const int tile = u / p.k_slabs, begin = u - tile * p.k_slabs;
      const int a = seg % kTcAccumulators;
      if (!mbar_wait(acc_full + 8 * a, (seg / kTcAccumulators) & 1)) timed_out = true;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      epilogue(tile, begin, p.k_slabs, acc_base + a * p.n_tile, 0, std::integral_constant<int, 1>{}, launch);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty + 8 * a);
      u = (tile + 1) * p.k_slabs;
    }
    last_epilogue(kSets);
  } else {
    // ---------------- dequantise ----------------
    const int set = warp >> 2, quarter = warp & 3;
    const int g = lane >> 2, t = lane & 3;
    const int r = sub_tile_of<SILU>(quarter, t), half = t & 1;  // the lane's row: 16 r + 8 half + g of its 64-row tile
    const int x = RowCodes<BITS>::first_piece(g, t);
    const uint32_t slab_off = (quarter >> 1) * (uint32_t)L::kSlabBytes;
    const uint32_t scale_off = slab_off + L::kCodeBytes + g * 16 + r * 4;
    const uint32_t lane_base = p.table_addr + T::lane_offset(lane);
    const uint32_t a_lane = tmem_base + ((uint32_t)(quarter * 32) << 16);
    // Codes and scale pair of the set's next block -> its number in the CTA's sequence; -1 at the end.
    // A warp may only skip the barriers of stages and code slots that it never uses: waiting
    // for a phase while the one before it is still open would succeed at once.  Stages, and
    // slots of slabs with one block, always belong to the same set (their number is a multiple
    // of four); the other slabs are seen by every warp.
    int u = KSB == 1 ? u0 + set : u0, slot = KSB == 1 ? set : 0, c_phase = 0;
    int ks = KSB == 1 ? 0 : u0 % p.k_slabs, i = 0;
    // Second uses of a code slot or stage wait for MMAs, hence for x; the first ones do not, and fill
    // tensor memory while the kernel before is still running.
    auto wait_for_x = [&] { asm volatile("griddepcontrol.wait;" ::: "memory"); };
    uint32_t held = 0;  // the barrier of the slot that the last fetch read, to be handed back
    auto fetch = [&](RowCodes<BITS>& codes, uint32_t& s2) -> int {
      while (u < u1) {
        const int nb = KSB == 1 ? 1 : blocks_of(ks);
        const int jb = KSB == 1 ? 0 : (set - i) & (kSets - 1);  // the set's block of this slab, if it has one
        const uint32_t slab = p.c_addr[slot], bar = c_empty + 8 * slot;
        if (!mbar_wait(c_full + 8 * slot, c_phase)) { timed_out = true; return -1; }
        const bool mine = jb < nb;
        if (mine) {
          codes.load(slab + slab_off, jb, g, r, half, x);
          const uint32_t scw = ring32(slab + scale_off + jb * 128);
          s2 = half ? prmt<0x3232>(scw, 0u) : prmt<0x1010>(scw, 0u);
          held = bar;
        } else if (lane == 0) {
          mbar_arrive(bar);
        }
        const int block = KSB == 1 ? u - u0 : i + jb;
        if constexpr (KSB == 1) {
          u += kSets;
          slot += kSets;
          if (slot >= p.code_slots) { slot -= p.code_slots; c_phase ^= 1; wait_for_x(); }
        } else {
          ++u;
          i += nb;
          if (++ks == p.k_slabs) ks = 0;
          if (++slot == p.code_slots) { slot = 0; c_phase ^= 1; wait_for_x(); }
        }
        if (mine) return block;
      }
      return -1;
    };
    // Hands the slot back.  The copy that refills it writes through the async proxy, which a barrier arrival
    // alone does not order after the reads above: with an arrival right behind them they were still on
    // their way (queued behind stores to tensor memory, with the tensor pipe busy) when the new codes came in,
    // about once in a million blocks at 1000 rows of 22528 x 3072.  Hence the fence, and it stands behind the
    // block's first store to tensor memory, which cannot issue before codes and scale are in registers: a fence
    // right behind the reads waits for them (48 rows of 11264 x 3072 13.9 us against 12.5, 2048 of 28672 x 4096
    // 362 against 344; where 128 batch rows leave a set one slot, 8192^2, 26.0 against 26.3).
    auto release = [&] {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(held);
    };
    // A block's stores to tensor memory are awaited and handed over while the lookups of the next
    // one are in flight, whose codes were fetched between the two halves of this one.
    auto hand_over = [&](int s) {
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(full + 8 * s);
    };
    RowCodes<BITS> codes;
    uint32_t s2 = 0;
    int block = fetch(codes, s2), stored = -1;
    while (block >= 0) {
      const int s = block & (S - 1);
      uint32_t v[16];
      codes.template decode<0, FP16, WIDE>(lane_base, s2, v, 0);
      codes.template decode<1, FP16, WIDE>(lane_base, s2, v, 8);
      if (stored >= 0) hand_over(stored);
      if (block == S + set) wait_for_x();  // the set's first second use
      if (!mbar_wait(empty + 8 * s, ((block >> p.stages_log2) & 1) ^ 1)) { timed_out = true; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      tmem_store16(a_lane + 32 * s, v);
      release();
      codes.template decode<2, FP16, WIDE>(lane_base, s2, v, 0);
      codes.template decode<3, FP16, WIDE>(lane_base, s2, v, 8);
      block = fetch(codes, s2);
      tmem_store16(a_lane + 32 * s + 16, v);
      stored = s;
    }
    if (stored >= 0 && !timed_out) hand_over(stored);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    last_epilogue(set);
  }
  if (timed_out && lane == 0) atomicOr(p.status, kTcStatusTimeout);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  if (__syncthreads_or(timed_out)) {
    // A role gave up: copies and MMAs may still be on their way into shared and tensor memory, and their
    // barriers no longer tell.  They take microseconds; the block keeps its memory for ten milliseconds.
    if (threadIdx.x == 0) {
      unsigned long long t0, now;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
      for (uint32_t spin = 0; spin < (1u << 20); ++spin) {
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if (now - t0 > 10000000ull) break;
        __nanosleep(1000);
      }
    }
    __syncthreads();
  }
  // Every CTA of a launch that cuts tiles has units, so this thread has waited for the launch before, and
  // every warp of the CTA has read the count.
  if (p.split && threadIdx.x == 0)
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p.launches),
                 "l"(rank == 0 ? (1ull << kTcLaunchShift) - (gridDim.x - 1) : 1ull)
                 : "memory");
  if (warp == kTcMmaWarp) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kTcTmemColumns) : "memory");
  }
}

// ---- host side ----------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int encode_fn(EncodeTiledFn* out) {
  static std::atomic<EncodeTiledFn> found{nullptr};
  EncodeTiledFn fn = found.load(std::memory_order_acquire);
  if (fn == nullptr) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    FDK_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres));
    FDK_CHECK_ARG(qres == cudaDriverEntryPointSuccess && sym != nullptr, FDK_ERR_CUDA, "cuTensorMapEncodeTiled not found");
    fn = (EncodeTiledFn)sym;
    found.store(fn, std::memory_order_release);
  }
  *out = fn;
  return FDK_OK;
}

inline uint32_t round_up(uint32_t v, uint32_t a) { return (v + a - 1) / a * a; }

// Shared memory: barriers, the table (a wide one at a multiple of 64 KB of the shared window, with
// buffers on both sides of it), the x stages (1024-byte aligned for the swizzle), the code
// ring: as many slots as fit, up to sixteen (68 KB of 4-bit codes in flight per SM; four are
// the least, see the dequantising warps).  Returns the dynamic size, or 0 if nothing fits.
template <int BITS>
size_t plan_tc_smem(uint32_t base, uint32_t limit, TcParams& p) {
  using L = Layout<BITS>;
  using T = Table<BITS, kTcWideTable<BITS>>;
  const uint32_t end = base + limit;
  uint32_t low = round_up(base, 128);  // next free address below the table
  p.smem_base = base;
  p.bar_addr = low;
  low += 512;
  p.table_addr = round_up(low, kTcWideTable<BITS> ? 65536 : 128);
  uint32_t high = p.table_addr + T::kBytes, used = high;
  if (high > end) return 0;
  auto take = [&](uint32_t bytes, uint32_t align) -> uint32_t {
    uint32_t a = round_up(low, align);
    if (a + bytes <= p.table_addr) { low = a + bytes; return a; }
    a = round_up(high, align);
    if (a + bytes > end) return 0;
    high = used = a + bytes;
    return a;
  };
  for (int s = 0; s < (1 << p.stages_log2); ++s)
    if ((p.b_addr[s] = take((uint32_t)p.n_tile * 128, 1024)) == 0) return 0;
  int slots = 0;
  while (slots < kTcMaxCodeSlots && (p.c_addr[slots] = take(round_up(2 * L::kSlabBytes, 128), 128)) != 0) ++slots;
  p.code_slots = slots & ~3;
  return p.code_slots >= 4 ? used - base : 0;
}

template <int BITS, bool FP16, TcForm FORM>
int launch_tc(TcParams p, const void* lut_host, const CUtensorMap& map, int grid, bool pdl, cudaStream_t stream) {
  InlineLut<BITS> inl;
  if (lut_host != nullptr) {
    memcpy(inl.w, lut_host, sizeof(inl.w));
    p.lut = nullptr;
  } else {
    memset(inl.w, 0, sizeof(inl.w));
  }
  uint32_t base = 0;
  if (int st = dynamic_smem_base(&base)) return st;
  DeviceInfo di;
  if (int st = device_info(&di)) return st;
  size_t smem = plan_tc_smem<BITS>(base, (uint32_t)di.max_smem_optin, p);
  // 4 bits: eight stages of 128 batch rows leave four code slots, one a set, which then waits for every copy; with four
  // stages there are sixteen (128 rows of 8192^2 24.8 us -> 21.75, of 3072^2 12.9 -> 11.8).  Eight slots beside
  // eight stages of 112 rows are better than that (20.0 against 20.95), and so are the four at 8 bits, whose blocks take
  // twice as long (27.2 against 28.1).
  if (BITS == 4 && p.stages_log2 == 3 && p.code_slots < 8) {
    p.stages_log2 = 2;
    smem = plan_tc_smem<BITS>(base, (uint32_t)di.max_smem_optin, p);
  }
  FDK_CHECK_ARG(smem != 0, FDK_ERR_CUDA, "no shared-memory plan fits %d bytes", di.max_smem_optin);
  auto kernel = gemm_lut_tc_kernel<BITS, FP16, FORM>;
  static std::atomic<bool> allowed[64] = {};
  if (int st = allow_all_smem(kernel, allowed, di)) return st;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kTcThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  FDK_CUDA(cudaLaunchKernelEx(&cfg, kernel, p, inl, map));
  return FDK_OK;
}

int gemm_rows(const void* x, const void* tiled, const void* lut, const void* lut_host, void* out, int m, int n,
              int k, int bits, bool fp16, bool silu, void* workspace, size_t workspace_bytes, int sm_count, bool pdl,
              cudaStream_t stream) {
  EncodeTiledFn encode = nullptr;
  if (int st = encode_fn(&encode)) return st;
  const TiledDims d = tiled_dims(n, k, bits);
  TcParams p{};
  p.tiled = (const uint8_t*)tiled;
  p.lut = lut;
  p.out = (uint16_t*)out;
  p.status = (int*)workspace + kStatusWord;
  p.m = m;
  p.n = n;
  p.m_tiles = (m + kTcMaxBatch - 1) / kTcMaxBatch;
  p.n_tile = (int)round_up((uint32_t)((m + p.m_tiles - 1) / p.m_tiles), 16);
  p.row_tiles = d.row_tiles;
  p.k_blocks = k / kBlock;
  p.k_slabs = d.k_slabs;
  const long long tiles = (long long)((n + kTcTileRows - 1) / kTcTileRows) * p.m_tiles, units = tiles * d.k_slabs;
  p.tiles = (int)tiles;
  // eight A stages fit tensor memory beside two accumulators of 128 columns, four beside two of 192
  p.stages_log2 = p.n_tile <= 128 ? 3 : 2;
  p.flags = (int*)((uint8_t*)workspace + kTcFlagsOffset);
  p.launches = (unsigned long long*)((uint8_t*)workspace + kTcLaunchesOffset);
  p.partial = (float*)((uint8_t*)workspace + kTcPartialOffset);
  // One CTA per SM.  Ranges cut tiles where the workspace has room for every CTA's partial sums.
  // Where a tile is shared by many CTAs its owner reads all their sums (about 10 cycles per CTA and
  // batch row), which has to stay below what the CTAs save (max(2 n_tile, 250) cycles per block):
  // the total  units t / G + G / tiles 10 n_tile  is least at the G below.
  int grid = sm_count;
  const size_t slot_bytes = (size_t)p.n_tile * kTcTileRows * sizeof(float);
  const size_t room = workspace_bytes > kTcPartialOffset ? (workspace_bytes - kTcPartialOffset) / slot_bytes : 0;
  if (tiles < grid) {
    const double block = 2.0 * p.n_tile > 250.0 ? 2.0 * p.n_tile : 250.0;
    const double best = std::sqrt((double)p.k_blocks * tiles * block * tiles / (10.0 * p.n_tile));
    const long long four = (long long)p.k_blocks * tiles / 4;  // at least four blocks each
    if (best < grid) grid = (int)best;
    if (four < grid) grid = (int)four;
    if (units < grid) grid = (int)units;
    if (grid < tiles) grid = (int)tiles;
  }
  p.split = room >= (size_t)grid;
  if (!p.split && tiles < grid) grid = (int)tiles;
  p.cut = make_tc_cut((int)(p.split ? units : tiles), grid);
  CUtensorMap map;
  const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)m};
  const cuuint64_t strides[1] = {(cuuint64_t)k * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)p.n_tile};
  const cuuint32_t elem[2] = {1, 1};
  CUresult r = encode(&map, fp16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)x, dims,
                      strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  FDK_CHECK_ARG(r == CUDA_SUCCESS, FDK_ERR_CUDA, "cuTensorMapEncodeTiled failed with %d", (int)r);
  auto launch = [&](auto bits_c) {
    constexpr int BITS = decltype(bits_c)::value;
    if (silu) return launch_tc<BITS, false, kTcSilu>(p, lut_host, map, grid, pdl, stream);
    if (p.n_tile <= kTcNarrowColumns)
      return fp16 ? launch_tc<BITS, true, kTcNarrow>(p, lut_host, map, grid, pdl, stream)
                  : launch_tc<BITS, false, kTcNarrow>(p, lut_host, map, grid, pdl, stream);
    return fp16 ? launch_tc<BITS, true, kTcPlain>(p, lut_host, map, grid, pdl, stream)
                : launch_tc<BITS, false, kTcPlain>(p, lut_host, map, grid, pdl, stream);
  };
  switch (bits) {
    case 1: return launch(std::integral_constant<int, 1>{});
    case 2: return launch(std::integral_constant<int, 2>{});
    case 3: return launch(std::integral_constant<int, 3>{});
    case 4: return launch(std::integral_constant<int, 4>{});
    default: return launch(std::integral_constant<int, 8>{});
  }
}

}  // namespace

// Batches above 16 rows.  Called by fdk_linear_lut and fdk_linear_lut_silu (silu: bf16, n a multiple of 64).  One launch, unless its units, and steps beyond
// them, would not fit 32 bits (100 thousand rows of 262080 x 65536): then one after another for as many whole
// batch tiles as do.
int gemm_lut_tc(const void* x, const void* tiled, const void* lut, const void* lut_host, void* out, int m, int n,
                int k, int bits, bool fp16, bool silu, void* workspace, size_t workspace_bytes, int sm_count, bool pdl,
                cudaStream_t stream) {
  const long long per_batch_tile = (long long)((n + kTcTileRows - 1) / kTcTileRows) * tiled_dims(n, k, bits).k_slabs;
  const long long most = ((1ll << 30) / per_batch_tile) * kTcMaxBatch;
  FDK_CHECK_ARG(most > 0, FDK_ERR_SHAPE, "n=%d, k=%d: too many slabs", n, k);
  for (long long m0 = 0; m0 < m; m0 += most) {
    const int rows = m - m0 < most ? (int)(m - m0) : (int)most;
    if (int st = gemm_rows((const uint16_t*)x + (size_t)m0 * k, tiled, lut, lut_host, (uint16_t*)out + (size_t)m0 * (silu ? n / 2 : n),
                           rows, n, k, bits, fp16, silu, workspace, workspace_bytes, sm_count, pdl, stream))
      return st;
  }
  return FDK_OK;
}

}  // namespace fdk
