// BSR SpMM for 16x16 bf16 blocks (and 8x8, 32x32: Shape below) on the Blackwell tensor cores:
// TMA (cp.async.bulk.tensor) -> shared memory -> tcgen05.mma -> TMEM -> tcgen05.ld.
//
// Reference arithmetic (ThreadPerOutputBSRSpMMPattern, SparseWaveToGPU.cpp:560-665):
//   C[br*16 + r, j] = sum over blocks bp of block row br, sum over lc:
//                     bv[bp][r][lc] * B[bci[bp]*16 + lc, j]
// with bf16 operands, f32 accumulation and one rounding to bf16 at the store.
//
// Mapping to the MMA.  A 16-row block would waste the M dimension (64 or 128)
// of tcgen05.mma, so the product is formed transposed: for one block row and
// 128 right-hand-side columns,
//   D[m, r] (+)= sum_k  Bt[m, k] * At[k, r],   m = column, k = lc,
// one tcgen05.mma of shape M=128, N=16, K=16 per nonzero block, all blocks of
// the block row accumulating into one 128-lane x 16-column f32 tile in TMEM.
// A unit of work is one block row and a tile of 128 or 256 right-hand-side
// columns, i.e. one or two such accumulators side by side in TMEM, so that each
// block and each block-column index is fetched once per tile.
//   - MMA operand A = a 16 x 128 slab B[bci*16 .. +16, n .. n+128).  Row k is
//     contiguous along m: MN-major.  TMA boxes of 64 columns x 16 rows with the
//     128-byte swizzle land it as the canonical MN-major SWIZZLE_128B layout
//     (128-byte rows, 1024 bytes between groups of 8 k rows = stride byte
//     offset, 2048 bytes between 64-column groups = leading byte offset).  A
//     tile of whole groups is one copy (a map of 64 columns x rows x groups).
//   - MMA operand B = the block itself, [r][lc] row-major: K-major.  A TMA box
//     of 16 columns with the 32-byte swizzle over the block values viewed as a
//     (nnzb*16) x 16 matrix lands it as the canonical K-major SWIZZLE_32B layout
//     (32-byte rows, 256 bytes between groups of 8 rows = stride byte offset).
//     Both accumulators' MMAs read the same copy.
//
// Pipeline.  Persistent CTAs, three (256 columns) to five per SM, walk the units.  A stage holds a group of four 16 x 16
// blocks (two of 32 x 32, one with 256 columns; eight of 8 x 8) with their slabs.  Lanes 0 of warps 4 - 7 copy: each takes its
// blocks of every group, block columns held 32 at a time in the warp's lanes and requested ahead.  Lane 0 of warp 8 issues the
// group's MMAs and lets tcgen05.commit arrive on `empty`.  There are two sets of accumulators: while warps 0 - 3 read one with tcgen05.ld,
// round to bf16 and store C, the MMAs of the next unit fill the other.
//
// What bounds it: no unit is at its limit on 1,024 block rows of 51, N = 512 (ncu, 64 us: 913 MB from L2 at 14.2 TB/s, which keeps
// L2's ports to the crossbar busy 61 % of the time and the SMs' intake 41 %; shared memory read by the tensor cores 44 %, tensor
// pipe 10 %, HBM 9 %).  The CTAs wait for their copies, and beside them pay the fixed cost of a step: a stage with one MMA takes its
// thread some 500 clocks and its copies 300 (wait, arrive, issue, commit), whatever its size.  Hence groups, several copying
// warps and persistence: with one block per stage, one copying thread and a CTA per unit, 3,419 block rows of 8, N = 128 took 29.6
// us (now 19.0), 847 of 16, N = 256 20.0 (15.2), 128 of 32, N = 512 21.3 (12.2), 1,024 of 51, N = 512 65.6 (61.8).  Tried: a CTA per
// unit with these stages (68 on the last), 1 or 2 CTAs per SM with deeper rings (142, 77), two chains of accumulators (no change).
//
// Every mbarrier wait is bounded: when one runs out the kernel raises the
// status word, frees its TMEM columns and returns.
#include <cuda.h>
#include <cuda_bf16.h>

#include <atomic>
#include <cstdio>

#include "swb_chain.cuh"
#include "swb_index.h"
#include "swb_kernels.h"

namespace swb {
namespace {

constexpr int HALF_N = 128;                  // right-hand-side columns of an MMA (M); a CTA takes one or two such halves
constexpr uint32_t WAIT_LIMIT = 1u << 22;
constexpr int STORE_WARPS = 4;               // warps 0 - 3 store C
constexpr int COPY_WARP = 4;                 // the first of up to four warps whose lanes 0 issue the TMA copies
constexpr int MMA_THREAD = 256;              // lane 0 of the last warp issues the MMAs
constexpr int THREADS = 288;
constexpr int MAX_STAGES = 16;
constexpr unsigned FULL = 0xffffffffu;

// A stage: GROUP blocks of a block row, their slabs of B and the blocks themselves.
template <int BS, int HALVES>
struct Shape {
  static constexpr int GROUP = BS == 32 && HALVES == 2 ? 1 : 64 / BS;  // blocks per stage
  static constexpr int COPY_WARPS = GROUP < 4 ? GROUP : 4;  // warps that issue its copies
  static constexpr int MMA_BLOCKS = BS == 8 ? 2 : 1;        // blocks per MMA: two of 8 x 8 side by side along k
  static constexpr int BOX_BYTES = BS * 64 * 2;             // 64 columns x BS rows of B
  static constexpr int SLAB_BYTES = 2 * HALVES * BOX_BYTES; // a block's rows of B
  static constexpr int VALUE_BYTES = BS * BS * 2;           // one block
  static constexpr int MMA_N = BS == 32 ? 32 : 16;          // at least 16 with M = 128: 8 rows are padded with zeros
  static constexpr int TMEM_COLS = 2 * HALVES * MMA_N;      // two sets of accumulators: 32, 64 or 128 columns
  static constexpr int VALUES_AT = GROUP * SLAB_BYTES;      // slabs first (1024-aligned), then the blocks, then (8 x 8) zeros
  static constexpr int ZEROS_AT = VALUES_AT + GROUP * VALUE_BYTES;
  static constexpr int STAGE_BYTES = ZEROS_AT + (BS == 8 ? GROUP * VALUE_BYTES : 0);  // a multiple of 1024
  // Block operand, K-major: rows of 32 or 64 bytes swizzled within themselves, or (8 x 8) unswizzled core matrices of
  // 8 rows x 16 bytes, each of which is one block: 128 bytes to the next along k, rows 8 - 15 among the zeros.
  static constexpr uint32_t LAYOUT = BS == 32 ? 4u : BS == 16 ? 6u : 0u;
  static constexpr uint32_t LBO = BS == 8 ? 128u : 16u;
  static constexpr uint32_t SBO = BS == 32 ? 512u : BS == 16 ? 256u : (uint32_t)(GROUP * VALUE_BYTES);
};

template <int BS, int HALVES>
constexpr int most_stages() {
  return 215 * 1024 / Shape<BS, HALVES>::STAGE_BYTES < MAX_STAGES ? 215 * 1024 / Shape<BS, HALVES>::STAGE_BYTES : MAX_STAGES;
}
// CTAs per SM, and the stages of each: the shared memory of an SM shared out among the CTAs that run on it.  More CTAs gain
// more than more stages each (1,024 x 1,024 16 x 16 blocks at 5 %, N = 512: one CTA of six stages 142 us, two of three 77,
// three of two 59; 32 x 32, 700 block rows of 24, N = 192, two stages each: four CTAs 30.7, five 26.3); their accumulators fit the
// 512 columns of TMEM, their registers the SM's.
template <int BS, int HALVES>
int ctas_per_sm(int64_t units, int sm_count, int *stages) {
  constexpr int MOST = HALVES == 1 ? 5 : BS == 32 ? 4 : 3;
  static_assert(MOST * Shape<BS, HALVES>::TMEM_COLS <= 512 && 222 * 1024 / MOST - 1024 >= 2 * Shape<BS, HALVES>::STAGE_BYTES, "");
  int64_t per_sm = (units + sm_count - 1) / sm_count;
  if (per_sm > MOST) per_sm = MOST;
  const int fit = (222 * 1024 / (int)per_sm - 1024) / Shape<BS, HALVES>::STAGE_BYTES;
  *stages = fit > most_stages<BS, HALVES>() ? most_stages<BS, HALVES>() : fit;
  return (int)per_sm;
}
template <int BS, int HALVES>
constexpr int smem_bytes(int stages) { return stages * Shape<BS, HALVES>::STAGE_BYTES + 1024; }  // + alignment slack

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor, version 1 (Blackwell): bits [0,14) address
// >> 4, [16,30) leading byte offset >> 4, [32,46) stride byte offset >> 4,
// [46,48) version, [61,64) layout type (0 = none, 2 = 128-byte swizzle, 4 = 64-byte, 6 = 32-byte).
__device__ __forceinline__ uint64_t make_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes,
                                              uint32_t layout) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32) | (1ull << 46) | ((uint64_t)layout << 61);
}

// Instruction descriptor for kind::f16: D f32 (bits 4-5 = 1), A and B bf16
// (bits 7-9 and 10-12 = 1), A MN-major (bit 15), B K-major (bit 16 = 0),
// N >> 3 at bits 17-22, M >> 4 at bits 24-28.
constexpr uint32_t instruction_descriptor(uint32_t n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

// Arrives on `bar` when the MMAs issued so far have completed.
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// PER_UNIT_STATUS: raise status[unit] instead of status[0] when a wait gives up.
template <bool PER_UNIT_STATUS, int BS, int HALVES>
__global__ void __launch_bounds__(THREADS, HALVES == 1 ? 5 : 3) bsr_spmm_tcgen05_kernel(
    const __grid_constant__ CUtensorMap map_slab, const __grid_constant__ CUtensorMap map_box,
    const __grid_constant__ CUtensorMap map_block, const __grid_constant__ CUtensorMap map_group, int64_t units, int64_t n_tiles,
    int64_t N, int cols, int value_rows, int stages, const int32_t *__restrict__ brp, const int32_t *__restrict__ bci,
    __nv_bfloat16 *__restrict__ C, int *status) {
  using S = Shape<BS, HALVES>;
  constexpr int TILE_N = HALVES * HALF_N;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[MAX_STAGES], bar_empty[MAX_STAGES];  // a stage has landed; has been read
  __shared__ __align__(8) uint64_t bar_sums[2], bar_stored[2];  // an accumulator pair is complete; has been read
  __shared__ uint32_t tmem_slot;
  __shared__ int failed;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t stage0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  after_previous_kernel();
  if (tid == 0) {
    failed = 0;
    for (int s = 0; s < stages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), S::COPY_WARPS);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&bar_sums[a]), 1);
      mbar_init(smem_u32(&bar_stored[a]), STORE_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_slab) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_block) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_group) : "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(S::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if constexpr (BS == 8) {  // rows 8 - 15 of the block operand, which no copy writes
    constexpr int WORDS = (S::STAGE_BYTES - S::ZEROS_AT) / 4;
    for (int i = tid; i < stages * WORDS; i += THREADS)
      asm volatile("st.shared.u32 [%0], %1;" ::"r"(stage0 + (uint32_t)(i / WORDS * S::STAGE_BYTES + S::ZEROS_AT + i % WORDS * 4)),
                   "r"(0u) : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;

  // All roles walk the CTA's units in the same order.  The offsets of a unit's block row are loaded a unit ahead.
  const int64_t first_unit = blockIdx.x, stride = gridDim.x;
  auto bounds = [&](int64_t unit) {
    if (unit >= units) return make_int2(0, 0);
    const int32_t *p = brp + unit / n_tiles;
    return make_int2(__ldg(p), __ldg(p + 1));
  };
  auto gave_up = [&](int64_t unit) {
    failed = 1;
    atomicExch(status + (PER_UNIT_STATUS ? unit : 0), 1);
  };
  if (warp >= COPY_WARP && warp < COPY_WARP + S::COPY_WARPS) {
    // Each of these warps copies its share of every group: blocks `mine`, mine + COPY_WARPS, ...  Lane l holds the block column
    // of the l-th of 32 blocks, and of the 32 behind them or of the next unit's first.
    const int mine = warp - COPY_WARP;
    auto column = [&](int2 b, int p) { return b.x + p + lane < b.y ? __ldg(bci + b.x + p + lane) : 0; };
    int2 b = bounds(first_unit), after = bounds(first_unit + stride);
    int s = 0, round = 0;
    int next_unit = column(b, 0);
    bool ok = true;
    for (int64_t unit = first_unit; ok && unit < units; unit += stride) {
      const int n0 = (int)(unit % n_tiles) * TILE_N;
      // The tile's boxes of 64 columns that reach into B.  One copy takes them all unless the last is a part of one: then, and
      // where there is one, each is a copy.  The others are not copied (or zeros): what lies in their place makes accumulator
      // lanes that are not stored.
      const int boxes = N - n0 >= TILE_N ? 2 * HALVES : (int)(N - n0 + 63) / 64;
      const bool one_copy = boxes > 1 && (N - n0 >= TILE_N || N % 64 == 0);
      const uint32_t block_bytes = (one_copy ? 2 * HALVES : boxes) * S::BOX_BYTES;
      int here = next_unit, ahead = column(b, 32);
      next_unit = column(after, 0);
      const int2 after2 = bounds(unit + 2 * stride);
      const int nblk = b.y - b.x;
      for (int p = 0; p < nblk; p += S::GROUP) {
        ok = round == 0 || mbar_wait(smem_u32(&bar_empty[s]), (uint32_t)(round - 1) & 1u);
        ok = __all_sync(FULL, ok);
        if (!ok) {  // the MMAs that read this stage last never released it
          if (lane == 0) gave_up(unit);
          break;
        }
        if (p != 0 && p % 32 == 0) { here = ahead; ahead = column(b, p + 32); }
        constexpr int SHARE = S::GROUP / S::COPY_WARPS;
        int block_column[SHARE];
#pragma unroll
        for (int i = 0; i < SHARE; ++i) block_column[i] = __shfl_sync(FULL, here, (p + mine + i * S::COPY_WARPS) & 31);
        if (lane == 0) {
          const uint32_t full = smem_u32(&bar_full[s]), base = stage0 + (uint32_t)s * S::STAGE_BYTES;
          const int left = nblk - p < S::GROUP ? nblk - p : S::GROUP;
          const bool group = left == S::GROUP;  // all values are one copy, this warp's if it is the first
          const int copies = (left + S::MMA_BLOCKS - 1) / S::MMA_BLOCKS * S::MMA_BLOCKS;  // past a row's blocks: zeros
          const int share = group ? SHARE : (copies - mine + S::COPY_WARPS - 1) / S::COPY_WARPS;
          const uint32_t bytes = share * block_bytes + (group ? (mine == 0 ? S::GROUP : 0) : share) * S::VALUE_BYTES;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full), "r"(bytes) : "memory");
          if (group && mine == 0) tma_load_2d(base + S::VALUES_AT, &map_group, 0, (b.x + p) * BS, full);
#pragma unroll
          for (int i = 0; i < SHARE; ++i) {
            if (i >= share) break;
            const int j = mine + i * S::COPY_WARPS;
            const int y_B = j < left ? block_column[i] * BS : cols;
            const uint32_t slab = base + (uint32_t)(j * S::SLAB_BYTES);
            if (one_copy) {
              tma_load_3d(slab, &map_slab, 0, y_B, n0 / 64, full);
            } else {
#pragma unroll
              for (int g = 0; g < 2 * HALVES; ++g)
                if (g < boxes) tma_load_2d(slab + (uint32_t)(g * S::BOX_BYTES), &map_box, n0 + 64 * g, y_B, full);
            }
            if (!group)
              tma_load_2d(base + (uint32_t)(S::VALUES_AT + j * S::VALUE_BYTES), &map_block, 0,
                          j < left ? (b.x + p + j) * BS : value_rows, full);
          }
        }
        __syncwarp();
        if (++s == stages) { s = 0; ++round; }
      }
      b = after;
      after = after2;
    }
    // the last arrivals on `empty` before the shared memory goes back
    for (int i = 0; ok && i < stages; ++i) {
      if (s == 0) { s = stages; --round; }
      --s;
      if (round < 0) break;
      ok = mbar_wait(smem_u32(&bar_empty[s]), (uint32_t)round & 1u);
    }
  } else if (tid == MMA_THREAD) {
    int2 b = bounds(first_unit);
    int s = 0, round = 0, made = 0;  // accumulator pairs begun
    bool ok = true;
    for (int64_t unit = first_unit; ok && unit < units; unit += stride) {
      const int2 after = bounds(unit + stride);
      const int nblk = b.y - b.x;
      if (nblk > 0) {
        const int halves = HALVES == 2 && (unit % n_tiles) * TILE_N + HALF_N < N ? 2 : 1;
        const uint32_t sums = tmem + (uint32_t)((made & 1) * HALVES * S::MMA_N);
        ok = made < 2 || mbar_wait(smem_u32(&bar_stored[made & 1]), (uint32_t)(made / 2 - 1) & 1u);
        for (int p = 0; ok && p < nblk; p += S::GROUP) {
          ok = mbar_wait(smem_u32(&bar_full[s]), (uint32_t)round & 1u);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t base = stage0 + (uint32_t)s * S::STAGE_BYTES;
#pragma unroll
          for (int j = 0; j < S::GROUP; j += S::MMA_BLOCKS) {
            if (p + j >= nblk) break;
#pragma unroll
            for (int h = 0; h < HALVES; ++h) {
              if (h >= halves) break;
#pragma unroll
              for (int k = 0; k < BS * S::MMA_BLOCKS / 16; ++k) {  // 16 rows of a box are 2048 bytes, 16 values of a block row 32
                const uint64_t adesc = make_desc(base + (uint32_t)(j * S::SLAB_BYTES + h * 2 * S::BOX_BYTES + k * 2048),
                                                 S::BOX_BYTES, BS == 8 ? S::SLAB_BYTES : 1024u, 2u);
                const uint64_t bdesc = make_desc(base + (uint32_t)(S::VALUES_AT + j * S::VALUE_BYTES + k * 32), S::LBO, S::SBO,
                                                 S::LAYOUT);
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(sums + (uint32_t)(h * S::MMA_N)),
                    "l"(adesc), "l"(bdesc), "r"(instruction_descriptor(S::MMA_N)), "r"((p > 0 || j > 0 || k > 0) ? 1u : 0u)
                    : "memory");
              }
            }
          }
          mma_commit(smem_u32(&bar_empty[s]));
          if (p + S::GROUP >= nblk) mma_commit(smem_u32(&bar_sums[made & 1]));
          if (++s == stages) { s = 0; ++round; }
        }
        if (!ok) gave_up(unit);
        ++made;
      }
      b = after;
    }
  } else if (warp < STORE_WARPS) {
    int2 b = bounds(first_unit);
    int made = 0;
    for (int64_t unit = first_unit; unit < units; unit += stride) {
      const int2 after = bounds(unit + stride);
      const int64_t br = unit / n_tiles;
      const int n0 = (int)(unit - br * n_tiles) * TILE_N;
      const bool empty = b.x == b.y;  // C = 0
      const int halves = HALVES == 2 && (int64_t)n0 + HALF_N < N ? 2 : 1;
      const uint32_t sums = tmem + (uint32_t)((made & 1) * HALVES * S::MMA_N) + ((uint32_t)(warp * 32) << 16);
      if (!empty) {
        const bool ok = mbar_wait(smem_u32(&bar_sums[made & 1]), (uint32_t)(made / 2) & 1u);
        if (!__all_sync(FULL, ok)) {
          if (lane == 0) gave_up(unit);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      // TMEM lane m of accumulator h = column n0 + 128 h + m of C; this warp reads lanes 32 warp .. +32 (16 rows of a 32 x 32 block
      // at a time, for registers that leave room for five CTAs).
      constexpr int AT_ONCE = BS == 32 ? 1 : HALVES, PARTS = BS == 32 ? 2 * HALVES : 1;
#pragma unroll(HALVES == 1 ? 1 : PARTS)
      for (int part = 0; part < PARTS; ++part) {
        const int h0 = BS == 32 ? part / 2 : 0, r0 = BS == 32 ? part % 2 * 16 : 0;
        uint32_t v[AT_ONCE][16];
#pragma unroll
        for (int h = 0; h < AT_ONCE; ++h) {
          uint32_t *w = v[h];
          if (empty || h0 + h >= halves) {
#pragma unroll
            for (int r = 0; r < 16; ++r) w[r] = 0;
          } else {
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
                "%15}, [%16];"
                : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]),
                  "=r"(w[8]), "=r"(w[9]), "=r"(w[10]), "=r"(w[11]), "=r"(w[12]), "=r"(w[13]), "=r"(w[14]), "=r"(w[15])
                : "r"(sums + (uint32_t)((h0 + h) * S::MMA_N + r0))
                : "memory");
          }
        }
        if (!empty) {
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (part == PARTS - 1) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if (lane == 0)
              asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&bar_stored[made & 1])) : "memory");
            ++made;
          }
        }
#pragma unroll
        for (int h = 0; h < AT_ONCE; ++h) {
          const int64_t col = (int64_t)n0 + (h0 + h) * HALF_N + warp * 32 + lane;
          if (col < N) {
            __nv_bfloat16 *out = C + (br * BS + r0) * N + col;
#pragma unroll
            for (int r = 0; r < (BS < 16 ? BS : 16); ++r) out[r * N] = __float2bfloat16_rn(__uint_as_float(v[h][r]));
          }
        }
      }
      b = after;
    }
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (failed) {
    // A wait gave up with copies or MMAs of this CTA possibly still in flight: give them a bounded time (1 ms)
    // to land before the shared memory and the TMEM columns go back to the SM.
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::TMEM_COLS) : "memory");
}

using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// 2-D bf16 tensor map: `inner` contiguous elements per row, `outer` rows.
bool make_map_2d(CUtensorMap *map, const void *base, uint64_t inner, uint64_t outer, uint32_t box_inner,
                 uint32_t box_outer, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {inner * 2};  // bytes between rows
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// B as groups of 64 columns: 64 elements, `rows` rows, n / 64 groups; a box of `box_rows` rows of `groups` groups.
bool make_map_3d(CUtensorMap *map, const void *base, uint64_t n, uint64_t rows, uint32_t box_rows, uint32_t groups) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {64, rows, n / 64};
  cuuint64_t strides[2] = {n * 2, 128};  // bytes between rows, between groups
  cuuint32_t box[3] = {64, box_rows, groups};
  cuuint32_t elem[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(base), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

namespace {
bool aligned_for_tma(const BsrSpmmArgs &a) {  // 16-byte aligned bases and row pitches
  return a.n_rhs % 8 == 0 && (reinterpret_cast<uintptr_t>(a.B) & 15u) == 0 &&
         (reinterpret_cast<uintptr_t>(a.block_values) & 15u) == 0;
}
}  // namespace

// Whether an output is one chain of MMAs, whose sums are cut off and not rounded, in this kernel and in the mma.sync one: by what
// does not change with the number of block rows or blocks, so that a part of a matrix has the bits of the whole.  The kernels on
// CUDA cores that used to take the other calls rounded every sum to nearest, and so does the mma.sync kernel there (f32 sums of
// products that cancel, root mean square over that of the sum, 400 blocks of 16 x 16 a block row: 6.7e-7 on CUDA cores,
// 3.4e-7 with sums of 16 added, 6.1e-6 as a chain; the rounding to bf16 is 1.1e-3).
bool bsr_chain_sums(const BsrSpmmArgs &a) { return a.n_rhs >= (a.block_size == 8 ? 96 : 64) && aligned_for_tma(a); }

bool bsr_tcgen05_supported(const BsrSpmmArgs &a) {
  // ... and 32-bit box coordinates: block rows of the value matrix (nnzb * block size) and B's extents.
  if (a.block_size != 8 && a.block_size != 16 && a.block_size != 32) return false;
  if (a.nnzb > 2147483647LL / a.block_size || a.cols > 2147483647LL - 64 || a.n_rhs > 2147483647LL - 256) return false;
  return a.nnzb > 0 && a.cols > 0 && aligned_for_tma(a);
}

// Against the mma.sync kernel, which reads its operands from global memory and takes any size: this one where a tile of columns
// is well filled, there is a unit for every SM and block rows are long enough to fill the pipeline.  Both give the same bits, so
// that the line only decides the time.  Measured on 80 to 5,000 block rows of 5 to 40 (us with mma.sync, here):
//   32 x 32: 300 block rows of 24, N = 64 19.5, 14.2; 1,200 of 12, N = 136 33.6, 33.5, N = 256 57.0, 28.3; from 104 columns on
//   less than a unit per SM too (80 of 24, N = 128 17.2, 11.8; of 6, N = 104 5.9, 6.5).
//   16 x 16: whole groups of 64 columns from 128 on whatever the rows' length (300 of 6, N = 128 6.9, 5.9; 1,200 of 30, N = 256
//   53.9, 26.9; but 80 of 6, N = 128 3.2, 4.4; 600 of 6, N = 192 8.5, 9.3); others from 8 blocks a row on (1,200 of 12, N = 160
//   19.1, 16.7; of 5 10.9, 11.7), from 6 where the tiles are four fifths full (3,605 of 7, N = 416 83.4, 50.0; 540 of 7 14.8, 11.8;
//   1,592 of 6, N = 224 17.4, 15.3; but of 5, N = 432 1.15 times), with rows of B that are no multiple of 32 bytes from 12 (150 of
//   40, N = 136 16.0, 11.1; 600 of 24 16.7, 18.5; 1,200 of 30 32.0, 31.7); 64 columns from 12 a row and two units per SM on (300 of
//   24 10.5, 8.7; 150 of 12 4.5, 6.0).
//   8 x 8, half of whose MMA is padding: whole groups of 64 columns from 128 on and rows of 20 blocks (300 of 24, N = 256 11.1, 8.8,
//   N = 192 8.2, 9.2; 1,200 of 30, N = 128 20.7, 12.6; but 2,500 of 20, N = 264 33.2, 43.3), or many units: of whole tiles (5,000 of
//   8, N = 512 78.1, 48.3; 1,200 of 12, N = 256 14.1, 11.9; 600 of 6 6.4, 8.3); of tiles four fifths full, from 12 a row with whole
//   groups (2,904 of 15, N = 448 52.5, 39.4; but of 9, N = 384 1.08 times), from 27 with other multiples of 32 bytes (3,350 of 48,
//   N = 240 91.5, 73.6; 2,002 of 54, N = 416 105, 90; 311 of 28, N = 496 16.7, 14.2; but of 18, N = 304 1.12 times).
//   16 x 16 and 8 x 8 on tiles three quarters full, where B is large (with C it then outgrows the half of L2 on an SM's die, whose
//   longer way the copies would hide and the loads not; the counters were not read): from 34 MB (16 x 16, blocks of 4 and 16 a row: N = 408 30 MB 1.07 and 0.82 times the time, 43 MB 0.78 and 0.75;
//   N = 344 34 MB 1.03 and 0.86; N = 504 53 MB 56.9 -> 42.2 us and 150 -> 106) and 44 MB, from nine blocks a row 36 MB (8 x 8:
//   N = 408 30 MB 1.40 and 1.10, 45 MB 1.02 and 0.89; N = 504 38 MB 1.05 and 0.86, 56 MB 0.88 and 0.79).
bool bsr_tcgen05_pays(const BsrSpmmArgs &a, int sm_count) {
  const int64_t n = a.n_rhs, brows = a.rows / a.block_size, units = brows * ceil_div(n, HALF_N);
  if (!bsr_chain_sums(a) || !bsr_tcgen05_supported(a) || brows == 0) return false;
  if (reinterpret_cast<uintptr_t>(a.C) % 16 != 0) return true;  // the mma.sync kernel has chains for aligned C only
  if (a.block_size == 32) return n >= 104 || units >= sm_count;
  if (units < sm_count) return false;
  const int64_t mean = a.nnzb / brows;
  const int64_t large = a.block_size == 16 ? 34000000 : mean >= 9 ? 36000000 : 44000000;
  if (a.cols * n * 2 >= large && 4 * n * brows >= 3 * HALF_N * units) return true;
  const bool groups = n >= HALF_N && n % 64 == 0;
  const bool full = 5 * n * brows >= 4 * HALF_N * units && n % 16 == 0;
  if (a.block_size == 8)
    return (groups && mean >= 20) ||
           (units >= 8 * (int64_t)sm_count && full && mean >= (n % (2 * HALF_N) == 0 ? 8 : groups ? 12 : 27));
  if (groups || (full && n > HALF_N && mean >= 6)) return true;
  if (n < 72) return mean >= 12 && units >= 2 * (int64_t)sm_count;
  return mean >= (n > HALF_N && n % 16 != 0 ? 12 : 8);
}

namespace {

// Opts a kernel into its largest shared memory, once per device; racing threads repeat an idempotent call.
template <bool PER_UNIT_STATUS, int BS, int HALVES>
cudaError_t configure() {
  static std::atomic<bool> configured[64];
  int device = 0;
  cudaGetDevice(&device);
  if (device >= 0 && device < 64 && configured[device].load(std::memory_order_acquire)) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(bsr_spmm_tcgen05_kernel<PER_UNIT_STATUS, BS, HALVES>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       smem_bytes<BS, HALVES>(most_stages<BS, HALVES>()));
  if (e == cudaSuccess && device >= 0 && device < 64) configured[device].store(true, std::memory_order_release);
  return e;
}

template <bool PER_UNIT_STATUS, int BS, int HALVES>
cudaError_t launch_halves(const BsrSpmmArgs &a, int *status, int sm_count, cudaStream_t s) {
  const int64_t n_tiles = ceil_div(a.n_rhs, HALVES * HALF_N), units = a.rows / BS * n_tiles;
  if (units == 0) return cudaSuccess;
  cudaError_t e = configure<PER_UNIT_STATUS, BS, HALVES>();
  if (e != cudaSuccess) return e;
  CUtensorMap map_slab, map_box, map_block, map_group;
  // B: cols x N bf16 (N at least 64), boxes of 64 columns x BS rows, 128-byte swizzle, one or (in whole groups of 64 columns) a tile's; block
  // values: (nnzb * BS) x BS, boxes of one block and of a group.
  const auto swizzle = BS == 8 ? CU_TENSOR_MAP_SWIZZLE_NONE : BS == 16 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_64B;
  if (!make_map_2d(&map_box, a.B, (uint64_t)a.n_rhs, (uint64_t)a.cols, 64, BS, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !make_map_2d(&map_block, a.block_values, BS, (uint64_t)a.nnzb * BS, BS, BS, swizzle) ||
      !make_map_2d(&map_group, a.block_values, BS, (uint64_t)a.nnzb * BS, BS, Shape<BS, HALVES>::GROUP * BS, swizzle))
    return cudaErrorInvalidValue;
  if (!make_map_3d(&map_slab, a.B, (uint64_t)a.n_rhs, (uint64_t)a.cols, BS, 2 * HALVES))
    return cudaErrorInvalidValue;
  int stages;
  const int per_sm = ctas_per_sm<BS, HALVES>(units, sm_count, &stages);
  const int64_t grid = units < (int64_t)per_sm * sm_count ? units : (int64_t)per_sm * sm_count;
  launch_chained(bsr_spmm_tcgen05_kernel<PER_UNIT_STATUS, BS, HALVES>, (unsigned)grid, THREADS,
                 (size_t)smem_bytes<BS, HALVES>(stages), s, map_slab, map_box, map_block, map_group, units, n_tiles, a.n_rhs,
                 (int)a.cols, (int)(a.nnzb * BS), stages, a.block_row_ptr, a.block_col_idx,
                 static_cast<__nv_bfloat16 *>(a.C), status);
  return cudaGetLastError();
}

template <bool PER_UNIT_STATUS, int BS>
cudaError_t launch_tcgen05(const BsrSpmmArgs &a, int *status, int sm_count, cudaStream_t s) {
  // Tiles of 256 columns fetch a block once for two accumulators; tiles of 128 where the second would be empty or nearly so,
  // and where 256 leave too few units (403 block rows of 9, N = 480: 13.2 us with 256, 12.4 with 128; 1,024 of 51, N = 512:
  // 59 and 64).  32 x 32 has one block per stage with 256, which only many whole tiles of short block rows make up for (us with
  // 128 and 256: 1,500 block rows of 4, N = 512 32.3, 28.2; 2,000 of 4, N = 192 23.1, 20.9; but 700 of 20, N = 512 40.0, 41.8;
  // 2,000 of 20, N = 256 56.9, 59.6), or very many of any (3,000 of 20, N = 448 161, 146; but 1,200 of 20 60.9, 63.5).  The status
  // words of the static entry point are per 256 columns.
  const int64_t n = a.n_rhs, pairs = a.rows / BS * ceil_div(n, 2 * HALF_N), tail = n % (2 * HALF_N);
  const int64_t many = a.nnzb < 8 * (a.rows / BS) ? 10 : 20;
  const bool narrow = BS == 32 ? n % 64 != 0 || (tail > 0 && tail < 192) || pairs < many * sm_count
                               : n <= HALF_N || (tail > 0 && tail <= 64) || pairs < 6 * (int64_t)sm_count;
  if constexpr (!PER_UNIT_STATUS)
    if (narrow) return launch_halves<PER_UNIT_STATUS, BS, 1>(a, status, sm_count, s);
  return launch_halves<PER_UNIT_STATUS, BS, 2>(a, status, sm_count, s);
}

}  // namespace

cudaError_t launch_bsr_spmm_tcgen05(const BsrSpmmArgs &a, int *status_flag, const DeviceInfo &dev, cudaStream_t s,
                                    int64_t *launches) {
  if (a.rows == 0) return cudaSuccess;
  ++*launches;
  switch (a.block_size) {
    case 8: return launch_tcgen05<false, 8>(a, status_flag, dev.sm_count, s);
    case 16: return launch_tcgen05<false, 16>(a, status_flag, dev.sm_count, s);
    case 32: return launch_tcgen05<false, 32>(a, status_flag, dev.sm_count, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace swb

// ---------------------------------------------------------------------------
// swb_bsr16_spmm_bf16_static: the tensor-core BSR SpMM for callers that must
// not allocate device memory.
//
// The regular entry point needs a context, and creating a context calls
// cudaMalloc for the status word its kernels raise when a bounded barrier wait
// gives up.  Some callers cannot do that: code running under a memory budget
// that was fixed at start-up (every byte handed out by the application's own
// pool), plug-ins that are loaded into a process which forbids driver
// allocations after initialisation, and code that runs while the allocator's
// lock may be held.  For them the status words live in the fixed array below,
// which is part of the library image: every GPU that loads the library holds
// its 128 KiB until the process exits, whether or not this entry point is used.
//
// One status word per unit (block row x tile of 256 columns), hence the limit
// of SWB_STATIC_MAX_CTAS units per call.  All calls share the array and a call
// begins by clearing the words it will use, so the array holds the outcome of
// the most recent call only, and two calls that overlap on the GPU (different
// streams) race on it.
// ---------------------------------------------------------------------------
namespace swb {
namespace {

constexpr int SWB_STATIC_MAX_CTAS = 32768;  // 32768 status words = 128 KiB

static __device__ __align__(256) int swb_static_status_words[SWB_STATIC_MAX_CTAS];

// In host code `swb_static_status_words` is only a handle for the symbol, not a
// device address; the address a kernel can use comes from
// cudaGetSymbolAddress, asked once per device with that device current.
// Host-side record per device: the array's device address and the number of words the most recent call
// on that device used.  Atomics, so that host threads may call concurrently (two threads that both find
// the address missing ask for it twice and store the same value).
struct StaticStatusSlot {
  std::atomic<int *> address{nullptr};
  std::atomic<int64_t> last_grid{0};
};
StaticStatusSlot g_static_slots[64];

int *static_status_address(cudaError_t *err, StaticStatusSlot **slot_out = nullptr) {
  int device = 0;
  *err = cudaGetDevice(&device);
  if (*err != cudaSuccess) return nullptr;
  if (device < 0 || device >= 64) {
    *err = cudaErrorInvalidDevice;
    return nullptr;
  }
  StaticStatusSlot &slot = g_static_slots[device];
  if (slot_out) *slot_out = &slot;
  int *address = slot.address.load(std::memory_order_acquire);
  if (!address) {
    void *p = nullptr;
    *err = cudaGetSymbolAddress(&p, swb_static_status_words);
    if (*err != cudaSuccess) return nullptr;
    address = static_cast<int *>(p);
    slot.address.store(address, std::memory_order_release);
  }
  return address;
}

// Counts the non-zero words among the first `grid` through pageable stack memory: no pinned or device
// allocation.  The stream must be idle.
cudaError_t count_status_words(const int *status, int64_t grid, int32_t *count_out) {
  int32_t count = 0;
  int piece[1024];
  for (int64_t off = 0; off < grid; off += 1024) {
    const int64_t n = grid - off < 1024 ? grid - off : 1024;
    cudaError_t e = cudaMemcpy(piece, status + off, (size_t)n * sizeof(int), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return e;
    for (int64_t i = 0; i < n; ++i) count += piece[i] != 0;
  }
  *count_out = count;
  return cudaSuccess;
}

int static_fail(int status, const char *fmt, long long a = 0, long long b = 0) {
  char buf[512];
  snprintf(buf, sizeof buf, fmt, a, b);
  set_thread_error(buf);
  return status;
}

}  // namespace
}  // namespace swb

extern "C" __attribute__((visibility("default"))) int swb_bsr16_spmm_bf16_static(
    int64_t rows, int64_t cols, int64_t nnzb, int64_t n_rhs, const int32_t *block_row_ptr,
    const int32_t *block_col_idx, const uint16_t *block_values, const uint16_t *B, uint16_t *C, void *stream,
    int32_t *gave_up_ctas) {
  using namespace swb;
  // Status codes are those of swb_status in sparsewave_b200.h.
  constexpr int kInvalidShape = -2, kInvalidArgument = -3, kCuda = -4, kUnsupported = -5, kCapacity = -7;
  if (rows < 0 || cols < 0 || nnzb < 0)
    return static_fail(kInvalidArgument, "bsr_spmm: rows, cols and nnzb must be non-negative");
  if (rows % 16 != 0)
    return static_fail(kInvalidShape, "output rows must be divisible by block size, but got %lld and 16", rows);
  if (cols % 16 != 0)
    return static_fail(kInvalidShape, "right-hand-side rows must be divisible by block size, but got %lld and 16", cols);
  if (n_rhs < 1) return static_fail(kInvalidShape, "bsr_spmm: right-hand side must have at least one column, but got %lld", n_rhs);
  if (rows > 2147483647LL || cols > 2147483647LL || nnzb > 2147483647LL / 16)
    return static_fail(kInvalidShape, "BSR dimensions and NNZ blocks must fit in i32");
  if (!block_row_ptr || (nnzb > 0 && (!block_col_idx || !block_values)) || (cols > 0 && !B) || (rows > 0 && !C))
    return static_fail(kInvalidArgument, "bsr_spmm: NULL operand pointer");
  BsrSpmmArgs a{rows, cols, nnzb, 16, n_rhs, block_row_ptr, block_col_idx, block_values, B, C};
  if (!bsr_tcgen05_supported(a))
    return static_fail(kUnsupported,
                       "the static-scratch BSR entry point needs at least one block, a column count that is a "
                       "multiple of 8 and 16-byte aligned block values and right-hand side");
  const int64_t n_tiles = ceil_div(n_rhs, 2 * HALF_N);
  const int64_t grid = (rows / 16) * n_tiles;
  if (grid > SWB_STATIC_MAX_CTAS)
    return static_fail(kCapacity,
                       "the static-scratch BSR entry point handles at most %lld (block row, 256-column tile) pairs "
                       "per call, but this call needs %lld",
                       (long long)SWB_STATIC_MAX_CTAS, (long long)grid);
  if (grid == 0) return 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaSuccess;
  StaticStatusSlot *slot = nullptr;
  int *status = static_status_address(&e, &slot);
  if (!status) return static_fail(kCuda, cudaGetErrorString(e));
  // The words keep the previous call's outcome: clear the ones this call uses.
  e = cudaMemsetAsync(status, 0, (size_t)grid * sizeof(int), s);
  if (e != cudaSuccess) return static_fail(kCuda, cudaGetErrorString(e));
  // The kernel that the regular entry point would choose, but for the SM count, which costs a call here; both kernels give the
  // same bits, and the one without tcgen05 never gives up.
  int64_t launches = 0;
  e = bsr_tcgen05_pays(a, DeviceInfo().sm_count) ? launch_tcgen05<true, 16>(a, status, DeviceInfo().sm_count, s)
                                                     : launch_bsr_spmm_mma(a, DeviceInfo(), s, &launches);
  if (e == cudaErrorInvalidValue) return static_fail(kCuda, "could not encode the TMA tensor maps");
  if (e != cudaSuccess) return static_fail(kCuda, cudaGetErrorString(e));
  slot->last_grid.store(grid, std::memory_order_release);
  if (gave_up_ctas) {
    e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = count_status_words(status, grid, gave_up_ctas);
    if (e != cudaSuccess) return static_fail(kCuda, cudaGetErrorString(e));
  }
  return 0;
}

// Outcome of the most recent swb_bsr16_spmm_bf16_static call on the current device, for callers that
// passed gave_up_ctas == NULL: waits for `stream` and counts the CTAs of that call whose bounded wait
// gave up.  Allocates nothing.
extern "C" __attribute__((visibility("default"))) int swb_bsr16_static_status(void *stream, int32_t *gave_up_ctas) {
  using namespace swb;
  constexpr int kInvalidArgument = -3, kCuda = -4;
  if (!gave_up_ctas) return static_fail(kInvalidArgument, "bsr16 static status: gave_up_ctas is NULL");
  *gave_up_ctas = 0;
  cudaError_t e = cudaSuccess;
  StaticStatusSlot *slot = nullptr;
  int *status = static_status_address(&e, &slot);
  if (!status) return static_fail(kCuda, cudaGetErrorString(e));
  e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
  if (e == cudaSuccess) e = count_status_words(status, slot->last_grid.load(std::memory_order_acquire), gave_up_ctas);
  if (e != cudaSuccess) return static_fail(kCuda, cudaGetErrorString(e));
  return 0;
}
