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
// A CTA owns one block row and a tile of 256 right-hand-side columns, i.e. two
// such accumulators side by side in TMEM (columns 0-15 and 16-31), so that each
// block and each block-column index is fetched once per 256 columns.
//   - MMA operand A = a 16 x 128 slab B[bci*16 .. +16, n .. n+128).  Row k is
//     contiguous along m: MN-major.  Two TMA boxes of 64 columns x 16 rows with
//     the 128-byte swizzle land it as the canonical MN-major SWIZZLE_128B layout
//     (128-byte rows, 1024 bytes between groups of 8 k rows = stride byte
//     offset, 2048 bytes between the two 64-column halves = leading byte
//     offset).  Columns past N are zero-filled by the TMA unit; a tile whose
//     second 128 columns lie wholly past N skips them.
//   - MMA operand B = the block itself, [r][lc] row-major: K-major.  One TMA box
//     of 16 x 16 with the 32-byte swizzle over the block values viewed as a
//     (nnzb*16) x 16 matrix lands it as the canonical K-major SWIZZLE_32B layout
//     (32-byte rows, 256 bytes between groups of 8 rows = stride byte offset).
//     Both accumulators' MMAs read the same copy.
// The slab rows are gathered by block-column index, four boxes per block.
//
// Pipeline.  Lane 0 of warp 4 is the producer: per chunk of blocks it waits for
// the stage's `empty` mbarrier, loads the chunk's block-column indices, arms the
// stage's `full` mbarrier with the byte count and issues the TMA copies.  Lane 0
// of warp 5 issues the MMAs: it waits for `full`, issues the chunk's MMAs and
// lets tcgen05.commit arrive on `empty` when they have read their operands, so
// index loads and copies of later chunks never wait behind a commit.  After the
// last chunk the commit arrives on `done`; warps 0-3 then read both accumulators
// with tcgen05.ld (each warp its own 32 TMEM lanes), round to bf16 and store C.
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

constexpr int TILE_N = 256;                  // right-hand-side columns per CTA (two MMA M = 128 halves)
constexpr int HALF_N = 128;
constexpr uint32_t WAIT_LIMIT = 1u << 22;
constexpr int PRODUCER_THREAD = 128;         // lane 0 of warp 4 issues the TMA copies
constexpr int MMA_THREAD = 160;              // lane 0 of warp 5 issues the MMAs
constexpr int THREADS = 192;
constexpr int MAX_STAGES = 8;

// A pipeline step: one block of 16 x 16 or 32 x 32, or two blocks of 8 x 8 side by side along k.
template <int BS>
struct Shape {
  static constexpr int BLOCKS = BS == 8 ? 2 : 1;            // blocks per step
  static constexpr int K = BS * BLOCKS;                     // rows of B per step: 16 or 32
  static constexpr int BOX_BYTES = BS * 64 * 2;             // 64 columns x BS rows of B
  static constexpr int GROUP_BYTES = K * 64 * 2;            // 64 columns x K rows
  static constexpr int HALF_BYTES = 2 * GROUP_BYTES;        // one accumulator's operand
  static constexpr int SLAB_BYTES = 2 * HALF_BYTES;
  static constexpr int VALUE_BYTES = BS * BS * 2;           // one block
  static constexpr int MMA_N = BS == 32 ? 32 : 16;          // at least 16 with M = 128: 8 rows are padded with zeros
  static constexpr int TMEM_COLS = 2 * MMA_N;               // two accumulators
  // slabs first (1024-aligned), then the blocks, padded so that the next stage's slabs are 1024-aligned again
  static constexpr int STAGE_BYTES = (SLAB_BYTES + (BS == 8 ? 512 : VALUE_BYTES) + 1023) / 1024 * 1024;
  // Block operand, K-major: rows of 32 or 64 bytes swizzled within themselves, or (8 x 8) unswizzled core matrices of
  // 8 rows x 16 bytes, each of which is one block: 128 bytes to the next along k, 256 bytes to the (zero) rows 8 - 15.
  static constexpr uint32_t LAYOUT = BS == 32 ? 4u : BS == 16 ? 6u : 0u;
  static constexpr uint32_t LBO = BS == 8 ? 128u : 16u;
  static constexpr uint32_t SBO = BS == 32 ? 512u : 256u;
};

// Stages of a launch.  What fills the path from L2 is the number of copies in flight per SM: with CTAs enough, three
// stages (28 KiB for 16 x 16 blocks, seven CTAs per SM: 1024 x 1024 blocks at 5 %, 512 columns 69.7 us; two stages 78.7,
// four 84.0); with fewer, the shared memory that is left over goes into more stages.
template <int BS>
int stages_for(int64_t grid, int sm_count) {
  int64_t per_sm = (grid + sm_count - 1) / sm_count;
  if (per_sm > 7) per_sm = 7;
  const int64_t fit = 210 * 1024 / (per_sm > 0 ? per_sm : 1) / Shape<BS>::STAGE_BYTES;
  const int least = BS == 32 ? 2 : 3;
  return fit < least ? least : fit > MAX_STAGES ? MAX_STAGES : (int)fit;
}
template <int BS>
constexpr int smem_bytes(int stages) { return stages * Shape<BS>::STAGE_BYTES + 1024; }  // + alignment slack

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

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// PER_CTA_STATUS: raise status[blockIdx.x] instead of status[0] when a wait gives up.  STAGES: the number of stages where
// it is a constant, or 0: `run_stages` of them.
template <bool PER_CTA_STATUS, int BS, int STAGES>
__global__ void __launch_bounds__(THREADS) bsr_spmm_tcgen05_kernel(
    const __grid_constant__ CUtensorMap map_B, const __grid_constant__ CUtensorMap map_A, int64_t n_tiles,
    int64_t N, int cols, int value_rows, int run_stages, const int32_t *__restrict__ brp, const int32_t *__restrict__ bci,
    __nv_bfloat16 *__restrict__ C, int *status) {
  using S = Shape<BS>;
  const int stages = STAGES ? STAGES : run_stages;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[STAGES ? STAGES : MAX_STAGES];
  __shared__ __align__(8) uint64_t bar_empty[STAGES ? STAGES : MAX_STAGES];
  __shared__ __align__(8) uint64_t bar_done;
  __shared__ uint32_t tmem_slot;
  __shared__ int failed;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t br = blockIdx.x / n_tiles;
  const int n0 = (int)((blockIdx.x % n_tiles) * TILE_N);
  const int halves = ((int64_t)n0 + HALF_N < N) ? 2 : 1;  // the second 128 columns may lie wholly past N
  const uint32_t stage0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  after_previous_kernel();
  const int start = brp[br], end = brp[br + 1];
  const int nblk = end - start;

  if (nblk == 0) {  // empty block row: C = 0
    for (int64_t col = (int64_t)n0 + tid; col < N && col < (int64_t)n0 + TILE_N; col += THREADS)
      for (int r = 0; r < BS; ++r) C[(br * BS + r) * N + col] = __float2bfloat16_rn(0.0f);
    return;
  }

  if (tid == 0) {
    failed = 0;
    for (int s = 0; s < stages; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar_full[s])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar_empty[s])) : "memory");
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar_done)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_B) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_A) : "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(S::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if constexpr (BS == 8) {  // rows 8 - 15 of the block operand, which no copy writes
    for (int i = tid; i < stages * 64; i += THREADS)
      asm volatile("st.shared.u32 [%0], %1;" ::"r"(stage0 + (uint32_t)(i / 64) * S::STAGE_BYTES + S::SLAB_BYTES + 256u +
                                                   (uint32_t)(i % 64) * 4u), "r"(0u) : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  const int steps = (nblk + S::BLOCKS - 1) / S::BLOCKS;

  if (tid == PRODUCER_THREAD) {
    for (int i = 0, s = 0, round = 0; i < steps; ++i) {
      if (round > 0 && !mbar_wait(smem_u32(&bar_empty[s]), (uint32_t)(round - 1) & 1u)) {
        failed = 1;  // the MMAs of step i - stages never released this stage
        atomicExch(status + (PER_CTA_STATUS ? blockIdx.x : 0), 1);
        break;
      }
      const int first = start + i * S::BLOCKS;
      int y_B[S::BLOCKS], y_A[S::BLOCKS];  // first rows in B and among the block values; past a row's blocks: zeros
#pragma unroll
      for (int j = 0; j < S::BLOCKS; ++j) {
        const bool in = first + j < end;
        y_B[j] = in ? __ldg(bci + first + j) * BS : cols;
        y_A[j] = in ? (first + j) * BS : value_rows;
      }
      const uint32_t full = smem_u32(&bar_full[s]);
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full),
                   "r"((uint32_t)(halves * S::HALF_BYTES + S::BLOCKS * S::VALUE_BYTES))
                   : "memory");
      const uint32_t base = stage0 + (uint32_t)s * S::STAGE_BYTES;
#pragma unroll
      for (int j = 0; j < S::BLOCKS; ++j) {
#pragma unroll
        for (int g = 0; g < 4; ++g)
          if (g < 2 || halves == 2)
            tma_load_2d(base + (uint32_t)(g * S::GROUP_BYTES + j * S::BOX_BYTES), &map_B, n0 + 64 * g, y_B[j], full);
        tma_load_2d(base + (uint32_t)(S::SLAB_BYTES + j * S::VALUE_BYTES), &map_A, 0, y_A[j], full);
      }
      if (++s == stages) { s = 0; ++round; }
    }
  } else if (tid == MMA_THREAD) {
    bool ok = true;
    for (int c = 0, s = 0, round = 0; c < steps; ++c) {
      ok = mbar_wait(smem_u32(&bar_full[s]), (uint32_t)round & 1u);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t base = stage0 + (uint32_t)s * S::STAGE_BYTES;
      for (int h = 0; h < halves; ++h) {
#pragma unroll
        for (int k = 0; k < S::K / 16; ++k) {  // 16 rows of a slab are 2048 bytes, 16 values of a block row 32
          const uint64_t adesc = make_desc(base + (uint32_t)(h * S::HALF_BYTES + k * 2048), S::GROUP_BYTES, 1024u, 2u);
          const uint64_t bdesc = make_desc(base + (uint32_t)(S::SLAB_BYTES + k * 32), S::LBO, S::SBO, S::LAYOUT);
          asm volatile(
              "{\n\t.reg .pred p;\n\t"
              "setp.ne.b32 p, %4, 0;\n\t"
              "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem + (uint32_t)(h * S::MMA_N)),
              "l"(adesc), "l"(bdesc), "r"(instruction_descriptor(S::MMA_N)), "r"((c > 0 || k > 0) ? 1u : 0u)
              : "memory");
        }
      }
      const uint32_t arrive_on = (c == steps - 1) ? smem_u32(&bar_done) : smem_u32(&bar_empty[s]);
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(arrive_on)
                   : "memory");
      if (++s == stages) { s = 0; ++round; }
    }
    if (!ok) {
      failed = 1;
      atomicExch(status + (PER_CTA_STATUS ? blockIdx.x : 0), 1);
      // Release the waiters below.
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&bar_done)) : "memory");
    }
  }
  // The four epilogue warps wait for the last MMA (or for the failure release).
  bool done_ok = warp < 4 ? mbar_wait(smem_u32(&bar_done), 0u) : true;
  done_ok = __syncthreads_and(done_ok);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (!done_ok && tid == 0) atomicExch(status + (PER_CTA_STATUS ? blockIdx.x : 0), 1);
  if (!done_ok || failed) {
    // A wait gave up with copies or MMAs of this CTA possibly still in flight: give them a bounded time (1 ms)
    // to land before the shared memory and the TMEM columns go back to the SM.
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }

  if (done_ok && !failed && warp < 4) {
    // TMEM lane m of accumulator h = column n0 + 128 h + m of C; this warp reads lanes 32 warp .. +32
    for (int h = 0; h < halves; ++h) {
      const int64_t col = (int64_t)n0 + h * HALF_N + warp * 32 + lane;
#pragma unroll
      for (int r0 = 0; r0 < BS; r0 += 16) {
        uint32_t v[16];
        const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(h * S::MMA_N + r0);
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
            "%15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
              "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(taddr)
            : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (col < N) {
#pragma unroll
          for (int r = 0; r < (BS < 16 ? BS : 16); ++r)
            C[(br * BS + r0 + r) * N + col] = __float2bfloat16_rn(__uint_as_float(v[r]));
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
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

}  // namespace

bool bsr_tcgen05_supported(const BsrSpmmArgs &a) {
  // TMA needs 16-byte aligned bases and row pitches.
  // ... and 32-bit box coordinates: block rows of the value matrix (nnzb * block size) and B's extents.
  if (a.block_size != 8 && a.block_size != 16 && a.block_size != 32) return false;
  if (a.nnzb > 2147483647LL / a.block_size || a.cols > 2147483647LL - 64 || a.n_rhs > 2147483647LL - 256) return false;
  return a.n_rhs % 8 == 0 && a.nnzb > 0 && a.cols > 0 &&
         (reinterpret_cast<uintptr_t>(a.B) & 15u) == 0 && (reinterpret_cast<uintptr_t>(a.block_values) & 15u) == 0;
}

// 16 x 16 and 32 x 32 blocks always gain; 8 x 8 half fill the MMA and a block row is little work for a CTA: they gain from
// some 96 columns (2,048 block rows of 32, N = 128: 74 -> 32 us), not below (8,000 block rows of 8, N = 64: 45 us on the
// CUDA cores, 67 here).
bool bsr_tcgen05_pays(const BsrSpmmArgs &a) { return a.block_size != 8 || a.n_rhs >= 96; }

namespace {

// Opts a kernel into its largest shared memory, once per device; racing threads repeat an idempotent call.
template <bool PER_CTA_STATUS, int BS, int STAGES>
cudaError_t configure() {
  static std::atomic<bool> configured[64];
  int device = 0;
  cudaGetDevice(&device);
  if (device >= 0 && device < 64 && configured[device].load(std::memory_order_acquire)) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(bsr_spmm_tcgen05_kernel<PER_CTA_STATUS, BS, STAGES>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       smem_bytes<BS>(STAGES ? STAGES : MAX_STAGES));
  if (e == cudaSuccess && device >= 0 && device < 64) configured[device].store(true, std::memory_order_release);
  return e;
}

template <bool PER_CTA_STATUS, int BS, int STAGES>
cudaError_t launch_stages(const BsrSpmmArgs &a, int *status, int stages, int64_t grid, int64_t n_tiles, cudaStream_t s) {
  cudaError_t e = configure<PER_CTA_STATUS, BS, STAGES>();
  if (e != cudaSuccess) return e;
  CUtensorMap map_B, map_A;
  // B: cols x N bf16, boxes of 64 columns x BS rows, 128-byte swizzle; block values: (nnzb * BS) x BS, one box per block.
  if (!make_map_2d(&map_B, a.B, (uint64_t)a.n_rhs, (uint64_t)a.cols, 64, BS, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !make_map_2d(&map_A, a.block_values, BS, (uint64_t)a.nnzb * BS, BS, BS,
                   BS == 8 ? CU_TENSOR_MAP_SWIZZLE_NONE : BS == 16 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_64B))
    return cudaErrorInvalidValue;
  launch_chained(bsr_spmm_tcgen05_kernel<PER_CTA_STATUS, BS, STAGES>, (unsigned)grid, THREADS,
                 (size_t)smem_bytes<BS>(stages), s, map_B, map_A, n_tiles, a.n_rhs, (int)a.cols, (int)(a.nnzb * BS), stages,
                 a.block_row_ptr, a.block_col_idx, static_cast<__nv_bfloat16 *>(a.C), status);
  return cudaGetLastError();
}

template <bool PER_CTA_STATUS, int BS>
cudaError_t launch_tcgen05(const BsrSpmmArgs &a, int *status, int sm_count, cudaStream_t s) {
  const int64_t n_tiles = ceil_div(a.n_rhs, TILE_N), grid = a.rows / BS * n_tiles;
  if (grid == 0) return cudaSuccess;
  if (grid > 2147483647LL) return cudaErrorInvalidConfiguration;
  const int stages = stages_for<BS>(grid, sm_count);
  if (stages == 3) return launch_stages<PER_CTA_STATUS, BS, 3>(a, status, stages, grid, n_tiles, s);
  return launch_stages<PER_CTA_STATUS, BS, 0>(a, status, stages, grid, n_tiles, s);
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
// One status word per CTA (block row x tile of 256 columns), hence the limit
// of SWB_STATIC_MAX_CTAS CTAs per call.  All calls share the array and a call
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
  const int64_t n_tiles = ceil_div(n_rhs, TILE_N);
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
  e = launch_tcgen05<true, 16>(a, status, DeviceInfo().sm_count, s);
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
