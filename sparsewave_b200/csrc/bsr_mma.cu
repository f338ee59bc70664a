// BSR SpMM for 8x8, 16x16 and 32x32 bf16 blocks with warp-level MMAs, operands from global memory straight into their
// fragments: any number of columns, any alignment, few block rows as well as many (arithmetic as in bsr_tcgen05.cu).
//
// A warp owns a block row and 16 T columns and forms the product transposed, so that one instruction shape fits all block
// sizes: mma.sync.m16n8k16 with m = 16 columns of B, n = 8 rows of a block, k = 16 local columns (two 8 x 8 blocks, one
// 16 x 16 block, half of a 32 x 32 block).  Which local column is which k, and which column of B which m, is free as long as
// both operands agree.  Lane (g, q) = (lane / 4, lane % 4) takes adjacent local columns ROWS q .. ROWS q + ROWS - 1 and
// adjacent columns 2 T g .. 2 T g + 2 T - 1: its share of the block values is one load per 8 rows, its share of a row of B one
// load of up to 16 bytes, and its results are adjacent columns of C.  Pairs of rows of B are interleaved by byte permutes.
// The next steps' loads are in flight during this step's MMAs, block columns are held 32 at a time by the warp's lanes.
// Where block rows are few, up to eight warps share one and its parts are added up through shared memory in their order.
//
// What bounds it: launch and latency on small calls, L1 on large ones (eight lanes of a load touch four lines, some 64 lookups
// for 2 KB of B; ncu: L1 data pipe 67 %, tensor pipe 18 % on 1,024 block rows of 51, N = 512), which bsr_tcgen05.cu then takes.
// Tried: the same loads through a ring in shared memory (178 us against 134 on that size).  Before, on the CUDA cores or with
// tcgen05 at any size: 123 block rows of 61 blocks of 32 x 32, N = 2 138 -> 6.2 us; 382 of 27, N = 29 111 -> 17.6; 1,438 of 15
// blocks of 8 x 8, N = 80 30.6 -> 10.4; 73 of 36 blocks of 16 x 16, N = 88 18.5 -> 5.9.
#include <cuda_bf16.h>

#include "swb_chain.cuh"
#include "swb_index.h"
#include "swb_kernels.h"

namespace swb {
namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int MMA_WARPS = 8;
// Steps in hand (one being multiplied, the others' loads in flight) and CTAs per SM that registers are kept for.  Narrow B leaves
// registers for more of both: 1,628 block rows of 14 blocks of 16 x 16, N = 24 9.8 -> 6.8 us with three CTAs; 2,970 of 52, N = 8
// 36.9 -> 30.0 with three steps and CTAs (37.6 with four CTAs of two steps, 37.1 with two of four).
// 8 x 8 blocks then have three CTAs for four: 2,744 block rows of 54, N = 16 15.3 -> 12.7, but 7,454 of 44, N = 8 20.7 -> 24.0.
constexpr int mma_depth(int bs, int T) { return bs == 32 || T > 1 ? 2 : 3; }
constexpr int mma_ctas(int bs, int T, int V) { return bs < 32 && T == 1 ? 3 : bs == 16 && T == 2 && V > 1 ? 3 : 2; }

template <int BS, int T, int V>
struct Fragments {
  static constexpr int ROWS = BS == 32 ? 8 : 4;   // rows of B per lane and step
  static constexpr int TILES = BS / 8;            // n8 tiles of block rows
  uint32_t slab[ROWS][T + (V == 0)];              // 2 T adjacent columns each (V = 0: the words that hold them)
  uint32_t block[TILES][ROWS / 2];                // block row 8 u + g, the lane's ROWS columns
};

// 2 T adjacent elements as loads of V (those at or past `valid` are zeros), two to a word.
template <int T, int V>
__device__ __forceinline__ void load_row(uint32_t (&w)[T], const __nv_bfloat16 *p, int valid) {
  if constexpr (V == 8) {
    static_assert(T == 4, "");
    uint4 t = make_uint4(0, 0, 0, 0);
    if (valid > 0) t = __ldg(reinterpret_cast<const uint4 *>(p));
    w[0] = t.x; w[1] = t.y; w[2] = t.z; w[3] = t.w;
  } else if constexpr (V == 4) {
#pragma unroll
    for (int i = 0; i < T / 2; ++i) {
      uint2 t = make_uint2(0, 0);
      if (4 * i < valid) t = __ldg(reinterpret_cast<const uint2 *>(p + 4 * i));
      w[2 * i] = t.x; w[2 * i + 1] = t.y;
    }
  } else if constexpr (V == 2) {
#pragma unroll
    for (int i = 0; i < T; ++i) {
      w[i] = 0;
      if (2 * i < valid) w[i] = __ldg(reinterpret_cast<const unsigned *>(p + 2 * i));
    }
  } else {
    const unsigned short *h = reinterpret_cast<const unsigned short *>(p);
#pragma unroll
    for (int i = 0; i < T; ++i) {
      unsigned lo = 0, hi = 0;
      if (2 * i < valid) lo = __ldg(h + 2 * i);
      if (2 * i + 1 < valid) hi = __ldg(h + 2 * i + 1);
      w[i] = lo | hi << 16;
    }
  }
}
// The T + 1 aligned words that hold 2 T adjacent elements, of which the first `valid` matter (`odd`: they start in the middle
// of a word).  A word that holds one of those lies in B, which has an even number of elements and starts at a word.
template <int T>
__device__ __forceinline__ void load_words(uint32_t (&w)[T + 1], const __nv_bfloat16 *p, int odd, int valid) {
  const unsigned *word = reinterpret_cast<const unsigned *>(p - odd);
#pragma unroll
  for (int i = 0; i <= T; ++i) {
    w[i] = 0;
    if (valid > 0 && 2 * i - odd < valid && (i < T || odd)) w[i] = __ldg(word + i);
  }
}
template <int T, int V>
__device__ __forceinline__ void store_row(__nv_bfloat16 *p, const uint32_t (&w)[T], int valid) {
  if constexpr (V == 8) {
    if (valid > 0) *reinterpret_cast<uint4 *>(p) = make_uint4(w[0], w[1], w[2], w[3]);
  } else if constexpr (V == 4) {
#pragma unroll
    for (int i = 0; i < T / 2; ++i)
      if (4 * i < valid) *reinterpret_cast<uint2 *>(p + 4 * i) = make_uint2(w[2 * i], w[2 * i + 1]);
  } else if constexpr (V == 2) {
#pragma unroll
    for (int i = 0; i < T; ++i)
      if (2 * i < valid) *reinterpret_cast<uint32_t *>(p + 2 * i) = w[i];
  } else {
    unsigned short *h = reinterpret_cast<unsigned short *>(p);
#pragma unroll
    for (int i = 0; i < T; ++i) {
      if (2 * i < valid) h[2 * i] = (unsigned short)w[i];
      if (2 * i + 1 < valid) h[2 * i + 1] = (unsigned short)(w[i] >> 16);
    }
  }
}

__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                    uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// V: elements per load of a row of B, or 0: N is odd and B starts at a word, so that rows in turn start at a word and in the
// middle of one.  WIDE: block values are aligned for loads of a lane's ROWS.
template <int BS, int T, int V, bool WIDE>
__global__ void __launch_bounds__(32 * MMA_WARPS, mma_ctas(BS, T, V))
    bsr_spmm_mma_kernel(int64_t units, int tiles, int split, int64_t N, const int32_t *__restrict__ brp,
                        const int32_t *__restrict__ bci, const __nv_bfloat16 *__restrict__ bv,
                        const __nv_bfloat16 *__restrict__ B, __nv_bfloat16 *__restrict__ C) {
  using F = Fragments<BS, T, V>;
  constexpr int BLOCKS = BS == 8 ? 2 : 1;  // blocks per step
  constexpr int BATCH = 32 / BLOCKS;       // steps whose block columns the warp holds
  after_previous_kernel();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  const int part = warp % split;
  const int64_t unit = (int64_t)blockIdx.x * (MMA_WARPS / split) + warp / split;
  const bool active = unit < units;
  const int64_t brow = active ? unit / tiles : 0;
  const int64_t col0 = (active ? unit - brow * tiles : 0) * (16 * T) + g * (2 * T);
  const int valid = N - col0 >= 2 * T ? 2 * T : N > col0 ? (int)(N - col0) : 0;
  int start = 0, end = 0;
  if (active) {
    start = brp[brow];
    end = brp[brow + 1];
  }
  const int steps = (end - start + BLOCKS - 1) / BLOCKS;
  const int share = (steps + split - 1) / split;
  const int k0 = part * share, k1 = k0 + share < steps ? k0 + share : steps;

  float acc[F::TILES][T][4];
#pragma unroll
  for (int u = 0; u < F::TILES; ++u)
#pragma unroll
    for (int t = 0; t < T; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[u][t][i] = 0.0f;

  const __nv_bfloat16 *Bt = B + col0 + (int64_t)(BS == 8 ? 4 * (q & 1) : F::ROWS * q) * N;
  auto column = [&](int k) {  // block columns of the steps from k on
    const int p = start + k * BLOCKS + lane;
    return p < end ? __ldg(bci + p) : 0;
  };
  int here = 0, ahead = 0;
  auto load = [&](F &f, int k) {
    const int i = k - k0;
    if (i % BATCH == 0 && i != 0) { here = ahead; ahead = column(k + BATCH); }
    const int j = BS == 8 ? q >> 1 : 0;
    const int bc = __shfl_sync(FULL, here, (i % BATCH) * BLOCKS + j);
    const int p = start + k * BLOCKS + j;
    const bool in = BS != 8 || p < end;  // the second block of a last step may be missing: zeros
    const __nv_bfloat16 *b = Bt + (int64_t)bc * BS * N;
#pragma unroll
    for (int r = 0; r < F::ROWS; ++r) {
      if constexpr (V == 0) load_words<T>(f.slab[r], b + r * N, r & 1, in ? valid : 0);
      else load_row<T, V>(f.slab[r], b + r * N, in ? valid : 0);
    }
    const __nv_bfloat16 *a = bv + (int64_t)p * (BS * BS) + g * BS + (BS == 8 ? 4 * (q & 1) : F::ROWS * q);
#pragma unroll
    for (int u = 0; u < F::TILES; ++u) load_row<F::ROWS / 2, WIDE ? F::ROWS : 1>(f.block[u], a + u * 8 * BS, in ? F::ROWS : 0);
  };
  auto compute = [&](const F &f) {
#pragma unroll
    for (int r = 0; r < F::ROWS; r += 4)
#pragma unroll
      for (int t = 0; t < T; ++t) {
        uint32_t x[4];  // columns 2 t and 2 t + 1 of four rows
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if constexpr (V == 0) x[i] = i & 1 ? __byte_perm(f.slab[r + i][t], f.slab[r + i][t + 1], 0x5432) : f.slab[r + i][t];
          else x[i] = f.slab[r + i][t];
        }
        const uint32_t a0 = __byte_perm(x[0], x[1], 0x5410), a1 = __byte_perm(x[0], x[1], 0x7632);
        const uint32_t a2 = __byte_perm(x[2], x[3], 0x5410), a3 = __byte_perm(x[2], x[3], 0x7632);
#pragma unroll
        for (int u = 0; u < F::TILES; ++u) mma(acc[u][t], a0, a1, a2, a3, f.block[u][r / 2], f.block[u][r / 2 + 1]);
      }
  };
  if (k0 < k1) {
    here = column(k0);
    ahead = column(k0 + BATCH);
    constexpr int DEPTH = mma_depth(BS, T);
    F f[DEPTH];
#pragma unroll
    for (int d = 0; d < DEPTH - 1; ++d)
      if (k0 + d < k1) load(f[d], k0 + d);
    for (int k = k0; k < k1;) {
#pragma unroll
      for (int d = 0; d < DEPTH; ++d) {
        if (k + DEPTH - 1 < k1) load(f[(d + DEPTH - 1) % DEPTH], k + DEPTH - 1);
        compute(f[d]);
        if (++k >= k1) break;
      }
    }
  }
  if (split > 1) {  // the parts' sums, added up by the unit's first warp in order
    constexpr int WORDS = F::TILES * T * 4;
    extern __shared__ __align__(16) float partial[];
    float *mine = partial + (warp - warp / split - 1) * (WORDS * 32) + lane;
    if (part > 0) {
#pragma unroll
      for (int i = 0; i < WORDS; ++i) mine[i * 32] = acc[i / (4 * T)][i / 4 % T][i % 4];
    }
    __syncthreads();
    if (part > 0) return;
    mine += WORDS * 32;
    for (int s = 1; s < split; ++s, mine += WORDS * 32)
#pragma unroll
      for (int i = 0; i < WORDS; ++i) acc[i / (4 * T)][i / 4 % T][i % 4] += mine[i * 32];
  }
  if (!active) return;
#pragma unroll
  for (int u = 0; u < F::TILES; ++u)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      uint32_t w[T];
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(acc[u][t][r], acc[u][t][2 + r]);
        w[t] = *reinterpret_cast<const uint32_t *>(&h);
      }
      store_row<T, V ? V : 1>(C + (brow * BS + 8 * u + 2 * q + r) * N + col0, w, valid);
    }
}

template <int BS, int T, int V, bool WIDE>
cudaError_t launch_mma(const BsrSpmmArgs &a, int sm_count, cudaStream_t s) {
  const int64_t tiles = ceil_div(a.n_rhs, 16 * T), units = a.rows / BS * tiles;
  // Parts of a block row: while there are fewer than 16 warps per SM and a part keeps 64 rows of B (140 block rows of 47 blocks
  // of 16 x 16, N = 4: 17.5 us whole, 4.7 in eight parts; 303 of 5, N = 504: 8.0 whole, 13.2 in four).
  int split = 1;
  while (split < MMA_WARPS && units * split < (int64_t)sm_count * 16 && a.nnzb * BS * BS >= split * 64 * a.rows) split *= 2;
  unsigned grid = 0;
  if (!grid_dim(ceil_div(units * split, MMA_WARPS), &grid)) return cudaErrorInvalidConfiguration;
  const size_t smem = (size_t)(MMA_WARPS - MMA_WARPS / split) * (BS / 8 * T * 4 * 32) * 4;
  launch_chained(bsr_spmm_mma_kernel<BS, T, V, WIDE>, grid, 32 * MMA_WARPS, smem, s, units, (int)tiles, split, a.n_rhs,
                 a.block_row_ptr, a.block_col_idx, static_cast<const __nv_bfloat16 *>(a.block_values),
                 static_cast<const __nv_bfloat16 *>(a.B), static_cast<__nv_bfloat16 *>(a.C));
  return cudaGetLastError();
}

template <int BS, int T, int V>
cudaError_t launch_wide(const BsrSpmmArgs &a, int sm_count, cudaStream_t s) {
  const bool wide = reinterpret_cast<uintptr_t>(a.block_values) % (BS == 32 ? 16 : 8) == 0;
  return wide ? launch_mma<BS, T, V, true>(a, sm_count, s) : launch_mma<BS, T, V, false>(a, sm_count, s);
}

template <int BS>
cudaError_t launch_bs(const BsrSpmmArgs &a, int sm_count, cudaStream_t s) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(a.B) | reinterpret_cast<uintptr_t>(a.C) | (uintptr_t)(a.n_rhs * 2);
  const int64_t n = a.n_rhs;
  // 64 columns per warp, fewer for narrow B; two-byte loads and the 32 rows of a large block leave registers for 32
  // (706 block rows of 9, N = 302 off a word: 22.9 us with 64, 19.5 with 32).
  const bool words = n % 2 == 1 && reinterpret_cast<uintptr_t>(a.B) % 4 == 0;
  const int T = n <= 16 ? 1 : n <= 32 || BS == 32 || (at % 4 != 0 && !words) ? 2 : 4;
  if (T == 1)
    return words ? launch_wide<BS, 1, 0>(a, sm_count, s) : at % 4 == 0 ? launch_wide<BS, 1, 2>(a, sm_count, s)
                                                                     : launch_wide<BS, 1, 1>(a, sm_count, s);
  if (T == 2)
    return words ? launch_wide<BS, 2, 0>(a, sm_count, s) : at % 8 == 0 ? launch_wide<BS, 2, 4>(a, sm_count, s)
           : at % 4 == 0 ? launch_wide<BS, 2, 2>(a, sm_count, s) : launch_wide<BS, 2, 1>(a, sm_count, s);
  if constexpr (BS != 32)
    return words ? launch_wide<BS, 4, 0>(a, sm_count, s) : at % 16 == 0 ? launch_wide<BS, 4, 8>(a, sm_count, s)
           : at % 8 == 0 ? launch_wide<BS, 4, 4>(a, sm_count, s)
                                                                             : launch_wide<BS, 4, 2>(a, sm_count, s);
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_bsr_spmm_mma(const BsrSpmmArgs &a, const DeviceInfo &dev, cudaStream_t s, int64_t *launches) {
  if (a.rows == 0) return cudaSuccess;
  ++*launches;
  switch (a.block_size) {
    case 8: return launch_bs<8>(a, dev.sm_count, s);
    case 16: return launch_bs<16>(a, dev.sm_count, s);
    case 32: return launch_bs<32>(a, dev.sm_count, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace swb
