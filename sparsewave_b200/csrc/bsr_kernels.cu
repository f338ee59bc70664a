// BSR SpMM, thread-per-output mapping (ThreadPerOutputBSRSpMMPattern, SparseWaveToGPU.cpp:560-665): row = element / N,
// column = element % N, block row = row / bs, local row = row % bs; for every block of the block row, in storage order,
// and every local column in ascending order: sum += value * B[block_col*bs + lc, column].  f32 blocks (the element type
// of the reference's runtime tests) and bf16 blocks with f32 accumulation and one final rounding to bf16.
//
// A thread holds TR rows of one block row and V adjacent columns: a value of B serves TR outputs and a value of a block V
// of them, where one thread per output reads both for every product.  Every output is still added up in the reference's
// order, bit for bit.  Block values are the same for all threads of a block row (one L1 access per load), rows of B are
// read V columns at a time.  With products and sums separate instructions the bound is the FP32 pipe (19 T products and sums a
// second), then the gather of slabs of B from L2: f32, 32,768 block rows of 24 blocks of 2 x 2, N = 32 23.3 us (201 M products: 10.6
// us of FP32 pipe); 4,096 of 20 of 16 x 16, N = 64 218 us (1.34 G: 71); bf16, 16,384 of 24 of 4 x 4, N = 32 43.5 us (180 with one
// output per thread; f32 alike).  f32 blocks of 4 x 4 and 8 x 8 with enough outputs go on to groups of lanes (bsr_rows.cuh), bf16
// blocks of 8, 16 and 32 to tensor cores.
#include <cuda_bf16.h>

#include "swb_chain.cuh"
#include "swb_index.h"
#include "swb_kernels.h"

namespace swb {
namespace {

__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }

// n adjacent elements as one load (their address is a multiple of their size), widened to f32.
template <int n>
__device__ __forceinline__ void load(float (&out)[n], const float *p) {
  if constexpr (n == 4) {
    const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
    out[0] = t.x; out[1] = t.y; out[2] = t.z; out[3] = t.w;
  } else if constexpr (n == 2) {
    const float2 t = __ldg(reinterpret_cast<const float2 *>(p));
    out[0] = t.x; out[1] = t.y;
  } else {
#pragma unroll
    for (int k = 0; k < n; ++k) out[k] = __ldg(p + k);
  }
}
__device__ __forceinline__ float low_half(unsigned u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float high_half(unsigned u) { return __uint_as_float(u & 0xffff0000u); }
template <int n>
__device__ __forceinline__ void load(float (&out)[n], const __nv_bfloat16 *p) {
  if constexpr (n == 4) {
    const uint2 t = __ldg(reinterpret_cast<const uint2 *>(p));
    out[0] = low_half(t.x); out[1] = high_half(t.x); out[2] = low_half(t.y); out[3] = high_half(t.y);
  } else if constexpr (n == 2) {
    const unsigned t = __ldg(reinterpret_cast<const unsigned *>(p));
    out[0] = low_half(t); out[1] = high_half(t);
  } else {
#pragma unroll
    for (int k = 0; k < n; ++k) out[k] = __bfloat162float(__ldg(p + k));
  }
}
template <int n>
__device__ __forceinline__ void store(float *p, const float (&v)[n]) {
  if constexpr (n == 4) *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else if constexpr (n == 2) *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
  else *p = v[0];
}
template <int n>
__device__ __forceinline__ void store(__nv_bfloat16 *p, const float (&v)[n]) {
  if constexpr (n == 1) {
    *p = __float2bfloat16_rn(v[0]);
  } else {
    __nv_bfloat162 t[n / 2];
#pragma unroll
    for (int k = 0; k < n / 2; ++k) t[k] = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
    if constexpr (n == 4) *reinterpret_cast<uint2 *>(p) = *reinterpret_cast<const uint2 *>(t);
    else *reinterpret_cast<unsigned *>(p) = *reinterpret_cast<const unsigned *>(t);
  }
}

// 4 x 4 blocks with four rows per thread: 72 registers, so that seven blocks fit an SM, at the price of 48 (f32) and 32 (bf16)
// bytes of spills with aligned block values and four columns.
constexpr int TILE_THREADS = 128;
template <int n> struct Count { static constexpr int value = n; };

// BS: the block size where it is a constant (K = BS or 4 local columns per load), or 0: any bs.  TR rows per thread.
// WIDE: block values are aligned for loads of K.
template <typename T, int BS, int TR, int V, bool WIDE>
__global__ void __launch_bounds__(TILE_THREADS, BS == 4 && TR == 4 ? 7 : 1) bsr_spmm_row_tile_kernel(int64_t brows, int64_t N, int64_t block_size, int tiles,
                                                                const int32_t *__restrict__ brp,
                                                                const int32_t *__restrict__ bci,
                                                                const T *__restrict__ bv, const T *__restrict__ B,
                                                                T *__restrict__ C) {
  after_previous_kernel();
  constexpr bool WHOLE = BS == TR;  // one tile per block row
  constexpr int K = BS ? (BS % 4 == 0 ? 4 : BS) : 4;
  constexpr bool AHEAD = (BS == 3 || BS == 4 || BS == 8) && WHOLE;  // rows of B requested a step ahead of their sums
  const int64_t bs = BS ? BS : block_size, G = N / V;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t unit = t / G, g = t - unit * G;
  const int64_t brow = WHOLE ? unit : unit / tiles;
  if (brow >= brows) return;
  const int r0 = WHOLE ? 0 : (int)(unit - brow * tiles) * TR;
  const T *Bt = B + g * V;
  float acc[TR][V];
#pragma unroll
  for (int r = 0; r < TR; ++r)
#pragma unroll
    for (int j = 0; j < V; ++j) acc[r][j] = 0.0f;

  // W local columns from lc on, whose rows of B are in bw: block values, then sums in local-column order.
  auto sums = [&](const T *a, int lc, const auto &bw, auto width) {
    constexpr int W = decltype(width)::value;
#pragma unroll
    for (int r = 0; r < TR; ++r) {
      // a tile that reaches past the block repeats its last row, which is not stored
      const int64_t row = WHOLE ? r : BS ? r0 + r : (r0 + r < bs ? r0 + r : bs - 1);
      float aw[W];
      const T *p = a + row * bs + lc;
      if constexpr (WIDE && W > 1) {
        load<W>(aw, p);
      } else {
#pragma unroll
        for (int k = 0; k < W; ++k) {
          float one[1];
          load<1>(one, p + k);
          aw[k] = one[0];
        }
      }
#pragma unroll
      for (int k = 0; k < W; ++k)
#pragma unroll
        for (int j = 0; j < V; ++j) acc[r][j] = add(acc[r][j], mul(aw[k], bw[k][j]));
    }
  };

  const int start = brp[brow], end = brp[brow + 1];
  const int64_t block = bs * bs;
  if (start < end) {
    // Block columns are read two blocks ahead.  For blocks of 3, 4 and 8 the rows of B of the next step are requested
    // before the sums of this one, and block values, which lie in storage order, are pulled into L1 three blocks ahead
    // (4 x 4 blocks, 24 per block row, N = 32: 84 -> 43 us); smaller blocks lose by the copies, larger ones have enough
    // rows of B in flight.
    int bc = __ldg(bci + start);
    int next = start + 1 < end ? __ldg(bci + start + 1) : bc;
    const T *a = bv + (int64_t)start * block;
    const int whole = BS ? BS / K * K : (int)(bs / K * K);
    float bn[K][V];
    auto request = [&](int column, int lc) {
      const T *b = Bt + ((int64_t)column * bs + lc) * N;
#pragma unroll
      for (int k = 0; k < K; ++k) load<V>(bn[k], b + (int64_t)k * N);
    };
    if (AHEAD) request(bc, 0);
    for (int bp = start; bp < end; ++bp, a += block) {
      const int after = end - bp > 2 ? __ldg(bci + bp + 2) : next;
      if (AHEAD && end - bp > 3) asm volatile("prefetch.global.L1 [%0];" ::"l"(a + 3 * block));
#pragma unroll
      for (int lc = 0; lc < whole; lc += K) {
        if (!AHEAD) request(bc, lc);
        float bw[K][V];
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
          for (int j = 0; j < V; ++j) bw[k][j] = bn[k][j];
        if (AHEAD) {
          if (lc + K < whole) request(bc, lc + K);
          else if (bp + 1 < end) request(next, 0);
        }
        sums(a, lc, bw, Count<K>());
      }
      if constexpr (BS == 0) {
        for (int lc = whole; lc < bs; ++lc) {
          float bw[1][V];
          load<V>(bw[0], Bt + ((int64_t)bc * bs + lc) * N);
          sums(a, lc, bw, Count<1>());
        }
      }
      bc = next;
      next = after;
    }
  }
#pragma unroll
  for (int r = 0; r < TR; ++r)
    if (BS || r0 + r < bs) store<V>(C + (brow * bs + r0 + r) * N + g * V, acc[r]);
}

template <typename T, int BS, int TR, int V>
cudaError_t launch_tiles(const BsrSpmmArgs &a, cudaStream_t s) {
  const int64_t bs = a.block_size, brows = a.rows / bs, tiles = ceil_div(bs, TR);
  unsigned grid = 0;  // refused, not truncated, beyond the CUDA grid limit
  if (!grid_dim(ceil_div(brows * tiles * (a.n_rhs / V), TILE_THREADS), &grid)) return cudaErrorInvalidConfiguration;
  // loads of K values start at multiples of K from an aligned base (K divides bs where BS is constant)
  const bool wide = reinterpret_cast<uintptr_t>(a.block_values) % (4 * sizeof(T)) == 0 && (BS == 2 || bs % 4 == 0);
#define SWB_BSR(WIDE)                                                                                             \
  launch_chained(bsr_spmm_row_tile_kernel<T, BS, TR, V, WIDE>, grid, TILE_THREADS, 0, s,                          \
      brows, a.n_rhs, bs, (int)tiles, a.block_row_ptr, a.block_col_idx, static_cast<const T *>(a.block_values), \
      static_cast<const T *>(a.B), static_cast<T *>(a.C))
  if (wide) SWB_BSR(true); else SWB_BSR(false);
#undef SWB_BSR
  return cudaGetLastError();
}

template <typename T, int V>
cudaError_t launch_columns(const BsrSpmmArgs &a, bool few, cudaStream_t s) {
  switch (a.block_size) {
    case 1: return launch_tiles<T, 1, 1, V>(a, s);
    case 2: return launch_tiles<T, 2, 2, V>(a, s);
    case 3: return launch_tiles<T, 3, 3, V>(a, s);
    case 4: return few ? launch_tiles<T, 4, 2, V>(a, s) : launch_tiles<T, 4, 4, V>(a, s);
  }
  if constexpr (sizeof(T) == sizeof(float))  // 8 x 8 blocks in bf16 run on tensor cores
    if (a.block_size == 8) return few ? launch_tiles<T, 8, 2, V>(a, s) : launch_tiles<T, 8, 8, V>(a, s);
  return few ? launch_tiles<T, 0, 2, V>(a, s) : launch_tiles<T, 0, 8, V>(a, s);
}

#include "bsr_rows.cuh"

template <typename T>
cudaError_t launch(const BsrSpmmArgs &a, cudaStream_t s, int64_t *launches) {
  ++*launches;
  // As many columns per thread, up to four, as rows of B and C are aligned to; small blocks keep 65,536 threads, enough to
  // hide the gathers (larger ones have more rows of B in flight per thread: 16 x 16 blocks, 20 per block row, N = 64
  // 77 us with four columns, 176 with one).  Two rows per thread where eight would leave less than 20,000 threads
  // (201 block rows of 52 blocks of 32 x 32, N = 24: 207 us with eight, 122 with two).
  const uintptr_t at = reinterpret_cast<uintptr_t>(a.B) | reinterpret_cast<uintptr_t>(a.C);
  int V = a.n_rhs % 4 == 0 && at % (4 * sizeof(T)) == 0 ? 4 : a.n_rhs % 2 == 0 && at % (2 * sizeof(T)) == 0 ? 2 : 1;
  if constexpr (sizeof(T) == sizeof(float)) {
    cudaError_t e = cudaSuccess;
    if (a.block_size == 4 && try_groups<4>(a, V, s, &e)) return e;
    if (a.block_size == 8 && try_groups<8>(a, V, s, &e)) return e;
  }
  if (a.block_size <= 8)
    while (V > 1 && a.rows / a.block_size * (a.n_rhs / V) < 65536) V /= 2;
  const bool few = a.rows / a.block_size * ceil_div(a.block_size, 8) * (a.n_rhs / V) < 20000;
  if (V == 4) return launch_columns<T, 4>(a, few, s);
  return V == 2 ? launch_columns<T, 2>(a, few, s) : launch_columns<T, 1>(a, few, s);
}

}  // namespace

cudaError_t launch_bsr_spmm_thread_per_output_f32(const BsrSpmmArgs &a, cudaStream_t s, int64_t *launches) {
  return launch<float>(a, s, launches);
}

cudaError_t launch_bsr_spmm_thread_per_output_bf16(const BsrSpmmArgs &a, cudaStream_t s, int64_t *launches) {
  return launch<__nv_bfloat16>(a, s, launches);
}

}  // namespace swb
