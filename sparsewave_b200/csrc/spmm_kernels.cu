// CSR SpMM kernels for sm_100a: thread-per-output, wave-per-row-tile and
// thread-per-position mappings of sparsewave.spmm.  B is cols x N and C is
// rows x N, row-major.  Products and sums are separate f32 operations.
#include "swb_chain.cuh"
#include "swb_index.h"
#include "swb_kernels.h"

namespace swb {
namespace {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }

// thread-per-output (ThreadPerOutputSpMMPattern, SparseWaveToGPU.cpp:489-558): sequential sums in position order,
// bit-identical to the CPU CSR loop.
#include "spmm_columns.cuh"
#include "spmm_staged_rows.cuh"
#include "spmm_team_rows.cuh"

// The reference's schedule itself: a thread per output, element = blockIdx * blockDim + threadIdx, row = element / N.  On very
// short rows there is nothing to stage and little to wait for; see takes_outputs.
__global__ void __launch_bounds__(256)
    spmm_thread_per_output_kernel(int64_t rows, uint32_t N, const int32_t *__restrict__ row_ptr,
                                  const int32_t *__restrict__ col, const float *__restrict__ val,
                                  const float *__restrict__ B, float *__restrict__ C) {
  after_previous_kernel();
  const int64_t first = (int64_t)blockIdx.x * 256, r0 = first / N;  // the same for the block
  const uint32_t from = (uint32_t)(first - r0 * N) + threadIdx.x;
  const int64_t row = r0 + from / N;
  if (row >= rows) return;
  const float *Bj = B + from % N;
  int p = row_ptr[row];
  const int end = row_ptr[row + 1];
  float sum = 0.0f;
  for (; end - p >= 4; p += 4) {
    const int c0 = __ldg(col + p), c1 = __ldg(col + p + 1), c2 = __ldg(col + p + 2), c3 = __ldg(col + p + 3);
    const float v0 = __ldg(val + p), v1 = __ldg(val + p + 1), v2 = __ldg(val + p + 2), v3 = __ldg(val + p + 3);
    const float b0 = __ldg(Bj + (int64_t)c0 * N), b1 = __ldg(Bj + (int64_t)c1 * N);
    const float b2 = __ldg(Bj + (int64_t)c2 * N), b3 = __ldg(Bj + (int64_t)c3 * N);
    sum = add(add(add(add(sum, mul(v0, b0)), mul(v1, b1)), mul(v2, b2)), mul(v3, b3));
  }
  for (; p < end; ++p) sum = add(sum, mul(__ldg(val + p), __ldg(Bj + (int64_t)__ldg(col + p) * N)));
  C[first + threadIdx.x] = sum;
}

// ---------------------------------------------------------------------------
// wave-per-row-tile (WavePerRowTileSpMMPattern, SparseWaveToGPU.cpp:1057-1256)
// tiles = ceil(N / T); unit = blockIdx * (blockDim/32) + threadIdx/32;
// row = unit / tiles; tile = unit % tiles; first column = tile * T.  Lanes
// stride the row's positions; each position's value is loaded once and used
// for the T right-hand-side columns of the tile.  A tile that reaches past N
// runs the guarded path.
//
// TCAP is T rounded up to a power of two (columns k >= T are inactive).  Full
// tiles of 4, 8, 16 or 32 columns on 16-byte aligned operands take the
// vectorised kernel further below instead.
//
// Reduction: instead of T independent 5-step butterflies (5*T shuffles) the
// warp does a halving exchange: at the step with lane distance `off` each
// lane keeps one half of its accumulators and sends the other half to its
// partner, so the accumulator count halves per step until one is left
// (TCAP-1 shuffles), then plain butterfly steps finish.  Lane l ends with the
// full sum of column (l >> (5 - log2 TCAP)) of the tile.
// ---------------------------------------------------------------------------
template <int TCAP>
__device__ __forceinline__ void tile_reduce(float (&acc)[TCAP], int lane) {
  int w = TCAP;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    if (w > 1) {
      const int half = w >> 1;
      const bool upper = (lane & off) != 0;
#pragma unroll
      for (int i = 0; i < TCAP / 2; ++i) {
        if (i < half) {
          const float send = upper ? acc[i] : acc[i + half];
          const float keep = upper ? acc[i + half] : acc[i];
          acc[i] = add(keep, __shfl_xor_sync(FULL, send, off));
        }
      }
      w = half;
    } else {
      acc[0] = add(acc[0], __shfl_xor_sync(FULL, acc[0], off));
    }
  }
}

// Column (within the tile) whose sum lane `lane` holds after tile_reduce.
template <int TCAP>
__device__ __forceinline__ int tile_column_of_lane(int lane) {
  int k = 0, w = TCAP;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    if (w > 1) {
      w >>= 1;
      if (lane & off) k += w;
    }
  }
  return k;
}

// Lowest lane holding column k: the lanes whose "kept" bits spell k and whose
// remaining low bits are zero.
template <int TCAP>
__device__ __forceinline__ bool lane_is_column_writer(int lane) {
  int w = TCAP, used = 0;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    if (w > 1) {
      w >>= 1;
      used |= off;
    }
  }
  return (lane & ~used) == 0;
}

template <int TCAP>
__global__ void spmm_wave_per_row_tile_kernel(int64_t rows, int64_t N, int T, int64_t tiles,
                                              const int32_t *__restrict__ row_ptr,
                                              const int32_t *__restrict__ col,
                                              const float *__restrict__ val,
                                              const float *__restrict__ B, float *__restrict__ C,
                                              bool accumulate) {
  after_previous_kernel();
  const int lane = threadIdx.x & 31;
  const int64_t unit = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (unit >= rows * tiles) return;
  const int64_t row = unit / tiles;
  const int64_t j0 = (unit % tiles) * T;
  const int start = row_ptr[row], end = row_ptr[row + 1];
  const bool full = j0 + T <= N;

  float acc[TCAP];
#pragma unroll
  for (int k = 0; k < TCAP; ++k) acc[k] = 0.0f;

  if (full && T == TCAP) {
    for (int p = start + lane; p < end; p += 32) {
      const int c = __ldcs(col + p);
      const float v = __ldcs(val + p);
      const float *b = B + (int64_t)c * N + j0;
#pragma unroll
      for (int k = 0; k < TCAP; ++k) acc[k] = add(acc[k], mul(v, __ldg(b + k)));
    }
  } else {
    // Guarded path: tail tile (or T below the register capacity).
    for (int p = start + lane; p < end; p += 32) {
      const int c = __ldcs(col + p);
      const float v = __ldcs(val + p);
      const float *b = B + (int64_t)c * N + j0;
#pragma unroll
      for (int k = 0; k < TCAP; ++k)
        if (k < T && j0 + k < N) acc[k] = add(acc[k], mul(v, __ldg(b + k)));
    }
  }

  tile_reduce<TCAP>(acc, lane);
  const int k = tile_column_of_lane<TCAP>(lane);
  if (lane_is_column_writer<TCAP>(lane) && k < T && j0 + k < N) {
    float *out = C + row * N + j0 + k;
    *out = accumulate ? add(*out, acc[0]) : acc[0];
  }
}

// Full tiles of 4, 8, 16 or 32 columns with 16-byte aligned B and C rows.  The
// unit <-> (row, tile) assignment is the same; inside the warp G = T/4 adjacent
// lanes share a position and read the tile's T floats of that B row as one
// contiguous run of G float4 (64 contiguous bytes per position for T = 16), and
// the 32/G lane groups stride the row's positions.  Each lane keeps one float4
// of partial sums.  Reduction over the lane groups: two halving exchanges (lane
// distance 16 keeps two of the four components, distance 8 keeps one), then
// plain butterfly steps down to distance G: 3 + log2(8/G) shuffles.
template <int G>
__global__ void spmm_wave_per_row_tile_vec_kernel(int64_t rows, int64_t N, int64_t tiles,
                                                  const int32_t *__restrict__ row_ptr,
                                                  const int32_t *__restrict__ col,
                                                  const float *__restrict__ val,
                                                  const float *__restrict__ B, float *__restrict__ C,
                                                  bool accumulate) {
  after_previous_kernel();
  constexpr int T = 4 * G, PG = 32 / G;
  const int lane = threadIdx.x & 31;
  const int64_t unit = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (unit >= rows * tiles) return;
  const int64_t row = unit / tiles;
  const int64_t j0 = (unit % tiles) * T;
  const int cq = lane % G, pg = lane / G;
  const int start = row_ptr[row], end = row_ptr[row + 1];
  const float *Bt = B + j0 + 4 * cq;

  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if constexpr (G >= 4) {
    // 32 positions per pass, read by the whole warp with one coalesced load of col and one of val and
    // handed to the lane groups by shuffles (see the fused-row kernel below); same order of additions
    auto fma4 = [&](float v, const float4 &b) {
      acc.x = add(acc.x, mul(v, b.x)); acc.y = add(acc.y, mul(v, b.y));
      acc.z = add(acc.z, mul(v, b.z)); acc.w = add(acc.w, mul(v, b.w));
    };
    int cn = start + lane < end ? __ldg(col + start + lane) : 0;
    float vn = start + lane < end ? __ldg(val + start + lane) : 0.0f;
    for (int base = start; base < end; base += 32) {
      const int cl = cn;
      const float vl = vn;
      const int mine = base + 32 + lane;
      cn = mine < end ? __ldg(col + mine) : 0;
      vn = mine < end ? __ldg(val + mine) : 0.0f;
      const int left = end - base < 32 ? end - base : 32;
      int j = 0;
      for (; j + 4 * PG <= left; j += 4 * PG) {
        const int k = j + pg;
        const int c0 = __shfl_sync(FULL, cl, k), c1 = __shfl_sync(FULL, cl, k + PG);
        const int c2 = __shfl_sync(FULL, cl, k + 2 * PG), c3 = __shfl_sync(FULL, cl, k + 3 * PG);
        const float4 b0 = __ldg(reinterpret_cast<const float4 *>(Bt + (int64_t)c0 * N));
        const float4 b1 = __ldg(reinterpret_cast<const float4 *>(Bt + (int64_t)c1 * N));
        const float4 b2 = __ldg(reinterpret_cast<const float4 *>(Bt + (int64_t)c2 * N));
        const float4 b3 = __ldg(reinterpret_cast<const float4 *>(Bt + (int64_t)c3 * N));
        const float v0 = __shfl_sync(FULL, vl, k), v1 = __shfl_sync(FULL, vl, k + PG);
        const float v2 = __shfl_sync(FULL, vl, k + 2 * PG), v3 = __shfl_sync(FULL, vl, k + 3 * PG);
        fma4(v0, b0); fma4(v1, b1); fma4(v2, b2); fma4(v3, b3);
      }
      for (; j < left; j += PG) {
        const int kk = j + pg;
        const int c0 = __shfl_sync(FULL, cl, kk & 31);
        const float v0 = __shfl_sync(FULL, vl, kk & 31);
        if (kk < left) fma4(v0, __ldg(reinterpret_cast<const float4 *>(Bt + (int64_t)c0 * N)));
      }
    }
  } else {
  int p = start + pg;
  for (; p + PG < end; p += 2 * PG) {
    const int c0 = __ldg(col + p), c1 = __ldg(col + p + PG);
    const float v0 = __ldg(val + p), v1 = __ldg(val + p + PG);
    const float4 b0 = __ldg(reinterpret_cast<const float4 *>(Bt + (int64_t)c0 * N));
    const float4 b1 = __ldg(reinterpret_cast<const float4 *>(Bt + (int64_t)c1 * N));
    acc.x = add(acc.x, mul(v0, b0.x)); acc.y = add(acc.y, mul(v0, b0.y));
    acc.z = add(acc.z, mul(v0, b0.z)); acc.w = add(acc.w, mul(v0, b0.w));
    acc.x = add(acc.x, mul(v1, b1.x)); acc.y = add(acc.y, mul(v1, b1.y));
    acc.z = add(acc.z, mul(v1, b1.z)); acc.w = add(acc.w, mul(v1, b1.w));
  }
  if (p < end) {
    const int c0 = __ldg(col + p);
    const float v0 = __ldg(val + p);
    const float4 b0 = __ldg(reinterpret_cast<const float4 *>(Bt + (int64_t)c0 * N));
    acc.x = add(acc.x, mul(v0, b0.x)); acc.y = add(acc.y, mul(v0, b0.y));
    acc.z = add(acc.z, mul(v0, b0.z)); acc.w = add(acc.w, mul(v0, b0.w));
  }
  }

  // distance 16: lanes with bit 4 set keep (z, w), the others (x, y)
  const bool up16 = (lane & 16) != 0;
  float k0 = up16 ? acc.z : acc.x, k1 = up16 ? acc.w : acc.y;
  const float s0 = up16 ? acc.x : acc.z, s1 = up16 ? acc.y : acc.w;
  k0 = add(k0, __shfl_xor_sync(FULL, s0, 16));
  k1 = add(k1, __shfl_xor_sync(FULL, s1, 16));
  // distance 8: lanes with bit 3 set keep the second of the two
  const bool up8 = (lane & 8) != 0;
  float r = up8 ? k1 : k0;
  const float s = up8 ? k0 : k1;
  r = add(r, __shfl_xor_sync(FULL, s, 8));
#pragma unroll
  for (int off = 4; off >= G; off >>= 1) r = add(r, __shfl_xor_sync(FULL, r, off));
  const int comp = (up16 ? 2 : 0) + (up8 ? 1 : 0);
  if ((lane & 7 & ~(G - 1)) == 0) {
    float *out = C + row * N + j0 + 4 * cq + comp;
    *out = accumulate ? add(*out, r) : r;
  }
}

// acc += v * b on four columns: products and sums rounded one by one.
__device__ __forceinline__ void add_products(float4 &acc, float v, const float4 &b) {
  acc.x = add(acc.x, mul(v, b.x)); acc.y = add(acc.y, mul(v, b.y));
  acc.z = add(acc.z, mul(v, b.z)); acc.w = add(acc.w, mul(v, b.w));
}

// Row c of B (a lane's columns of it), rows `pitch` bytes apart: one 32 x 32 -> 64 bit multiply-add, where 64-bit factors
// take four instructions (2,097,152 rows of 64, N = 64, where the board's power limit holds the clock down: 3.32 -> 3.22 ms;
// 110,000 ragged rows of 60: 151 -> 147 us).  N <= 512 in the kernels below.
__device__ __forceinline__ const float4 *row_of(const float *B, int c, uint32_t pitch) {
  return reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(B) + (uint64_t)(uint32_t)c * pitch);
}

// Whole rows of B of 16 to 128 floats (G = N/4 = 4 to 32 lanes per row): every tile of a matrix row is
// computed by one warp in one pass - the (row, tile) units of a row are fused - so the row's col/val
// stream is read once instead of once per tile and each nonzero fetches its B row as one contiguous
// run of 64 to 512 bytes.  The warp reads 32 positions of col and val with one coalesced load each (the
// next 32 are requested before the rows of B of the current ones) and hands them to the 32/G lane groups
// by shuffles; a group takes every (32/G)-th position, four rows of B in flight per group.  Reading col
// and val per group with broadcast loads instead costs one L1 request per position and group and was
// 16 % slower on 2 M rows of 64 nonzeros with N = 64 (3.46 -> 2.90 ms).  The partial float4 sums of the
// groups are added with butterfly steps and group 0 stores the row of C.
template <int G>
__global__ void spmm_wave_per_row_fused_kernel(int64_t rows, int64_t N, const int32_t *__restrict__ row_ptr,
                                               const int32_t *__restrict__ col, const float *__restrict__ val,
                                               const float *__restrict__ B, float *__restrict__ C,
                                               bool accumulate) {
  after_previous_kernel();
  constexpr int PG = 32 / G;
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int cq = lane % G, pg = lane / G;
  const int start = row_ptr[row], end = row_ptr[row + 1];
  const float *Bt = B + 4 * cq;
  const uint32_t pitch = (uint32_t)N * 4u;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  auto fma4 = [&](float v, const float4 &b) { add_products(acc, v, b); };
  // 32 positions per pass: one coalesced load of col and of val by the whole warp, handed to the lane
  // groups by shuffles (group pg takes positions base + pg, base + pg + PG, ... as before: same sums)
  int cn = start + lane < end ? __ldg(col + start + lane) : 0;
  float vn = start + lane < end ? __ldg(val + start + lane) : 0.0f;
  for (int base = start; base < end; base += 32) {
    const int cl = cn;
    const float vl = vn;
    const int mine = base + 32 + lane;  // the next pass is requested before this one's rows of B
    cn = mine < end ? __ldg(col + mine) : 0;
    vn = mine < end ? __ldg(val + mine) : 0.0f;
    const int left = end - base < 32 ? end - base : 32;  // positions of this pass
    int j = 0;  // warp-uniform: positions of the pass handed out so far (every lane joins every shuffle)
    for (; j + 4 * PG <= left; j += 4 * PG) {
      const int k = j + pg;  // position of this group inside the pass
      const int c0 = __shfl_sync(FULL, cl, k), c1 = __shfl_sync(FULL, cl, k + PG);
      const int c2 = __shfl_sync(FULL, cl, k + 2 * PG), c3 = __shfl_sync(FULL, cl, k + 3 * PG);
      const float4 b0 = __ldg(row_of(Bt, c0, pitch));
      const float4 b1 = __ldg(row_of(Bt, c1, pitch));
      const float4 b2 = __ldg(row_of(Bt, c2, pitch));
      const float4 b3 = __ldg(row_of(Bt, c3, pitch));
      const float v0 = __shfl_sync(FULL, vl, k), v1 = __shfl_sync(FULL, vl, k + PG);
      const float v2 = __shfl_sync(FULL, vl, k + 2 * PG), v3 = __shfl_sync(FULL, vl, k + 3 * PG);
      fma4(v0, b0); fma4(v1, b1); fma4(v2, b2); fma4(v3, b3);
    }
    for (; j + 2 * PG <= left; j += 2 * PG) {  // short rows and row ends: two rows of B in flight
      const int k = j + pg;
      const int c0 = __shfl_sync(FULL, cl, k), c1 = __shfl_sync(FULL, cl, k + PG);
      const float4 b0 = __ldg(row_of(Bt, c0, pitch));
      const float4 b1 = __ldg(row_of(Bt, c1, pitch));
      const float v0 = __shfl_sync(FULL, vl, k), v1 = __shfl_sync(FULL, vl, k + PG);
      fma4(v0, b0); fma4(v1, b1);
    }
    // the ragged end of the pass: every lane takes part in the shuffles, only lanes with a position add
    for (; j < left; j += PG) {
      const int kk = j + pg;
      const int c0 = __shfl_sync(FULL, cl, kk & 31);
      const float v0 = __shfl_sync(FULL, vl, kk & 31);
      if (kk < left) fma4(v0, __ldg(row_of(Bt, c0, pitch)));
    }
  }
#pragma unroll
  for (int off = G; off < 32; off <<= 1) {
    acc.x = add(acc.x, __shfl_xor_sync(FULL, acc.x, off));
    acc.y = add(acc.y, __shfl_xor_sync(FULL, acc.y, off));
    acc.z = add(acc.z, __shfl_xor_sync(FULL, acc.z, off));
    acc.w = add(acc.w, __shfl_xor_sync(FULL, acc.w, off));
  }
  if (pg == 0) {
    float4 *out = reinterpret_cast<float4 *>(C + row * N) + cq;
    if (accumulate) {
      const float4 old = *out;
      acc.x = add(old.x, acc.x); acc.y = add(old.y, acc.y); acc.z = add(old.z, acc.z); acc.w = add(old.w, acc.w);
    }
    *out = acc;
  }
}

// Rows of B of 4 * G floats with G no power of two (N = 12, 20, 24, 28, 36 ... 124): the same fusion with
// PG = 32 / G (rounded down) lane groups on PG * G of the warp's lanes; the other lanes only take part in the
// shuffles.  The groups' partial sums are added into group 0 one after the other.
__global__ void spmm_wave_per_row_any_kernel(int64_t rows, int64_t N, int G, const int32_t *__restrict__ row_ptr,
                                             const int32_t *__restrict__ col, const float *__restrict__ val,
                                             const float *__restrict__ B, float *__restrict__ C,
                                             bool accumulate) {
  after_previous_kernel();
  const int PG = 32 / G;
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const bool active = lane < PG * G;
  const int cq = lane % G, pg = active ? lane / G : 0;
  const int start = row_ptr[row], end = row_ptr[row + 1];
  const float *Bt = B + 4 * cq;
  const uint32_t pitch = (uint32_t)N * 4u;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  auto fma4 = [&](float v, const float4 &b) { add_products(acc, v, b); };
  int cn = start + lane < end ? __ldg(col + start + lane) : 0;
  float vn = start + lane < end ? __ldg(val + start + lane) : 0.0f;
  for (int base = start; base < end; base += 32) {
    const int cl = cn;
    const float vl = vn;
    const int mine = base + 32 + lane;
    cn = mine < end ? __ldg(col + mine) : 0;
    vn = mine < end ? __ldg(val + mine) : 0.0f;
    const int left = end - base < 32 ? end - base : 32;
    int j = 0;  // warp-uniform
    for (; j + 4 * PG <= left; j += 4 * PG) {
      const int k = j + pg;
      const int c0 = __shfl_sync(FULL, cl, k), c1 = __shfl_sync(FULL, cl, k + PG);
      const int c2 = __shfl_sync(FULL, cl, k + 2 * PG), c3 = __shfl_sync(FULL, cl, k + 3 * PG);
      const float v0 = __shfl_sync(FULL, vl, k), v1 = __shfl_sync(FULL, vl, k + PG);
      const float v2 = __shfl_sync(FULL, vl, k + 2 * PG), v3 = __shfl_sync(FULL, vl, k + 3 * PG);
      if (active) {
        const float4 b0 = __ldg(row_of(Bt, c0, pitch));
        const float4 b1 = __ldg(row_of(Bt, c1, pitch));
        const float4 b2 = __ldg(row_of(Bt, c2, pitch));
        const float4 b3 = __ldg(row_of(Bt, c3, pitch));
        fma4(v0, b0); fma4(v1, b1); fma4(v2, b2); fma4(v3, b3);
      }
    }
    for (; j < left; j += PG) {
      const int kk = j + pg;
      const int c0 = __shfl_sync(FULL, cl, kk & 31);
      const float v0 = __shfl_sync(FULL, vl, kk & 31);
      if (active && kk < left) fma4(v0, __ldg(row_of(Bt, c0, pitch)));
    }
  }
  for (int g = 1; g < PG; ++g) {  // group g's sums into group 0, in group order
    const int src = (lane + g * G) & 31;
    const float tx = __shfl_sync(FULL, acc.x, src), ty = __shfl_sync(FULL, acc.y, src);
    const float tz = __shfl_sync(FULL, acc.z, src), tw = __shfl_sync(FULL, acc.w, src);
    if (lane < G) { acc.x = add(acc.x, tx); acc.y = add(acc.y, ty); acc.z = add(acc.z, tz); acc.w = add(acc.w, tw); }
  }
  if (lane < G) {
    float4 *out = reinterpret_cast<float4 *>(C + row * N) + cq;
    if (accumulate) {
      const float4 old = *out;
      acc.x = add(old.x, acc.x); acc.y = add(old.y, acc.y); acc.z = add(old.z, acc.z); acc.w = add(old.w, acc.w);
    }
    *out = acc;
  }
}

// Rows of B of 128 * R floats (R = 2, 3, 4): the same fusion with the whole warp on one position; a lane
// holds R float4 of the row of C (columns 4 * lane + 128 * r) and reads the position's row of B as R
// coalesced 512-byte runs.  Two positions are in flight for R = 2, one for wider rows (as many bytes per
// lane as in the kernel above).
template <int R>
__global__ void spmm_wave_per_row_wide_kernel(int64_t rows, int64_t N, const int32_t *__restrict__ row_ptr,
                                              const int32_t *__restrict__ col, const float *__restrict__ val,
                                              const float *__restrict__ B, float *__restrict__ C,
                                              bool accumulate) {
  after_previous_kernel();
  constexpr int U = R == 2 ? 2 : 1;  // positions in flight
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int start = row_ptr[row], end = row_ptr[row + 1];
  const float *Bt = B + 4 * lane;
  const uint32_t pitch = (uint32_t)N * 4u;
  float4 acc[R];
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
  auto fma4 = [&](float4 &a, float v, const float4 &b) { add_products(a, v, b); };
  int cn = start + lane < end ? __ldg(col + start + lane) : 0;
  float vn = start + lane < end ? __ldg(val + start + lane) : 0.0f;
  for (int base = start; base < end; base += 32) {
    const int cl = cn;
    const float vl = vn;
    const int mine = base + 32 + lane;
    cn = mine < end ? __ldg(col + mine) : 0;
    vn = mine < end ? __ldg(val + mine) : 0.0f;
    const int left = end - base < 32 ? end - base : 32;
    int j = 0;
    for (; j + U <= left; j += U) {
      float4 b[U][R];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float4 *brow = row_of(Bt, __shfl_sync(FULL, cl, j + u), pitch);
#pragma unroll
        for (int r = 0; r < R; ++r) b[u][r] = __ldg(brow + 32 * r);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float v = __shfl_sync(FULL, vl, j + u);
#pragma unroll
        for (int r = 0; r < R; ++r) fma4(acc[r], v, b[u][r]);
      }
    }
    if (U > 1 && j < left) {  // U == 2: one position left over
      const float4 *brow = row_of(Bt, __shfl_sync(FULL, cl, j), pitch);
      const float v = __shfl_sync(FULL, vl, j);
#pragma unroll
      for (int r = 0; r < R; ++r) fma4(acc[r], v, __ldg(brow + 32 * r));
    }
  }
  float4 *out = reinterpret_cast<float4 *>(C + row * N) + lane;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float4 a = acc[r];
    if (accumulate) {
      const float4 old = out[32 * r];
      a.x = add(old.x, a.x); a.y = add(old.y, a.y); a.z = add(old.z, a.z); a.w = add(old.w, a.w);
    }
    out[32 * r] = a;
  }
}

// Short matrix rows with rows of B of up to 32 floats: a full warp per row leaves most lanes with one
// position or none and the kernel waits on three dependent loads per warp.  Here L = 4, 8 or 16 lanes
// serve one matrix row (32/L rows per warp): G = N/4 adjacent lanes cover the row of B with one float4
// each, the L/G lane groups stride the row's positions with four positions in flight, butterfly steps
// over the lane distances G ... L/2 add the groups' partial sums, group 0 stores the row of C.
template <int G, int L>
__global__ void spmm_subwarp_row_kernel(int64_t rows, int64_t N, const int32_t *__restrict__ row_ptr,
                                        const int32_t *__restrict__ col, const float *__restrict__ val,
                                        const float *__restrict__ B, float *__restrict__ C, bool accumulate) {
  after_previous_kernel();
  constexpr int PG = L / G, RW = 32 / L;
  static_assert(L >= G && L < 32 && PG >= 1, "lanes per row");
  const int lane = threadIdx.x & 31;
  const int64_t warp = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (warp * RW >= rows) return;  // whole warp out of range
  const int l = lane % L, cq = l % G, pg = l / G;
  const int64_t row = warp * RW + lane / L;
  const bool live = row < rows;  // lanes past the last row still take part in the shuffles
  const int start = live ? row_ptr[row] : 0, end = live ? row_ptr[row + 1] : 0;
  const float *Bt = B + 4 * cq;
  auto b_row = [&](int c) {  // the 64-bit form schedules better for narrow rows of B (300,000 rows of 20, N = 8: 63 us against 66)
    if constexpr (G > 2) return row_of(Bt, c, (uint32_t)N * 4u);
    else return reinterpret_cast<const float4 *>(Bt + (int64_t)c * N);
  };
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  auto fma4 = [&](float v, const float4 &b) { add_products(acc, v, b); };
  int p = start + pg;
  for (; p + 3 * PG < end; p += 4 * PG) {
    const int c0 = __ldg(col + p), c1 = __ldg(col + p + PG), c2 = __ldg(col + p + 2 * PG), c3 = __ldg(col + p + 3 * PG);
    const float v0 = __ldg(val + p), v1 = __ldg(val + p + PG), v2 = __ldg(val + p + 2 * PG), v3 = __ldg(val + p + 3 * PG);
    const float4 b0 = __ldg(b_row(c0));
    const float4 b1 = __ldg(b_row(c1));
    const float4 b2 = __ldg(b_row(c2));
    const float4 b3 = __ldg(b_row(c3));
    fma4(v0, b0); fma4(v1, b1); fma4(v2, b2); fma4(v3, b3);
  }
  for (; p < end; p += PG) {
    const int c0 = __ldg(col + p);
    const float v0 = __ldg(val + p);
    fma4(v0, __ldg(b_row(c0)));
  }
#pragma unroll
  for (int off = G; off < L; off <<= 1) {
    acc.x = add(acc.x, __shfl_xor_sync(FULL, acc.x, off));
    acc.y = add(acc.y, __shfl_xor_sync(FULL, acc.y, off));
    acc.z = add(acc.z, __shfl_xor_sync(FULL, acc.z, off));
    acc.w = add(acc.w, __shfl_xor_sync(FULL, acc.w, off));
  }
  if (live && pg == 0) {
    float4 *out = reinterpret_cast<float4 *>(C + row * N) + cq;
    if (accumulate) {
      const float4 old = *out;
      acc.x = add(old.x, acc.x); acc.y = add(old.y, acc.y); acc.z = add(old.z, acc.z); acc.w = add(old.w, acc.w);
    }
    *out = acc;
  }
}

// ---------------------------------------------------------------------------
// thread-per-position (DecomposePositionSpMMPattern,
// PositionSpMMDecomposition.cpp:19-73, scheduled with the thread/atomic
// schedule, Pipelines.cpp:262-271).  The iteration space is [0, nnz*N):
// position = i / N, column = i % N, key = row*N + column; worker w owns
// iterations [w*chunk, min(nnz*N, (w+1)*chunk)) and issues one atomicAdd per
// iteration.
// ---------------------------------------------------------------------------
__global__ void spmm_thread_per_position_kernel(int64_t rows, int64_t nnz, int64_t N, int64_t chunk,
                                                const int32_t *__restrict__ row_ptr,
                                                const int32_t *__restrict__ col,
                                                const float *__restrict__ val,
                                                const float *__restrict__ B, float *__restrict__ C) {
  after_previous_kernel();
  const int64_t worker = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t begin, end;
  chunk_bounds(0, nnz * N, worker, chunk, begin, end);
  if (begin >= end) return;
  int64_t p = begin / N, j = begin % N;
  int64_t row = row_at_position(row_ptr, rows + 1, p);
  int64_t next = row_ptr[row + 1];
  int c = __ldg(col + p);
  float v = __ldg(val + p);
  for (int64_t i = begin; i < end; ++i) {
    atomicAdd(C + row * N + j, mul(v, __ldg(B + (int64_t)c * N + j)));
    if (++j == N) {
      j = 0;
      ++p;
      if (i + 1 < end) {
        while (next <= p) {
          ++row;
          next = row_ptr[row + 1];
        }
        c = __ldg(col + p);
        v = __ldg(val + p);
      }
    }
  }
}

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// CUDA grids hold at most 2^31 - 1 blocks in x; a launch that needs more is refused instead of truncated.
#define SWB_GRID(name, blocks)                                      \
  unsigned name = 0;                                                 \
  if (!grid_dim(blocks, &name)) return cudaErrorInvalidConfiguration

template <int TCAP>
cudaError_t launch_tile(const CsrSpmmArgs &a, int block, int T, cudaStream_t s) {
  const int64_t tiles = ceil_div(a.n_rhs, T);
  const int64_t units = a.rows * tiles;
  SWB_GRID(grid, ceil_div(units, block / 32));
  const bool vec = (T == TCAP) && (TCAP % 4 == 0) && (a.n_rhs % 4 == 0) && (a.n_rhs % T == 0) &&
                   aligned16(a.B) && aligned16(a.C);
  if (vec) {
    if constexpr (TCAP >= 4)
      launch_chained(spmm_wave_per_row_tile_vec_kernel<TCAP / 4>, grid, block, 0, s, a.rows, a.n_rhs, tiles, a.row_ptr,
                                                                          a.col_idx, a.val, a.B, a.C, a.accumulate);
  } else {
    launch_chained(spmm_wave_per_row_tile_kernel<TCAP>, grid, block, 0, s,
        a.rows, a.n_rhs, T, tiles, a.row_ptr, a.col_idx, a.val, a.B, a.C, a.accumulate);
  }
  return cudaGetLastError();
}

// Lanes per matrix row for rows of B of 4*G floats: at least 4 lanes (and at least G), at most the warp,
// doubled while a lane group would get more than positions_per_lane_group(G) of the mean row's positions.
// The figures are measured (1 M and 2 M rows, uniform columns, 2 to 64 positions per row): few lanes per row
// mean more rows in flight per warp and fewer butterfly steps, and win until the per-group chain of
// positions gets long.  Against four positions per group for every width: N = 8, 24 per row 0.226 -> 0.125 ms;
// N = 16, 24 per row 0.492 -> 0.205 ms; N = 32, 10 per row 0.514 -> 0.246 ms; N = 64, 5 per row (half a warp
// instead of a warp) 1.02 -> 0.53 ms.
constexpr int64_t positions_per_lane_group(int G) { return G == 1 ? 6 : G == 2 ? 12 : G <= 8 ? 16 : 12; }

// ... and doubled for few rows, which leave the GPU idle, so that the time is that of the longest row: up to 200,000 lanes (42
// warps per SM) where a row's lanes have less than a mean row in flight (four positions per group), up to 100,000 where less
// than two.  Ragged rows (times in a CUDA graph): 3,476 of 16, N = 32 16.8 -> 4.3 us; 10,651 of 16, N = 16 17.4 -> 7.9; 4,963 of 39, N = 8
// 12.5 -> 5.8; equal rows 0.8 to 1.1.  More lanes lose on short rows (12,068 of 7, N = 16 with 380,000: 5.0 -> 7.4), and on equal
// rows below eight positions (6,090 of 6, N = 64 2.7 -> 3.7, ragged 7.3 -> 4.2) or above 15,000 rows (18,489 of 15, N = 16 4.1 -> 5.2,
// ragged 17.1 -> 11.7), which therefore keep theirs.
inline int lanes_per_row(int64_t rows, int64_t mean, int G) {
  int lanes = G > 4 ? G : 4;
  while (lanes < 32 && (int64_t)(lanes / G) * positions_per_lane_group(G) < mean) lanes *= 2;
  while (lanes < 32 && ((lanes / G * 4 < mean && mean >= 8 && rows <= 15000 && rows * lanes <= 100000) ||
                        (lanes / G * 4 < 2 * mean && rows * lanes <= 50000)))
    lanes *= 2;
  return lanes;
}

// ---- launches of the staged-rows kernel -------------------------------------------------------

// Lanes per row and rows per block for M runs of columns, R of them per lane.
struct RowsShape {
  int64_t tiles, per;
  int G;
};

// A block takes about 640 positions, which fit its shared memory with room for uneven rows, but no more rows than leave
// 8 blocks for every SM (one wave of them), and at least one row for every group of lanes.
inline RowsShape rows_shape(int64_t rows, int64_t nnz, int64_t M, int R) {
  RowsShape h;
  h.tiles = ceil_div(M, 32 * R);
  h.G = (int)(M < 32 ? M : ceil_div(ceil_div(M, h.tiles), R));
  const int64_t mean = rows > 0 ? nnz / rows : 0, in_hand = 32 / h.G * (STAGE_THREADS / 32);
  const int64_t spread = ceil_div(rows * h.tiles, 148 * 8);
  h.per = 640 / (mean > 0 ? mean : 1);
  if (h.per > spread) h.per = spread;
  if (h.per < in_hand) h.per = in_hand;
  if (h.per > STAGE_ROWS) h.per = STAGE_ROWS;
  return h;
}

// Positions of a row that its group of lanes takes; the block takes the rest.  Above what a block holds in all (some 640
// positions), so that ordinary blocks need not look for such rows, and above the length of ordinary rows.
inline int long_row_of(int64_t rows, int64_t nnz) {
  const int64_t mean = rows > 0 ? nnz / rows : 0;
  return mean <= 128 ? 1024 : mean < 0x0fffffff ? (int)(8 * mean) : 0x7fffffff;
}

// `per` > 0: rows per block, instead of the rule above.
template <int V, int R, int Q, typename Pitch = uint32_t>
cudaError_t launch_rows_as(const CsrSpmmArgs &a, cudaStream_t s, int64_t per = 0) {
  RowsShape h = rows_shape(a.rows, a.nnz, a.n_rhs / V, R);
  if (per > 0) h.per = per;
  SWB_GRID(grid, ceil_div(a.rows, h.per) * h.tiles);
  launch_chained(spmm_staged_rows_kernel<V, R, Q, Pitch>, grid, STAGE_THREADS, 0, s,
      a.rows, a.n_rhs, (Pitch)(a.n_rhs * 4), h.G, (int)h.per, h.tiles, long_row_of(a.rows, a.nnz),
      a.row_ptr, a.col_idx, a.val, a.B, a.C, a.accumulate);
  return cudaGetLastError();
}

// Runs of columns per lane for M runs of V columns: the fewest lane slots (column tiles x runs), the larger number of runs
// where two take as many; and from 33 runs so that two rows fit a warp.  150,000 ragged rows of 15 (us with 2 / 3 / 4 / 5
// runs): N = 35 84 / 69 / 66 / 75, N = 63 87 / 107 / 80 / 100, N = 75 - / 108 / 117 / 101, N = 147 - / 222 / 256 / 177,
// N = 187 - / 248 / 277 / 321; N = 66 (V = 2) 100 / 92 / 93; N = 132 (V = 4) 177 / 154.
inline int runs_per_lane(int64_t M, int V) {
  if (M <= 32) return 1;
  if (M <= 48) return 3;
  if (V == 1 && M <= 80) return M <= 64 ? 4 : 5;
  int best = V == 1 ? 5 : V == 2 ? 4 : 3;  // more runs than this spill registers
  for (int R = best - 1; R >= (V == 1 ? 3 : 2); --R)
    if (ceil_div(M, 32 * R) * R < ceil_div(M, 32 * best) * best) best = R;
  return best;
}

template <int V>
cudaError_t launch_rows_columns(const CsrSpmmArgs &a, cudaStream_t s) {
  const int R = runs_per_lane(a.n_rhs / V, V);
  // Twelve positions a step take most short rows at once (285,639 rows of 10, N = 9: 41 us with eight, 36 with twelve; 100,000
  // ragged rows of 6, N = 13: 18.0 and 16.3); from 16 they only add masked ones.
  if constexpr (V == 1) if (R == 1 && a.nnz <= 12 * a.rows) return launch_rows_as<V, 1, 12>(a, s);
  if (R == 1) return launch_rows_as<V, 1, V <= 2 ? 8 : 4>(a, s);
  if (R == 3) return launch_rows_as<V, 3, 4>(a, s);
  if constexpr (V > 1) if (R == 2) return launch_rows_as<V, 2, 4>(a, s);
  if constexpr (V < 4) if (R == 4) return launch_rows_as<V, 4, 4>(a, s);
  if constexpr (V == 1) if (R == 5) return launch_rows_as<V, 5, 4>(a, s);
  return cudaErrorInvalidValue;
}

// Up to four columns, and up to eight on few rows, the sums run over products staged by the whole block (row_products.cuh):
// 300,000 ragged rows of 20, N = 4: 55 us against 77 here; 3,000 rows of 40, N = 8: 12.6 against 16.7.
inline bool takes_row_products(int64_t rows, int64_t n_rhs) { return n_rhs <= 4 || (n_rhs <= 8 && rows <= 8192); }

// Columns per lane: the widest run that divides N and that the rows of B and C are aligned to, for the fewest
// instructions per position.  With few rows lanes would idle, and what counts is how many rows of B a row of A has in
// flight: narrower runs then, and column tiles rather than several runs per lane.  Measured (us with 1 / 2 / 4 columns):
// 3,000 rows of 40: N = 64 18.5 / 22 / 29, N = 256 29 / 26 / 31; 18,772 rows of 21: N = 16 16.5 / 16.6 / 22,
// N = 32 18.7 / 19.9 / 21.6, N = 64 27 / 22 / 25, N = 128 41 / 33 / 30; 60,000 rows of 10: N = 8 9.1 / 8.9 / 5.9,
// N = 32 20 / 16 / 13.
// A narrow C has many rows in hand per block; narrower runs keep their positions within the staged ones.
inline int columns_per_lane(int64_t rows, int64_t nnz, int64_t n_rhs, uintptr_t alignment_bits) {
  int V = n_rhs % 4 == 0 && alignment_bits % 16 == 0 ? 4 : n_rhs % 2 == 0 && alignment_bits % 8 == 0 ? 2 : 1;
  const int most = rows <= 8192 ? (n_rhs <= 128 ? 1 : 2) : rows <= 32768 ? (n_rhs <= 32 ? 1 : n_rhs <= 64 ? 2 : 4) : 4;
  if (V > most) V = most;
  while (V > 1 && n_rhs / V < 32 && 32 / (n_rhs / V) * (STAGE_THREADS / 32) * (nnz / (rows > 0 ? rows : 1)) > 1300) V /= 2;
  return V;
}
// ... and whether each lane keeps to one run, with more positions a step.
inline bool few_rows(int64_t rows, int64_t n_rhs) { return rows <= 8192 || (rows <= 32768 && n_rhs <= 32); }

// Whether thread-per-output takes a thread per output: where that wins on rows of equal length, which have no longest row to
// wait for, by more than it loses on ragged ones.  Measured (time against the kernels below, equal / ragged rows): N = 2
// 0.83 to 0.92 / 0.97 to 1.12, N = 3 0.72 to 0.91 / 0.89 to 1.07 with up to 12 positions a row (1 M equal rows of 12: 82 -> 59
// us), from 16 on 1.0 to 1.2; up to 4 positions a row: 2,048 to 8,000 rows, N = 33 to 128 0.45 to 0.77 / 0.66 to 1.08 (N = 200
// 1.0 / 1.1), 9,000 to 32,000 rows, N = 5 to 32 0.49 to 0.95 / 0.74 to 1.27, up to 600,000 rows, N = 5, 7, 9, whose rows are
// read by single columns, 0.61 to 0.81 / 0.90 to 1.20.  What is left to the kernels below can still be slower than a thread per
// output on equal rows (N = 5 to 10 with 6 to 24 positions by up to 1.5), by less than ragged rows of the same size gain.
inline bool takes_outputs(int64_t rows, int64_t nnz, int64_t n_rhs) {
  if (n_rhs == 2 || n_rhs == 3) return rows >= 262144 && nnz < 13 * rows;
  if (nnz >= 5 * rows) return false;
  if (rows <= 8192) return n_rhs > 32 && n_rhs <= 128;
  if (rows <= 32768) return n_rhs >= 5 && n_rhs <= 32;
  return rows <= 700000 && (n_rhs == 5 || n_rhs == 7 || n_rhs == 9);
}

cudaError_t launch_rows(const CsrSpmmArgs &a, cudaStream_t s) {
  if (takes_row_products(a.rows, a.n_rhs)) return launch_row_products(a, s);
  if (a.n_rhs > 0x3fffffffLL) return launch_rows_as<1, 5, 4, uint64_t>(a, s);
  const int V = columns_per_lane(a.rows, a.nnz, a.n_rhs, reinterpret_cast<uintptr_t>(a.B) | reinterpret_cast<uintptr_t>(a.C));
  if (few_rows(a.rows, a.n_rhs)) return V == 2 ? launch_rows_as<2, 1, 8>(a, s) : launch_rows_as<1, 1, 16>(a, s);
  if (V == 4) return launch_rows_columns<4>(a, s);
  return V == 2 ? launch_rows_columns<2>(a, s) : launch_rows_columns<1>(a, s);
}

int64_t rows_physical_grid(int64_t rows, int64_t nnz, int64_t n_rhs) {  // 16-byte aligned operands
  if (takes_row_products(rows, n_rhs)) return row_products_physical_grid(rows, nnz, n_rhs);
  const bool wide = n_rhs > 0x3fffffffLL;
  const int V = wide ? 1 : columns_per_lane(rows, nnz, n_rhs, 0);
  const RowsShape h = rows_shape(rows, nnz, n_rhs / V, !wide && few_rows(rows, n_rhs) ? 1 : runs_per_lane(n_rhs / V, V));
  return max1(ceil_div(rows, h.per) * h.tiles);
}

// Whether wave-per-row-tile takes the staged-rows kernel.  It wins where there are rows enough to balance the blocks.  A
// row many times longer than usual is one block's work there (200,000 power-law rows of up to 63,402, N = 32 / 50 / 64 / 128:
// 1.46 / 2.39 / 2.21 / 3.73 ms, with a warp or part of one per row 3.95 / 2.10 / 2.76 / 6.12).  Measured against those kernels:
//   N = 16, 32, 64, 128 (300,000 ragged rows of 5: 41 -> 29, 69 -> 45, 110 -> 89, 184 -> 141 us), with the sizes and mean
//   lengths up to which each wins; N = 8 and long rows do not gain (154,183 ragged rows of 36, N = 32: 106 us there, 111 here);
//   other multiples of 4 from 12 to 124 (150,000 rows of 20, N = 100: 182 -> 126 us; 15,000 rows of 20, N = 24: a draw);
//   the rest up to 512 columns, which else read B by single columns (250,001 rows of 20, N = 50: 664 -> 128 us;
//   102,040 rows of 20, N = 147: 742 -> 145 us; 15,000 rows of 20, N = 7: 10 us there against 13 here).
inline bool tile_takes_staged_rows(int64_t rows, int64_t nnz, int64_t N) {
  const int64_t outputs = rows * N, mean = rows > 0 ? nnz / rows : 0;
  switch (N) {
    case 1: return true;
    case 2: case 3: return rows > 8192;  // products summed per row: 300,000 rows of 20, N = 1: 113 -> 37 us
    case 4: case 8: case 256: case 384: case 512: return false;
    case 16: return outputs >= 2500000 && mean <= 14;
    case 32: return outputs >= 4000000 && mean <= 32;
    case 64: return outputs >= 6000000 && mean <= 48;
    case 128: return outputs >= 8000000;
  }
  if (N > 512 || rows < 100 * mean) return false;
  if (N % 4 == 0 && N >= 12 && N < 128 && mean >= 8) return outputs >= 512000 && (N >= 32 || mean <= 32);
  return outputs >= 256000;
}

// Rows per block of that kernel for N = 64 and short rows: from blocks of 256 on those of a block of the (row, tile) units, half
// a warp or a warp per row, which is the grid that such a launch is known by.  Against the kernel's own rule (0: some 50 to
// 128 rows) it costs with blocks of 256 up to 39 % on very short rows (1 M ragged rows of 3: 236 us against 170; of 5: 300
// against 227; of 12: 520 against 448) and gains up to 14 % (100,000 equal rows of 10: 24.3 against 28.3); with blocks of 512
// and 1,024 the two are within 10 %.  Blocks of 128 would have 4 or 8 rows and cost up to twice the time (300,000 ragged rows
// of 3: 95 against 52).
inline int64_t tile_rows_per_block(int64_t N, int64_t mean, int block) {
  return N == 64 && mean <= 13 && block >= 256 ? (mean <= 12 ? 2 : 1) * (block / 32) : 0;
}

// Columns per lane, lanes per tile and warps per row of a team, or no warps where the team kernel is not for these sizes: N that
// is no power of two up to 128, not the staged-rows kernel's, and few rows.  The (row, tile) kernel's lanes deal with one column
// of a tile at a time, for all positions at once, which fills tiles well that are about as wide as N.  It keeps
//   tiles of 8 and up to 40 columns, of 16 and 17 to 48 (3,076 ragged rows of 9, N = 35 5.8 us, 10.7 here; 2,451 of 12,
//   N = 39 5.3, 6.4), and up to 8 columns in narrower tiles (3,706 ragged rows of 17, N = 5 in tiles of 4: 3.6, 4.7);
//   odd N with more than 16 a row (8,533 of 35, N = 25 in tiles of 4: 19.4, 25.6), unless rows are long and tiles wide
//   (6,244 ragged rows of 35, N = 29 in tiles of 32: 49.5, 19.6; 1,961 of 31, N = 93 37.2, 17.6);
//   fewer than 1,024 rows, whose columns it spreads over more warps.
// A warp per row (spmm_wave_per_row_any_kernel) keeps short rows and more than 4,736 (5,900 of 27, N = 40: 4.9, 6.5).  A row gets
// a second and then a third and fourth warp while a warp has not three mean rows' positions in flight and all warps are one
// wave, or not one mean row and they are three (4,164 ragged rows of 40, N = 18: 12.9 us with one warp, 10.2 with two; 2,172 of
// 64, N = 19: 44, 27 and with four 15.5).  With four columns per lane, two warps in blocks of 128 threads take the place of four
// that would be more than one wave, where they have half a mean row in flight: equal rows pay for warps that they do not need
// (us without teams, with four warps and with two, equal and ragged rows: 4,736 of 28, N = 40 4.9, 8.3, 5.6 and 15.0, 9.3, 7.5; 3,151 of
// 35, N = 36 4.3, 6.1, 4.8 and 16.8, 8.0, 7.6; 4,600 of 60, N = 28 6.8, 8.3, 6.0 and 18.5, 10.7, 11.1).
struct Team {
  int V, G, S;
  int64_t tiles;
  int threads;
};

inline Team team_of(int64_t rows, int64_t nnz, int64_t N, int tile, uintptr_t alignment_bits) {
  Team t{1, 0, 0, 0, TEAM_THREADS};
  if (rows < 1024 || N > 512) return t;
  const int64_t mean = nnz / rows;
  const int V = N % 4 == 0 && alignment_bits % 16 == 0 ? 4 : N % 2 == 0 && alignment_bits % 8 == 0 ? 2 : 1;
  const bool any = N % 4 == 0 && N >= 12 && N < 128 && mean >= 8;
  if (rows > (any ? 4736 : 8192) || (any && mean < 24)) return t;
  if (V == 1 && mean > 16 && (mean < 30 || tile < (N >= 64 ? 8 : 32))) return t;
  if (N <= 8 && tile < (N <= 4 ? 32 : 16)) return t;
  if (!any && ((tile == 8 && N <= 40) || (tile == 16 && N > 16 && N <= 48))) return t;
  t.V = V;
  const int64_t M = N / t.V;
  t.tiles = ceil_div(M, 32);
  t.G = (int)ceil_div(M, t.tiles);
  const int64_t units = rows * t.tiles, in_flight = 32 / t.G * team_positions(t.V);
  t.S = 1;
  while (t.S < 4 && t.S * in_flight < 3 * mean && units * t.S <= (t.S * in_flight < mean ? 13000 : 4750)) t.S *= 2;
  if (V == 4 && t.S == 4 && 4 * units > 148 * 64 && 4 * in_flight >= mean) {
    t.S = 2;
    t.threads = TEAM_THREADS / 2;
  }
  return t;
}

template <int V>
cudaError_t launch_team_rows(const CsrSpmmArgs &a, const Team &t, cudaStream_t s) {
  const int64_t units = a.rows * t.tiles;
  SWB_GRID(grid, ceil_div(units, t.threads / 32 / t.S));
  // Rows that a whole block takes: those of more than 32 steps of a team, and of more than 12 times the mean, which ragged rows do
  // not reach (1,988 ragged rows of 61, N = 136, where 32 steps are 512 positions: 18.5 us, 30.4 without the second limit).
  const int64_t steps = 32 * team_positions(V) * t.S * (32 / t.G), ragged = 12 * (a.nnz / a.rows);
  const int longest = (int)(steps > ragged ? steps : ragged < INT32_MAX ? ragged : INT32_MAX);
  launch_chained(spmm_team_rows_kernel<V>, grid, t.threads, 0, s, a.rows, a.n_rhs, (uint32_t)(a.n_rhs * 4), t.G, t.S, t.tiles,
                 longest, a.row_ptr, a.col_idx, a.val, a.B, a.C, a.accumulate);
  return cudaGetLastError();
}

template <int G, int L>
cudaError_t launch_subwarp(const CsrSpmmArgs &a, int block, cudaStream_t s) {
  const int64_t warps = ceil_div(a.rows, 32 / L);
  SWB_GRID(grid, ceil_div(warps, block / 32));
  launch_chained(spmm_subwarp_row_kernel<G, L>, grid, block, 0, s,
      a.rows, a.n_rhs, a.row_ptr, a.col_idx, a.val, a.B, a.C, a.accumulate);
  return cudaGetLastError();
}

template <int G>
cudaError_t launch_row_of_tiles(const CsrSpmmArgs &a, int block, cudaStream_t s) {
  const int64_t mean = a.rows > 0 ? a.nnz / a.rows : 0;
  const int lanes = lanes_per_row(a.rows, mean, G);
  if constexpr (G <= 4) if (lanes == 4) return launch_subwarp<G, 4>(a, block, s);
  if constexpr (G <= 8) if (lanes == 8) return launch_subwarp<G, 8>(a, block, s);
  if (lanes == 16) return launch_subwarp<G, 16>(a, block, s);
  if constexpr (G >= 4) {  // a warp per row, col/val handed to the lane groups by shuffles
    SWB_GRID(grid, ceil_div(a.rows, block / 32));
    launch_chained(spmm_wave_per_row_fused_kernel<G>, grid, block, 0, s, a.rows, a.n_rhs, a.row_ptr, a.col_idx, a.val, a.B, a.C,
                                                             a.accumulate);
    return cudaGetLastError();
  } else {
    return launch_tile<4 * G>(a, block, 4 * G, s);
  }
}

}  // namespace

cudaError_t launch_spmm_thread_per_output(const CsrSpmmArgs &a, cudaStream_t s, int64_t *launches) {
  ++*launches;
  if (takes_outputs(a.rows, a.nnz, a.n_rhs)) {
    SWB_GRID(grid, ceil_div(a.rows * a.n_rhs, 256));
    launch_chained(spmm_thread_per_output_kernel, grid, 256, 0, s, a.rows, (uint32_t)a.n_rhs, a.row_ptr, a.col_idx, a.val,
                   a.B, a.C);
    return cudaGetLastError();
  }
  return launch_rows(a, s);
}

cudaError_t launch_spmm_wave_per_row_tile(const CsrSpmmArgs &a, int block, int tile,
                                          cudaStream_t s, int64_t *launches) {
  ++*launches;
  // Rows of B of 4, 8, ... 128 floats on 16-byte aligned operands: all tiles of a matrix row are fused
  // into one pass (the tile size then only names the logical units, SparseWaveToGPU.cpp:1078-1084), by a
  // warp, or by part of a warp where the rows are short.
  const int64_t N = a.n_rhs;
  const bool pow2_row = N >= 4 && N <= 128 && (N & (N - 1)) == 0;
  const bool aligned = aligned16(a.B) && aligned16(a.C);
  if (tile_takes_staged_rows(a.rows, a.nnz, N) && (aligned || N % 4 != 0)) {
    const int64_t per = tile_rows_per_block(N, a.nnz / a.rows, block);
    return per > 0 ? launch_rows_as<4, 1, 4>(a, s, per) : launch_rows(a, s);
  }
  if ((N == 256 || N == 384 || N == 512) && aligned16(a.B) && aligned16(a.C)) {
    SWB_GRID(grid, ceil_div(a.rows, block / 32));
    if (N == 256)
      launch_chained(spmm_wave_per_row_wide_kernel<2>, grid, block, 0, s, a.rows, N, a.row_ptr, a.col_idx, a.val, a.B, a.C, a.accumulate);
    else if (N == 384)
      launch_chained(spmm_wave_per_row_wide_kernel<3>, grid, block, 0, s, a.rows, N, a.row_ptr, a.col_idx, a.val, a.B, a.C, a.accumulate);
    else
      launch_chained(spmm_wave_per_row_wide_kernel<4>, grid, block, 0, s, a.rows, N, a.row_ptr, a.col_idx, a.val, a.B, a.C, a.accumulate);
    return cudaGetLastError();
  }
  const Team team = pow2_row ? Team{1, 0, 0, 0, 0}
                             : team_of(a.rows, a.nnz, N, tile, reinterpret_cast<uintptr_t>(a.B) | reinterpret_cast<uintptr_t>(a.C));
  if (team.S > 0)
    return team.V == 4 ? launch_team_rows<4>(a, team, s) : team.V == 2 ? launch_team_rows<2>(a, team, s) : launch_team_rows<1>(a, team, s);
  // other multiples of 4 up to 124 (rows of B of 12, 20, 24 ... floats) where a matrix row has enough positions
  // for a warp: one warp per row as well
  if (N >= 12 && N < 128 && N % 4 == 0 && !pow2_row && a.rows > 0 && a.nnz / a.rows >= 8 && aligned16(a.B) &&
      aligned16(a.C)) {
    SWB_GRID(grid, ceil_div(a.rows, block / 32));
    launch_chained(spmm_wave_per_row_any_kernel, grid, block, 0, s, a.rows, N, (int)(N / 4), a.row_ptr, a.col_idx, a.val, a.B,
                                                       a.C, a.accumulate);
    return cudaGetLastError();
  }
  if (pow2_row && aligned16(a.B) && aligned16(a.C)) {
    if (N == 4) return launch_row_of_tiles<1>(a, block, s);
    if (N == 8) return launch_row_of_tiles<2>(a, block, s);
    if (N == 16) return launch_row_of_tiles<4>(a, block, s);
    if (N == 32) return launch_row_of_tiles<8>(a, block, s);
    if (N == 64) return launch_row_of_tiles<16>(a, block, s);  // half a warp per row where rows are short
    SWB_GRID(grid, ceil_div(a.rows, block / 32));
    launch_chained(spmm_wave_per_row_fused_kernel<32>, grid, block, 0, s, a.rows, N, a.row_ptr, a.col_idx, a.val, a.B, a.C,
                                                               a.accumulate);
    return cudaGetLastError();
  }
  if (tile <= 1) return launch_tile<1>(a, block, tile, s);
  if (tile <= 2) return launch_tile<2>(a, block, tile, s);
  if (tile <= 4) return launch_tile<4>(a, block, tile, s);
  if (tile <= 8) return launch_tile<8>(a, block, tile, s);
  if (tile <= 16) return launch_tile<16>(a, block, tile, s);
  return launch_tile<32>(a, block, tile, s);
}

int64_t thread_per_output_physical_grid(int64_t rows, int64_t nnz, int64_t n_rhs) {
  return takes_outputs(rows, nnz, n_rhs) ? max1(ceil_div(rows * n_rhs, 256)) : rows_physical_grid(rows, nnz, n_rhs);
}

int64_t wave_per_row_tile_physical_grid(int64_t rows, int64_t nnz, int64_t n_rhs, int block, int tile) {
  // Mirrors launch_spmm_wave_per_row_tile and launch_row_of_tiles for 16-byte aligned operands.
  const int64_t wpb = block / 32;
  if (tile_takes_staged_rows(rows, nnz, n_rhs)) {
    const int64_t per = tile_rows_per_block(n_rhs, nnz / rows, block);
    return per > 0 ? max1(ceil_div(rows, per)) : rows_physical_grid(rows, nnz, n_rhs);
  }
  const bool pow2_row = n_rhs >= 4 && n_rhs <= 128 && (n_rhs & (n_rhs - 1)) == 0;
  if (n_rhs == 256 || n_rhs == 384 || n_rhs == 512) return max1(ceil_div(rows, wpb));
  const Team team = pow2_row ? Team{1, 0, 0, 0, 0} : team_of(rows, nnz, n_rhs, tile, 0);
  if (team.S > 0) return max1(ceil_div(rows * team.tiles, team.threads / 32 / team.S));
  if (n_rhs >= 12 && n_rhs < 128 && n_rhs % 4 == 0 && !pow2_row && rows > 0 && nnz / rows >= 8)
    return max1(ceil_div(rows, wpb));
  if (!pow2_row) return max1(ceil_div(rows * ceil_div(n_rhs, tile), wpb));
  if (n_rhs > 64) return max1(ceil_div(rows, wpb));
  const int64_t G = n_rhs / 4, mean = rows > 0 ? nnz / rows : 0;
  const int lanes = lanes_per_row(rows, mean, (int)G);
  return max1(ceil_div(ceil_div(rows, 32 / lanes), wpb));
}

cudaError_t launch_spmm_thread_per_position(const CsrSpmmArgs &a, int block, int64_t chunk,
                                            cudaStream_t s, int64_t *launches) {
  // Zero fill of the flattened output, then the atomic schedule.
  const int64_t workers = ceil_div(a.nnz * a.n_rhs, chunk);
  SWB_GRID(grid, ceil_div(workers, block));
  if (!a.accumulate) {
    cudaError_t e = launch_fill_zero(a.C, a.rows * a.n_rhs, block, s, launches);
    if (e != cudaSuccess) return e;
  }
  launch_chained(spmm_thread_per_position_kernel, grid, block, 0, s, a.rows, a.nnz, a.n_rhs, chunk, a.row_ptr,
                                                         a.col_idx, a.val, a.B, a.C);
  ++*launches;
  return cudaGetLastError();
}

}  // namespace swb
