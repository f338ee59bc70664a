// SpMM by groups of lanes that take whole rows of C in turn (included by spmm_kernels.cu inside namespace
// swb::{anonymous}).
//
// A block owns a run of rows.  It stages their col and val in shared memory with coalesced loads, so that the chain
// row offset -> column -> row of B is paid once per block and not once per row.  A group of G lanes then holds a row of
// C (R runs of V adjacent columns per lane), 32 / G groups in a warp; a group adds up Q positions a step with up to Q
// rows of B in flight, stores the row when it ends and fetches the block's next one, so uneven rows do not hold up the
// other groups.  Every output is added up by one lane in position order: bit for bit the sequential sum.
//
// What bounds it is issue slots first (hence the predicated loads and sums, and one wide multiply-add per address), then
// the gather of rows of B from L2.  Handing columns out by shuffles instead of shared memory costs two shuffles a
// position (182 us against 97 on 300,000 ragged rows of 20, N = 32); one thread per four outputs with no staging leaves
// a warp waiting for its longest row (146 us).  250,001 ragged rows of 20, N = 50: 128 us (1.0 GB of B rows, 7.8 TB/s
// from L2); 117,187 rows of 20, N = 128: 103 us (11.6 TB/s).  The positions of a block that do not fit the tile (rows far
// above the mean) are read from global memory.
#pragma once

constexpr int STAGE_THREADS = 128, STAGE_POSITIONS = 1536, STAGE_ROWS = 256;

// Blocks per SM: as many as the rows of B in flight and the sums leave registers for.  One block too many spills inside the
// loop and costs a factor of two (40,000 rows of 20, N = 187, seven columns per lane in 64 registers: 242 us).
constexpr int stage_min_blocks(int V, int R, int Q) {
  const int words = V * R;
  return words <= 3 || (words == 4 && R == 1) ? (Q > 8 ? 8 : 10) : words <= 5 ? 8 : words <= 8 ? 6 : 5;
}

template <int V, int R, int Q, typename Pitch>
__global__ void __launch_bounds__(STAGE_THREADS, stage_min_blocks(V, R, Q))
    spmm_staged_rows_kernel(int64_t rows, int64_t N, Pitch pitch, int G, int rows_per_block, int64_t tiles,
                            const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ col,
                            const float *__restrict__ val, const float *__restrict__ B, float *__restrict__ C,
                            bool accumulate) {
  after_previous_kernel();
  constexpr int U = V * R >= 16 ? 1 : V * R >= 8 ? 2 : Q;  // rows of B in flight: at most 16 registers of them, or Q
  __shared__ __align__(16) int2 s_pos[STAGE_POSITIONS + 16];  // (column, value bits)
  __shared__ int s_off[STAGE_ROWS + 1];
  __shared__ int s_next;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t unit = tiles == 1 ? blockIdx.x : blockIdx.x / tiles;
  const int64_t r0 = unit * rows_per_block;
  const int count = r0 + rows_per_block < rows ? rows_per_block : (int)(rows - r0);
  const int groups = 32 / G;                     // rows in hand per warp
  for (int i = tid; i <= count; i += STAGE_THREADS) s_off[i] = row_ptr[r0 + i];
  if (tid == 0) s_next = groups * (STAGE_THREADS / 32);
  __syncthreads();
  const int first = s_off[0], last = s_off[count];
  const bool staged = last - first <= STAGE_POSITIONS;
  if (staged) {
    for (int i = first + tid; i < last; i += STAGE_THREADS)
      s_pos[i - first] = make_int2(__ldg(col + i), __float_as_int(__ldg(val + i)));
    __syncthreads();
  }

  const int l = lane % G, group = lane / G;
  const bool member = group < groups;
  const int leader = member ? group * G : 0;
  const int64_t first_col = (tiles == 1 ? 0 : (blockIdx.x - unit * tiles) * ((int64_t)G * V * R));
  int64_t c0[R];  // first of this lane's columns; a lane past the last column repeats it and stores nothing
#pragma unroll
  for (int r = 0; r < R; ++r) {
    c0[r] = first_col + (int64_t)(r * G + l) * V;
    if (c0[r] >= N) c0[r] = N - V;
  }
  const char *Bt = reinterpret_cast<const char *>(B + c0[0]);
  int run[R];
#pragma unroll
  for (int r = 0; r < R; ++r) run[r] = (int)((c0[r] - c0[0]) * 4);

  Columns<V> acc[R];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int k = 0; k < V; ++k) acc[r].f[k] = 0.0f;
  int row = member ? warp * groups + group : count;
  int q = 0, left = 0;  // next position of the row (from the tile's first), positions left
  if (row < count) { q = s_off[row] - first; left = s_off[row + 1] - first - q; }
  while (true) {
    const bool done = left <= Q;  // the row ends with this step (idle groups: always)
    if (left > 0) {
      int2 cv[Q];
      if (staged) {
#pragma unroll
        for (int k = 0; k < Q; ++k) cv[k] = s_pos[q + k];
      } else {
#pragma unroll
        for (int k = 0; k < Q; ++k)
          cv[k] = k < left ? make_int2(__ldg(col + first + q + k), __float_as_int(__ldg(val + first + q + k))) : make_int2(0, 0);
      }
#pragma unroll
      for (int k0 = 0; k0 < Q; k0 += U) {
        Columns<V> b[U][R];
#pragma unroll
        for (int k = 0; k < U; ++k) {
          const char *src = Bt + (Pitch)cv[k0 + k].x * (uint64_t)pitch;
#pragma unroll
          for (int r = 0; r < R; ++r) load_if<V>(b[k][r], src + run[r], k0 + k, left);
        }
#pragma unroll
        for (int k = 0; k < U; ++k)
#pragma unroll
          for (int r = 0; r < R; ++r) add_if<V>(acc[r], __int_as_float(cv[k0 + k].y), b[k][r], k0 + k, left);
      }
    }
    q += Q;
    left -= Q;
    if (__any_sync(FULL, done && row < count)) {
      int next = 0;
      if (done && row < count && l == 0) next = atomicAdd(&s_next, 1);
      next = __shfl_sync(FULL, next, leader);
      if (done && row < count) {
        float *out = C + (r0 + row) * N;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if (first_col + (int64_t)(r * G + l) * V < N) {
            if (accumulate) {
#pragma unroll
              for (int k = 0; k < V; ++k) acc[r].f[k] = add(out[c0[r] + k], acc[r].f[k]);
            }
            store_columns<V>(out + c0[r], acc[r]);
          }
#pragma unroll
          for (int k = 0; k < V; ++k) acc[r].f[k] = 0.0f;
        }
        row = next;
        left = 0;
        if (row < count) { q = s_off[row] - first; left = s_off[row + 1] - first - q; }
      }
      if (!__any_sync(FULL, row < count)) break;
    } else if (!__any_sync(FULL, left > 0)) {
      break;
    }
  }
}
