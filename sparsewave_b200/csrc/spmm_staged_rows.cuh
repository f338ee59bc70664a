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
//
// A row of thousands of positions would be one group's chain, four to sixteen positions a step (190 ns a position with
// N = 64, so that eight rows of 65,536 among a million of 20 took 12.8 ms).  Its group takes `long_min` positions of it, and
// the block, when its groups are through, the rest, still in position order: 3.0 ms.  1 M power-law rows of up to 65,119,
// N = 32 / 50 / 64 / 128: 11.2 / 10.0 / 12.6 / 13.7 -> 2.4 / 3.4 / 3.4 / 5.5 ms.  A block without such a row pays one
// minimum per row and one test (1 to 4 %).
#pragma once

constexpr int STAGE_THREADS = 128, STAGE_POSITIONS = 1536, STAGE_ROWS = 256;
constexpr int LONG_ROW_WORDS = 2 * STAGE_POSITIONS;  // a tile of a long row, in the memory of the positions

// Blocks per SM: as many as the rows of B in flight and the sums leave registers for.  One block too many spills inside the
// loop and costs a factor of two (40,000 rows of 20, N = 187, seven columns per lane in 64 registers: 242 us; N = 33 with ten
// blocks of three runs: 128 -> 260).
constexpr int stage_min_blocks(int V, int R, int Q) {
  const int words = V * R;
  if (words < 3 || (words == 4 && R == 1)) return Q > 8 ? 8 : 10;
  return words == 3 ? 9 : words == 4 ? 8 : words == 5 ? 7 : words <= 8 ? 6 : 5;
}

// The end of a long row: n positions from `start` on, added to the `width` columns from first_col on that its group has
// stored.  The block takes a tile of positions at a time, copies their rows of B to shared memory with all of them in flight
// (and requests the next tile's positions beside them), and one thread per column adds them up in position order.
template <int V, int R, typename Pitch>
__device__ __forceinline__ void finish_long_row(int2 *positions, float *out, int start, int n, int64_t first_col, int width,
                                                Pitch pitch, const int32_t *__restrict__ col, const float *__restrict__ val,
                                                const float *__restrict__ B) {
  constexpr int SLOTS = (32 * V * R + STAGE_THREADS - 1) / STAGE_THREADS;  // columns per thread
  const int tid = threadIdx.x, M = width / V;
  const int fit = (LONG_ROW_WORDS / (width + 2)) & ~1;  // even: the rows of B behind the positions stay 16-byte aligned
  const int per_tile = fit < STAGE_THREADS ? fit : STAGE_THREADS;
  float *rows_of_b = reinterpret_cast<float *>(positions + per_tile);
  const char *Bt = reinterpret_cast<const char *>(B + first_col);
  float sum[SLOTS];
#pragma unroll
  for (int k = 0; k < SLOTS; ++k) {
    const int o = tid + k * STAGE_THREADS;
    sum[k] = o < width ? out[o] : 0.0f;
  }
  auto position = [&](int k) {  // this thread's of the tile that starts k positions on
    return tid < per_tile && tid < n - k ? make_int2(__ldg(col + start + k + tid), __float_as_int(__ldg(val + start + k + tid)))
                                         : make_int2(0, 0);
  };
  int2 mine = position(0);
  for (int left = n; left > 0; left -= per_tile) {
    const int have = left < per_tile ? left : per_tile;
    if (tid < per_tile) positions[tid] = mine;
    __syncthreads();
#pragma unroll 1
    for (int i = tid; i < have * M; i += STAGE_THREADS) {
      const int q = i / M;
      const char *src = Bt + (Pitch)positions[q].x * (uint64_t)pitch + (i - q * M) * (4 * V);
      const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(rows_of_b + i * V));
      asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(4 * V) : "memory");
    }
    if (left > per_tile) mine = position(n - left + per_tile);  // the next tile's, beside the rows of B
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int k = 0; k < SLOTS; ++k) {
      const int o = tid + k * STAGE_THREADS;
      if (o < width) {
#pragma unroll 4
        for (int q = 0; q < have; ++q)
          sum[k] = add(sum[k], mul(__int_as_float(positions[q].y), rows_of_b[q * width + o]));
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < SLOTS; ++k) {
    const int o = tid + k * STAGE_THREADS;
    if (o < width) out[o] = sum[k];
  }
}

template <int V, int R, int Q, typename Pitch>
__global__ void __launch_bounds__(STAGE_THREADS, stage_min_blocks(V, R, Q))
    spmm_staged_rows_kernel(int64_t rows, int64_t N, Pitch pitch, int G, int rows_per_block, int64_t tiles,
                            int long_min, const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ col,
                            const float *__restrict__ val, const float *__restrict__ B, float *__restrict__ C,
                            bool accumulate) {
  after_previous_kernel();
  constexpr int U = V * R >= 16 ? 1 : V * R >= 8 ? 2 : Q;  // rows of B in flight: at most 16 registers of them, or Q
  __shared__ __align__(16) int2 s_pos[STAGE_POSITIONS + 16];  // (column, value bits)
  __shared__ int s_off[STAGE_ROWS + 1];
  __shared__ int s_next;
  __shared__ bool s_many;  // more positions than a group may take of a row
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // 32-bit: a 64-bit division is a call, for which the groups' loop would spill
  const int64_t unit = tiles == 1 ? blockIdx.x : blockIdx.x / (unsigned)tiles;
  const int64_t r0 = unit * rows_per_block;
  const int count = r0 + rows_per_block < rows ? rows_per_block : (int)(rows - r0);
  const int groups = 32 / G;                     // rows in hand per warp
  for (int i = tid; i <= count; i += STAGE_THREADS) s_off[i] = row_ptr[r0 + i];
  if (tid == 0) {
    s_next = groups * (STAGE_THREADS / 32);
    s_many = row_ptr[r0 + count] - row_ptr[r0] > long_min;
  }
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
  if (row < count) { q = s_off[row] - first; left = min(s_off[row + 1] - first - q, long_min); }
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
        if (row < count) { q = s_off[row] - first; left = min(s_off[row + 1] - first - q, long_min); }
      }
      if (!__any_sync(FULL, row < count)) break;
    } else if (!__any_sync(FULL, left > 0)) {
      break;
    }
  }
  if (!s_many) return;
  // Everything again from the launch's parameters, so that nothing is kept in registers across the groups' loop for this.
  unsigned block;
  int g = G, per_block = rows_per_block;
  asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(block), "+r"(g), "+r"(per_block));
  const unsigned u = block / (unsigned)tiles;
  const int64_t row0 = (int64_t)u * per_block;
  const int rows_here = row0 + per_block < rows ? per_block : (int)(rows - row0);
  bool mine = false;
  for (int i = threadIdx.x; i < rows_here; i += STAGE_THREADS) mine |= s_off[i + 1] - s_off[i] > long_min;
  if (!__syncthreads_or(mine)) return;
  const int64_t col0 = (int64_t)(block - u * (unsigned)tiles) * (g * V * R);
  const int width = N - col0 < (int64_t)g * V * R ? (int)(N - col0) : g * V * R;
#pragma unroll 1
  for (int r = 0; r < rows_here; ++r) {
    const int start = s_off[r] + long_min, n = s_off[r + 1] - s_off[r] - long_min;
    if (n > 0) finish_long_row<V, R>(s_pos, C + (row0 + r) * N + col0, start, n, col0, width, pitch, col, val, B);
  }
}
