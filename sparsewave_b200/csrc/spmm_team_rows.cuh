// SpMM by teams of warps, one per row of C (included by spmm_kernels.cu inside namespace swb::{anonymous}).
//
// For matrices of few rows, where the time is that of the longest row: some six times the mean on ragged rows, and as many
// dependent loads of rows of B as its positions are not in flight at once.  A warp holds as many groups of G lanes as fit, each
// with four or eight positions in flight, and a row may have several warps.  Against one column at a time per lane
// (spmm_wave_per_row_tile_kernel): 3,167 rows of 43, N = 130 35.1 -> 18.3 us; 2,376 of 52, N = 62 15.4 -> 8.6; 7,791 of 13,
// N = 25 12.1 -> 6.6; against a warp per row (spmm_wave_per_row_any_kernel): 3,508 ragged rows of 57, N = 40 26.8 -> 11.3.
// Requesting a step's positions beside the rows of B of the step before gains nothing: the loads' issue is what counts.
#pragma once

constexpr int TEAM_THREADS = 256;  // or half of them
constexpr int LONG_ROW_SHARE = 128;  // rows that each of the first blocks looks through
constexpr int team_positions(int V) { return V == 4 ? 4 : 8; }  // in flight per group

// A position's column and value where k < n, as predicated loads (see spmm_columns.cuh).
__device__ __forceinline__ void position_if(int &c, float &v, const int32_t *col, const float *val, int k, int n) {
  asm("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %4, %5;\n\t@p ld.global.nc.s32 %0, [%2];\n\t@p ld.global.nc.f32 %1, [%3];\n\t}"
      : "=r"(c), "=f"(v) : "l"(col), "l"(val), "r"(k), "r"(n));
}

// A team of S warps holds a row and a tile of G * V columns: groups of G lanes take the row's positions in turn, Q in flight
// each, and the groups' sums are added up in shared memory.  Rows of more than `longest` positions are left to whole blocks: each
// of the first blocks looks through its share of the rows before it begins its own, and takes those among them behind its own.
// Without that a row of half of 5,000 columns among rows of 12 ran on in one team (N = 50: 97 us, now 34; 31 by
// spmm_wave_per_row_tile_kernel); rows without any cost 0.84 to 1.08 times the time, 1.00 over 120 sizes.  Tried: the look
// behind the block's own rows (1.09), its own offsets loaded before it (1.06: the loop over positions compiles to slower code).
template <int V>
__global__ void __launch_bounds__(TEAM_THREADS)
    spmm_team_rows_kernel(int64_t rows, int64_t N, uint32_t pitch, int G, int S, int64_t tiles, int longest,
                          const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ col, const float *__restrict__ val,
                          const float *__restrict__ B, float *__restrict__ C, bool accumulate) {
  after_previous_kernel();
  constexpr int Q = team_positions(V);
  __shared__ __align__(16) float s_sums[TEAM_THREADS * V];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, team = warp / S;
  const int64_t unit = (int64_t)blockIdx.x * (int)(blockDim.x / 32 / S) + team;
  const int per_warp = 32 / G, group = lane / G, l = lane - group * G;
  int64_t row = tiles == 1 ? unit : unit / tiles, tile = tiles == 1 ? 0 : unit - row * tiles;
  int warps = S, member = warp - team * S;
  bool whole = false;  // the block has rows of its share to take together
  const int64_t share = (int64_t)blockIdx.x * LONG_ROW_SHARE;
  if (share < rows) {
    bool found = false;
#pragma unroll
    for (int i = 0; i < LONG_ROW_SHARE; i += 32) {
      const int64_t r = share + i + lane;
      if (r < rows) found |= __ldg(row_ptr + r + 1) - __ldg(row_ptr + r) > longest;
    }
    whole = __any_sync(0xffffffffu, found);
  }
  for (int64_t at = share - 1;;) {
    const int groups = warps * per_warp, mine = member * per_warp + group;
    const int64_t first_col = tile * (G * V);
    bool works = row < rows;
    int64_t c0 = first_col + l * V;
    if (c0 >= N) c0 = N - V;  // a lane past the last column repeats it; its sums are not used
    Columns<V> acc;
#pragma unroll
    for (int j = 0; j < V; ++j) acc.f[j] = 0.0f;
    if (works) {
      const int start = __ldg(row_ptr + row), n = __ldg(row_ptr + row + 1) - start;
      works = n <= longest || at >= share;
      const char *Bt = reinterpret_cast<const char *>(B + c0);
      int c[Q];
      float v[Q];
      auto positions = [&](int left) {  // the step's that begins `left` positions before the row's end
        const int p = start + (n - left);
#pragma unroll
        for (int k = 0; k < Q; ++k) {
          position_if(c[k], v[k], col + p + k * groups, val + p + k * groups, k * groups, left);
        }
      };
      for (int left = works && group < per_warp ? n - mine : 0; left > 0; left -= Q * groups) {
        Columns<V> b[Q];
        float w[Q];
        positions(left);
#pragma unroll
        for (int k = 0; k < Q; ++k) {
          load_if<V>(b[k], Bt + (uint32_t)c[k] * (uint64_t)pitch, k * groups, left);
          w[k] = v[k];
        }
#pragma unroll
        for (int k = 0; k < Q; ++k) add_if<V>(acc, w[k], b[k], k * groups, left);
      }
    }
    const int width = N - first_col < (int64_t)G * V ? (int)(N - first_col) : G * V;
    float *sums = s_sums + (warp - member) * 32 * V;
    if (group < per_warp) store_columns<V>(sums + mine * G * V + l * V, acc);
    if (warps == 1) __syncwarp(); else __syncthreads();
    if (works) {
      float *out = C + row * N + first_col;
      for (int j = member * 32 + lane; j < width; j += warps * 32) {
        float t = sums[j];
        for (int g = 1; g < groups; ++g) t = add(t, sums[g * G * V + j]);
        out[j] = accumulate ? add(out[j], t) : t;
      }
    }
    if (!whole) return;
    __syncthreads();
    // the next of the block's long rows, or of its tiles
    if (at < share || ++tile == tiles) {
      tile = 0;
      const int64_t end = share + LONG_ROW_SHARE < rows ? share + LONG_ROW_SHARE : rows;
      do
        if (++at >= end) return;
      while (__ldg(row_ptr + at + 1) - __ldg(row_ptr + at) <= longest);
      row = at;
      warps = blockDim.x / 32;
      member = warp;
    }
  }
}
