// Row mappings of SpMV: a group of lanes per row for short rows, and a stream of rows with x in shared memory (included by
// spmv_kernels.cu inside namespace swb::{anonymous}).
#pragma once

constexpr int ROWS_THREADS = 256;
constexpr int ROWS_LONGEST = 2048;      // positions of a row that a warp takes: what the block takes at a time
constexpr int SHARED_X_FLOATS = 49152;  // 192 KB
constexpr int SHARED_X_THREADS = 1024;  // one block per SM

struct Quad {
  int4 c;
  float4 v;
};

// Quad at position q, a multiple of 4, of a row that ends at e: positions past e may be loaded, past the arrays not.
__device__ __forceinline__ Quad load_quad(const int32_t *__restrict__ col, const float *__restrict__ val, int64_t nnz,
                                          int q, int e) {
  Quad t = {make_int4(0, 0, 0, 0), make_float4(0.f, 0.f, 0.f, 0.f)};
  if (q < e) {
    if ((int64_t)q + 4 <= nnz) {
      t.c = ld_stream(reinterpret_cast<const int4 *>(col + q));
      t.v = ld_stream(reinterpret_cast<const float4 *>(val + q));
    } else {
      t.c.x = ld_stream(col + q); t.v.x = ld_stream(val + q);
      if (q + 1 < e) { t.c.y = ld_stream(col + q + 1); t.v.y = ld_stream(val + q + 1); }
      if (q + 2 < e) { t.c.z = ld_stream(col + q + 2); t.v.z = ld_stream(val + q + 2); }
    }
  }
  return t;
}

__device__ __forceinline__ bool inside(int p, int s, int e) { return (unsigned)(p - s) < (unsigned)(e - s); }  // s <= e

// Columns of a quad as far as they are the row's, which is [s, e).  The others, which may belong to no row at all (spare
// capacity of the arrays, rows of a larger matrix in front of this one's and behind), are not used as an index into x.
__device__ __forceinline__ int4 own_columns(const int4 &c, int q, int s, int e) {
  return make_int4(inside(q, s, e) ? c.x : 0, inside(q + 1, s, e) ? c.y : 0, inside(q + 2, s, e) ? c.z : 0,
                   inside(q + 3, s, e) ? c.w : 0);
}

// Sum of the products of a quad's positions inside [s, e); g: x at its columns.
__device__ __forceinline__ float quad_sum(const float4 &v, const float4 &g, int q, int s, int e) {
  const float p0 = inside(q, s, e) ? mul(v.x, g.x) : 0.0f, p1 = inside(q + 1, s, e) ? mul(v.y, g.y) : 0.0f;
  const float p2 = inside(q + 2, s, e) ? mul(v.z, g.z) : 0.0f, p3 = inside(q + 3, s, e) ? mul(v.w, g.w) : 0.0f;
  return add(add(p0, p1), add(p2, p3));
}

// Rows that the warps of a block have left out, because they are far longer than the others, by the whole block, one at a
// time.  `row_of(i)` is the block's i-th row, in any order, `end(i)` whether there is none from i on.  A sum depends on its
// row alone.
template <int THREADS, typename Gather, typename RowOf, typename End>
__device__ __forceinline__ void sum_rows_left_out(int most, int64_t rows, int64_t nnz, const int32_t *__restrict__ row_ptr,
                                                  const int32_t *__restrict__ col, const float *__restrict__ val,
                                                  float *__restrict__ y, Gather gather, RowOf row_of, End end) {
  __shared__ unsigned found[THREADS / 32];  // of THREADS rows looked at
  __shared__ float sums[THREADS / 32];
  const int tid = threadIdx.x;
  for (int i0 = 0; !end(i0); i0 += THREADS) {
    const int64_t r = row_of(i0 + tid);
    const unsigned mask = __ballot_sync(FULL, r < rows && __ldg(row_ptr + r + 1) - __ldg(row_ptr + r) > most);
    if ((tid & 31) == 0) found[tid >> 5] = mask;
    __syncthreads();
    for (int w = 0; w < THREADS / 32; ++w) {
      for (unsigned todo = found[w]; todo != 0; todo &= todo - 1) {
        const int64_t row = row_of(i0 + 32 * w + __ffs(todo) - 1);
        const int s = __ldg(row_ptr + row), e = __ldg(row_ptr + row + 1);
        float sum = 0.0f;
        int p = (s & ~3) + 4 * tid;
        for (; p + 4 * THREADS < e; p += 8 * THREADS) {
          const Quad t = load_quad(col, val, nnz, p, e), u = load_quad(col, val, nnz, p + 4 * THREADS, e);
          const float4 g = gather(own_columns(t.c, p, s, e)), h = gather(own_columns(u.c, p + 4 * THREADS, s, e));
          sum = add(sum, add(quad_sum(t.v, g, p, s, e), quad_sum(u.v, h, p + 4 * THREADS, s, e)));
        }
        if (p < e) {
          const Quad t = load_quad(col, val, nnz, p, e);
          sum = add(sum, quad_sum(t.v, gather(own_columns(t.c, p, s, e)), p, s, e));
        }
        sum = warp_sum(sum);
        if ((tid & 31) == 0) sums[tid >> 5] = sum;
        __syncthreads();
        if (tid < 32) {
          sum = warp_sum(tid < THREADS / 32 ? sums[tid] : 0.0f);
          if (tid == 0) y[row] = sum;
        }
        __syncthreads();
      }
    }
    __syncthreads();  // `found` is written again
  }
}

// A warp per short row leaves most lanes without a position, a block per row even more, and both pay the chain row offset
// -> col/val -> x -> reduction for every row.  Here L = 4 to 16 lanes take a row in 16-byte quads of four positions, two
// quads per lane (8 L positions) in flight; the grid is eight blocks per SM, of which four run at a time (64 registers), a
// group walks rows a grid apart and requests the next row's quads (and the offsets of the one behind it) before it sums this
// one.  Rows of more than 16 L positions are finished by the whole warp, and rows of more than ROWS_LONGEST are left to the
// block, which takes eight times as many positions at once, in the end: as one warp's, a row of 65,536 is 256 steps (4 M
// power-law rows 775 -> 540 us; 300,000 rows of 10 with eight of 65,536 183 -> 37).  Large matrices are then bound by the gather of x from L2 (253 G/s): 700,000 rows of 40
// 165 -> 112 us, 1 M ragged rows of 16 149 -> 82 us, 400,000 rows of 70 (block-per-row) 220 -> 114 us.
template <int L>
__global__ void __launch_bounds__(ROWS_THREADS)
    spmv_rows_kernel(int64_t rows, int64_t nnz, const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ col,
                     const float *__restrict__ val, const float *__restrict__ x, float *__restrict__ y, bool apart) {
  __shared__ bool left_out;  // some row
  if (threadIdx.x == 0) left_out = false;
  __syncthreads();
  after_previous_kernel();
  const int lane = threadIdx.x & 31, l = lane % L;
  constexpr int WARPS = ROWS_THREADS / 32;
  // `apart`: the warps of a block lie a grid apart, so that neighbouring rows, which are long together where rows are sorted
  // by length, are other blocks' (1 M sorted power-law rows 2260 -> 460 us)
  auto warp_of = [&](int w) { return apart ? (int64_t)w * gridDim.x + blockIdx.x : (int64_t)blockIdx.x * WARPS + w; };
  const int64_t warp = warp_of(threadIdx.x >> 5);
  const int64_t stride = (((int64_t)gridDim.x * blockDim.x) >> 5) * (32 / L);
  auto bounds = [&](int64_t r, int &s, int &e) {  // empty past the last row
    s = r < rows ? __ldg(row_ptr + r) : 0;
    e = r < rows ? __ldg(row_ptr + r + 1) : 0;
  };
  auto load = [&](int q, int e) { return load_quad(col, val, nnz, q, e); };
  auto gather = [&](const int4 &c) { return make_float4(__ldg(x + c.x), __ldg(x + c.y), __ldg(x + c.z), __ldg(x + c.w)); };
  auto sum_of = [&](const Quad &t, int q, int s, int e) {
    return quad_sum(t.v, gather(own_columns(t.c, q, s, e)), q, s, e);
  };
  int s, e, s1, e1;
  int64_t r = warp * (32 / L) + lane / L;
  bounds(r, s, e);
  bounds(r + stride, s1, e1);
  Quad a = load((s & ~3) + 4 * l, e), b = load((s & ~3) + 4 * (l + L), e);
  for (int64_t first = warp * (32 / L); first < rows; first += stride, r += stride) {  // uniform in the warp
    int s2, e2;
    bounds(r + 2 * stride, s2, e2);
    const Quad an = load((s1 & ~3) + 4 * l, e1), bn = load((s1 & ~3) + 4 * (l + L), e1);
    const int q = (s & ~3) + 4 * l;
    if (e - s > ROWS_LONGEST) {  // no position, then: the zero that is stored is overwritten in the end
      left_out = true;
      e = s;
    }
    const bool is_long = e - s > 16 * L;
    float sum = 0.0f;
    if (q < e) sum = sum_of(a, q, s, e);
    if (q + 4 * L < e) sum = add(sum, sum_of(b, q + 4 * L, s, e));
    if (!is_long)
      for (int p = q + 8 * L; p < e; p += 4 * L) sum = add(sum, sum_of(load(p, e), p, s, e));
    for (unsigned todo = __ballot_sync(FULL, is_long && l == 0); todo != 0; todo &= todo - 1) {
      const int owner = __ffs(todo) - 1;  // what lies behind its first 8 L positions, by all lanes
      const int os = __shfl_sync(FULL, s, owner), oe = __shfl_sync(FULL, e, owner);
      float part = 0.0f;
      int p = (os & ~3) + 8 * L + 4 * lane;
      for (; p + 128 < oe; p += 256) {
        const Quad t = load(p, oe), u = load(p + 128, oe);
        part = add(part, add(sum_of(t, p, os, oe), sum_of(u, p + 128, os, oe)));
      }
      if (p < oe) part = add(part, sum_of(load(p, oe), p, os, oe));
      part = warp_sum(part);
      if (lane == owner) sum = add(sum, part);
    }
#pragma unroll
    for (int off = L / 2; off >= 1; off >>= 1) sum = add(sum, __shfl_xor_sync(FULL, sum, off));
    if (l == 0 && r < rows) y[r] = sum;
    s = s1; e = e1; s1 = s2; e1 = e2;
    a = an; b = bn;
  }
  __syncthreads();
  if (!left_out) return;
  constexpr int TURN = ROWS_THREADS / L;  // rows of the block in one turn of its warps
  auto row_of = [&](int i) {
    const int w = i % TURN / (32 / L), k = i % (32 / L);
    return warp_of(w) * (32 / L) + k + i / TURN * stride;
  };
  sum_rows_left_out<ROWS_THREADS>(ROWS_LONGEST, rows, nnz, row_ptr, col, val, y, gather, row_of,
                                  [&](int i) { return i / TURN * stride >= rows; });
}

// Longer rows are bound by the gather of x alone.  L1 serves two of them per clock and SM while x fits it (570 G/s), but
// beyond 192 KB they go to L2, which serves 253 G/s.  From there to a few times that the first 192 KB of x are staged in
// shared memory, once per SM, and only the others are gathered through L1.  One block of 32 warps fits an SM: a warp
// takes rows a grid apart as one stream of steps of 128 positions and requests the quads of the next step before it
// gathers for it, and gathers before it sums this one, across the ends of rows.  (Requesting further ahead takes more
// registers than 1,024 threads have.)  Rows of more than `longest` positions are left to the block (180,000 rows of 150 with
// eight of 65,536: 400 -> 119 us).  65,536 rows of 256: 60 -> 34 us; 100,000 ragged rows of 200: 77 -> 73;
// 150,000: 134 -> 121.
__device__ __forceinline__ float gather_x(const float *__restrict__ x, uint32_t staged, int c) {
  float v;  // one of two predicated loads: a branch would split the warp at every gather
  asm("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %1, %2;\n\t@p ld.shared.f32 %0, [%3];\n\t@!p ld.global.nc.f32 %0, [%4];\n\t}"
      : "=f"(v) : "r"(c), "n"(SHARED_X_FLOATS), "r"(staged + 4u * (uint32_t)c), "l"(x + c));
  return v;
}

__global__ void __launch_bounds__(SHARED_X_THREADS, 1)
    spmv_row_stream_kernel(int64_t rows, int64_t nnz, const int32_t *__restrict__ row_ptr,
                           const int32_t *__restrict__ col, const float *__restrict__ val, const float *__restrict__ x,
                           float *__restrict__ y, int longest) {
  extern __shared__ float4 staged_x[];
  __shared__ bool left_out;  // some row
  if (threadIdx.x == 0) left_out = false;
  __syncthreads();
  after_previous_kernel();
  for (int i = threadIdx.x; i < SHARED_X_FLOATS / 4; i += SHARED_X_THREADS)
    staged_x[i] = __ldg(reinterpret_cast<const float4 *>(x) + i);
  uint32_t staged = static_cast<uint32_t>(__cvta_generic_to_shared(staged_x));
  const int lane = threadIdx.x & 31;
  const int warps = (int)((gridDim.x * blockDim.x) >> 5);
  struct Step { int64_t row; int s, e, q; };  // row, its bounds, first position of the step (a multiple of 4)
  auto bounds = [&](int64_t r, int &s, int &e) {
    s = r < rows ? __ldg(row_ptr + r) : 0;
    e = r < rows ? __ldg(row_ptr + r + 1) : 0;
    if (e - s > longest) {  // no position, as above
      left_out = true;
      e = s;
    }
  };
  Step ahead;
  int ns, ne;  // bounds of the row behind that step's
  ahead.row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  bounds(ahead.row, ahead.s, ahead.e);
  ahead.q = ahead.s & ~3;
  bounds(ahead.row + warps, ns, ne);
  auto advance = [&]() {
    ahead.q += 128;
    if (ahead.q >= ahead.e) {
      ahead.row += warps;
      ahead.s = ns; ahead.e = ne; ahead.q = ns & ~3;
      bounds(ahead.row + warps, ns, ne);
    }
  };
  auto load = [&](const Step &t) { return load_quad(col, val, nnz, t.q + 4 * lane, t.e); };
  auto gather_of = [&](const int4 &c) {
    return make_float4(gather_x(x, staged, c.x), gather_x(x, staged, c.y), gather_x(x, staged, c.z),
                       gather_x(x, staged, c.w));
  };
  auto gather = [&](const Quad &t, const Step &of) { return gather_of(own_columns(t.c, of.q + 4 * lane, of.s, of.e)); };
  Step now = ahead;
  Quad a = load(now);
  advance();
  Step next = ahead;
  Quad b = load(next);
  advance();
  __syncthreads();
  // A gather reads shared memory, but says to the compiler only that it depends on its operands: `staged` comes from here on
  // from behind the barrier, and so do the gathers.
  asm volatile("" : "+r"(staged) : : "memory");
  float4 g = gather(a, now);
  float sum = 0.0f;
  while (now.row < rows) {
    const Step fresh = ahead;
    const Quad c = load(fresh);
    advance();
    const float4 gn = gather(b, next);
    sum = add(sum, quad_sum(a.v, g, now.q + 4 * lane, now.s, now.e));
    if (now.q + 128 >= now.e) {
      sum = warp_sum(sum);
      if (lane == 0) y[now.row] = sum;
      sum = 0.0f;
    }
    g = gn;
    a = b; b = c;
    now = next; next = fresh;
  }
  __syncthreads();
  if (!left_out) return;
  sum_rows_left_out<SHARED_X_THREADS>(
      longest, rows, nnz, row_ptr, col, val, y, gather_of,
      [&](int i) { return (int64_t)blockIdx.x * 32 + (i & 31) + (int64_t)(i >> 5) * warps; },
      [&](int i) { return (int64_t)(i >> 5) * warps >= rows; });
}
