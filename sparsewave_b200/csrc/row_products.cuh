// Sequential row sums over products formed in position order by the whole block: thread-per-row SpMV and SpMM with up to
// four right-hand sides, eight on few rows (included by spmv_kernels.cu inside namespace swb::{anonymous}).
//
// The reference mapping gives a thread a row, so that lanes read col and val a row length apart: 32 sectors a load, each
// fetched for four bytes, and a chain of dependent loads as long as the longest row.  Here a block owns a run of rows,
// hence one range of positions.  It forms the products of a tile of positions with coalesced loads (every gather of a
// tile in flight at once) and leaves them in shared memory; then one thread per output adds up its row's part of the
// tile in position order.  The sum is the reference's, bit for bit; the range of positions and not the longest row
// decides the number of dependent loads.  Bound by launch and three dependent latencies on small matrices and by the
// gather of x on large ones: 206,501 rows of 6 on average 13.0 -> 9.6 us, 1 M rows of 32 289 -> 139 us (32 M gathers
// at 230 G/s), 50,000 power-law rows of up to 25,000 positions 1163 -> 140 us.
//
// N = 1, 2, 4, 8 on aligned rows of B: a thread forms the products of a position, with one or two vector loads.  Other N
// up to 8: a thread forms one product, so that neighbouring lanes read a row of B together.
//
// The tile is padded by one element (of 4, 8 or 16 bytes) in 32, so that rows of 32 or 64 positions do not start in one
// bank.
#pragma once

// Threads of a block, most rows of a block, and products of a tile before padding.  Where 512 threads and 4,096 products per
// block cover the matrix with four blocks per SM, all of it is in flight at once and evenly spread (206,501 ragged rows of 6:
// 12.0 -> 9.7 us a call against blocks of 256, of which some SMs get six and others five).  (Three blocks fit an SM with N = 3
// and unaligned 4, which take 40 registers, and two with N = 5 to 7 and unaligned 8, which take 56 to 64 and run on up to
// 8,192 rows only; the rest waits.)  Larger matrices take blocks of
// 128 and tiles of 2,048, whose gaps between gathers and sums interleave better (1 M ragged rows of 10: 52.4 -> 51.0); with
// several columns those hold too few positions, and blocks are of 256 (404,892 banded rows of 19, N = 4: 49 -> 46).
struct ProductsOnce { static constexpr int THREADS = 512, WORDS = 4096; };
template <int N> struct ProductsMany { static constexpr int THREADS = N == 1 ? 128 : 256, WORDS = N == 1 ? 2048 : 4096; };

template <int W> struct Words;  // what one load brings
template <> struct Words<1> { using T = float; };
template <> struct Words<2> { using T = float2; };
template <> struct Words<4> { using T = float4; };

// N right-hand sides; W words per load: N (8 takes two loads of 4), or 1 for the thread-per-product form.
template <int N, int W, typename Shape>
__global__ void __launch_bounds__(Shape::THREADS)
    row_products_kernel(int64_t rows, int rows_per_block, const int32_t *__restrict__ row_ptr,
                        const int32_t *__restrict__ col, const float *__restrict__ val, const float *__restrict__ B,
                        float *__restrict__ C, bool accumulate) {
  after_previous_kernel();
  using T = typename Words<W>::T;
  constexpr int PRODUCT_THREADS = Shape::THREADS, PRODUCT_WORDS = Shape::WORDS;
  constexpr int TILE = PRODUCT_WORDS / N;     // positions
  constexpr bool BY_PRODUCT = W == 1;         // items are products, else positions
  constexpr int ITEMS = BY_PRODUCT ? N : 1;   // items per position
  constexpr int LOADS = BY_PRODUCT ? 1 : N / W;
  constexpr int PER = LOADS * W >= 8 ? 2 : 4; // items in flight per thread
  constexpr int UNITS = PRODUCT_WORDS / W;    // the tile in units of one load
  __shared__ T tile_mem[UNITS + UNITS / 32];
  const float *products = reinterpret_cast<const float *>(tile_mem);
  __shared__ int offsets[PRODUCT_THREADS + 1];
  const int tid = threadIdx.x;
  const int64_t r0 = (int64_t)blockIdx.x * rows_per_block;
  if (r0 >= rows) return;
  const int count = r0 + rows_per_block < rows ? rows_per_block : (int)(rows - r0);
  for (int i = tid; i <= count; i += PRODUCT_THREADS) offsets[i] = row_ptr[r0 + i];
  __syncthreads();
  const int first = offsets[0], last = offsets[count];
  float sum[N];  // of outputs tid, tid + PRODUCT_THREADS, ... (rows_per_block <= PRODUCT_THREADS)
#pragma unroll
  for (int k = 0; k < N; ++k) sum[k] = 0.0f;
  // unsigned: behind the last tile of a matrix of up to 2^31 - 1 nonzeros `tile` passes the int32 maximum
  for (unsigned tile = first; tile < (unsigned)last; tile += TILE) {
    const int items = (last - tile < TILE ? (int)(last - tile) : TILE) * ITEMS;
    for (int i0 = tid; i0 < items; i0 += PER * PRODUCT_THREADS) {
      int c[PER];
      float v[PER];
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const int i = i0 + k * PRODUCT_THREADS;
        const unsigned p = tile + i / ITEMS;
        c[k] = i < items ? ld_stream(col + p) : 0;
        v[k] = i < items ? ld_stream(val + p) : 0.0f;
      }
      T b[PER][LOADS];
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const int i = i0 + k * PRODUCT_THREADS;
        if (i < items) {
          const T *src = reinterpret_cast<const T *>(B + (int64_t)c[k] * N + (BY_PRODUCT ? i % ITEMS : 0));
#pragma unroll
          for (int j = 0; j < LOADS; ++j) b[k][j] = __ldg(src + j);
        }
      }
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const int i = i0 + k * PRODUCT_THREADS;
        if (i < items) {
#pragma unroll
          for (int j = 0; j < LOADS; ++j) {
            T w = b[k][j];
            float *f = reinterpret_cast<float *>(&w);
#pragma unroll
            for (int e = 0; e < W; ++e) f[e] = mul(v[k], f[e]);
            const int unit = i * LOADS + j;
            tile_mem[unit + (unit >> 5)] = w;
          }
        }
      }
    }
    __syncthreads();
    auto product = [&](int word) { return products[word + (word / (32 * W)) * W]; };
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int o = tid + k * PRODUCT_THREADS;
      if (o < count * N) {
        const int r = o / N, j = o - r * N;
        int p = (int)(offsets[r] - tile), end = (int)(offsets[r + 1] - tile);
        if (p < 0) p = 0;
        if (end > TILE) end = TILE;
        float s = sum[k];
        for (; p + 4 <= end; p += 4) {
          const float a0 = product(p * N + j), a1 = product((p + 1) * N + j);
          const float a2 = product((p + 2) * N + j), a3 = product((p + 3) * N + j);
          s = add(add(add(add(s, a0), a1), a2), a3);
        }
        for (; p < end; ++p) s = add(s, product(p * N + j));
        sum[k] = s;
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const int o = tid + k * PRODUCT_THREADS;
    if (o < count * N) {
      float *out = C + r0 * N + o;
      *out = accumulate ? add(*out, sum[k]) : sum[k];
    }
  }
}

// Rows per block: as many as fill a tile, but no fewer blocks than four per SM while a block keeps 16 rows (the sums
// take one thread per row and column).
template <typename Shape>
int64_t product_rows_per_block(int64_t rows, int64_t nnz, int64_t n_rhs) {
  const int64_t mean = rows > 0 ? nnz / rows : 0;
  int64_t per = Shape::WORDS / n_rhs * 7 / 8 / (mean > 0 ? mean : 1);
  const int64_t spread = ceil_div(rows, 148 * 4);
  if (per > spread) per = spread;
  if (per < 16) per = 16;
  return per > Shape::THREADS ? Shape::THREADS : per;
}
inline bool products_once(int64_t rows, int64_t nnz, int64_t n_rhs) {
  return rows <= (int64_t)148 * 4 * ProductsOnce::THREADS && nnz * n_rhs <= (int64_t)148 * 4 * ProductsOnce::WORDS * 7 / 8;
}

template <int N, int W, typename Shape>
cudaError_t launch_row_products_in(const CsrSpmmArgs &a, cudaStream_t s) {
  const int64_t per = product_rows_per_block<Shape>(a.rows, a.nnz, N);
  unsigned grid = 0;
  if (!grid_dim(ceil_div(a.rows, per), &grid)) return cudaErrorInvalidConfiguration;
  launch_chained(row_products_kernel<N, W, Shape>, grid, Shape::THREADS, 0, s, a.rows, (int)per, a.row_ptr, a.col_idx, a.val,
                 a.B, a.C, a.accumulate);
  return cudaGetLastError();
}

template <int N, int W>
cudaError_t launch_row_products_of(const CsrSpmmArgs &a, cudaStream_t s) {
  return products_once(a.rows, a.nnz, N) ? launch_row_products_in<N, W, ProductsOnce>(a, s)
                                         : launch_row_products_in<N, W, ProductsMany<N>>(a, s);
}
