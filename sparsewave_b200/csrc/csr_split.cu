// Column parts of an uploaded CSR matrix, made on the device: entries whose column lies below a cut and the rest, each
// part in the original order of its entries.  A warp per row; run once per upload, bound by reading and writing the
// matrix once (on one host core the same takes some 10 ns an entry).
#include "swb_index.h"
#include "swb_kernels.h"

namespace swb {
namespace {

constexpr unsigned FULL = 0xffffffffu;

__global__ void count_below_kernel(int64_t rows, const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ col,
                                   int32_t cut, int32_t *__restrict__ below) {
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const int64_t end = row_ptr[row + 1];
  int n = 0;
  for (int64_t p = row_ptr[row] + lane; p < end; p += 32) n += col[p] < cut;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) n += __shfl_xor_sync(FULL, n, off);
  if (lane == 0) below[row] = n;
}

__global__ void split_columns_kernel(int64_t rows, const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ col,
                                     const float *__restrict__ val, int32_t cut, const int32_t *__restrict__ low_ptr,
                                     const int32_t *__restrict__ high_ptr, int32_t *__restrict__ low_col,
                                     float *__restrict__ low_val, int32_t *__restrict__ high_col,
                                     float *__restrict__ high_val) {
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const unsigned before = (1u << lane) - 1u;
  int64_t lo = low_ptr[row], hi = high_ptr[row];
  const int64_t end = row_ptr[row + 1];
  for (int64_t base = row_ptr[row]; base < end; base += 32) {  // uniform in the warp
    const int64_t p = base + lane;
    const bool in = p < end;
    const int32_t c = in ? col[p] : 0;
    const unsigned lows = __ballot_sync(FULL, in && c < cut), all = __ballot_sync(FULL, in);
    if (in && c < cut) {
      const int64_t at = lo + __popc(lows & before);
      low_col[at] = c;
      low_val[at] = val[p];
    } else if (in) {
      const int64_t at = hi + __popc(~lows & all & before);
      high_col[at] = c;
      high_val[at] = val[p];
    }
    lo += __popc(lows);
    hi += __popc(all & ~lows);
  }
}

}  // namespace

cudaError_t launch_count_below(int64_t rows, const int32_t *row_ptr, const int32_t *col, int32_t cut, int32_t *below,
                               cudaStream_t s) {
  unsigned grid = 0;
  if (!grid_dim(ceil_div(rows, 8), &grid)) return cudaErrorInvalidConfiguration;
  count_below_kernel<<<grid, 256, 0, s>>>(rows, row_ptr, col, cut, below);
  return cudaGetLastError();
}

cudaError_t launch_split_columns(int64_t rows, const int32_t *row_ptr, const int32_t *col, const float *val, int32_t cut,
                                 const int32_t *low_ptr, const int32_t *high_ptr, int32_t *low_col, float *low_val,
                                 int32_t *high_col, float *high_val, cudaStream_t s) {
  unsigned grid = 0;
  if (!grid_dim(ceil_div(rows, 8), &grid)) return cudaErrorInvalidConfiguration;
  split_columns_kernel<<<grid, 256, 0, s>>>(rows, row_ptr, col, val, cut, low_ptr, high_ptr, low_col, low_val, high_col,
                                            high_val);
  return cudaGetLastError();
}

}  // namespace swb
