// f32 BSR SpMM of 4 x 4 and 8 x 8 blocks, a group of lanes per block row (included by bsr_kernels.cu inside namespace
// swb::{anonymous}).
//
// With products and sums rounded separately the operator is bound by issue slots: the threads of bsr_spmm_row_tile_kernel
// spent one of two on loads, addresses and branches (16,384 block rows of 24 blocks of 4 x 4, N = 32: 26.3 M instructions for
// 12.6 M products and sums).  Here a group of lanes copies its block row's blocks and block columns to shared memory with
// cp.async, a chunk of four or eight blocks ahead, so that a step has no load but its rows of B and broadcasts from shared
// memory, and two adjacent columns are one packed instruction: 15.6 M instructions with four columns per lane, 19.3 M with two.
// The rows of B of a step are requested together; what hides them is other warps.  Every output is added up by one lane in
// storage order, bit for bit.
//
// 16,384 block rows of 24, N = 32: 43.0 -> 32.6 us in a row of calls; 8 x 8, 2,953 of 29, N = 96 76 -> 57, 7,427 of 10, N = 208
// 125 -> 97, 4 x 4, 7,430 of 5, N = 472 56 -> 44, 111 of 33, N = 360 16.2 -> 10.8; geometric mean over 60 sizes 0.87.  What
// remains is the end: the longest block rows run on in a few warps.  Blocks of 2 x 2 have too little to add per block (14,720 of
// 5, N = 56: 7.4 us with the other kernel, 7.9 to 15 here).
#pragma once

constexpr int GROUP_THREADS = 64;

constexpr int group_chunk(int bs) { return bs == 4 ? 8 : 4; }                // blocks staged at a time
// Blocks per step.  More rows of B in flight help narrow lanes; with four columns more warps help more (4 x 4, N = 32: 30.1 us
// with two blocks a step, 28.9 with one).
constexpr int group_blocks(int bs, int V) { return V == 4 ? 1 : bs == 4 ? 4 : 2; }
// A stage: a chunk of blocks, then their block columns.
constexpr int group_stage_words(int bs) { return group_chunk(bs) * (bs * bs + 1); }

template <int bytes>
__device__ __forceinline__ void copy_async(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src),
               "n"(bytes)
               : "memory");
}

// Two f32 in a register pair.  The assembler would fuse a packed product and a packed sum, whose roundings have to stay apart,
// so the product is a fused one with a -0 that it cannot know (x + -0 is x for every x, signed zeros and NaN among them).
typedef unsigned long long Pair;
__device__ __forceinline__ Pair pair(float a, float b) {
  Pair p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(a), "f"(b));
  return p;
}
__device__ __forceinline__ Pair mul_pair(Pair a, Pair b, Pair minus_zero) {
  Pair p;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p) : "l"(a), "l"(b), "l"(minus_zero));
  return p;
}
__device__ __forceinline__ Pair add_pair(Pair a, Pair b) {
  Pair p;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(p) : "l"(a), "l"(b));
  return p;
}

// G lanes of V adjacent columns hold a block row and a tile of G * V columns.  WIDE: block values are 16-byte aligned.
// Offset: the type that holds B's size in bytes.
template <int BS, int V, bool WIDE, typename Offset>
__global__ void __launch_bounds__(GROUP_THREADS, BS == 4 && V == 4 ? 16 : 1)
    bsr_spmm_row_group_kernel(int64_t units, int64_t N, int tiles, int G, float minus_zero, const int32_t *__restrict__ brp,
                              const int32_t *__restrict__ bci, const float *__restrict__ bv, const float *__restrict__ B,
                              float *__restrict__ C) {
  after_previous_kernel();
  constexpr int U = group_blocks(BS, V), BLOCK = BS * BS, CHUNK = group_chunk(BS), WORDS = group_stage_words(BS);
  constexpr int P = V / 2;
  extern __shared__ __align__(16) float ring[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int groups = 32 / G, group = lane / G, l = lane - group * G;
  const int64_t unit = ((int64_t)blockIdx.x * (GROUP_THREADS / 32) + warp) * groups + group;
  const bool member = group < groups && unit < units;
  const int64_t brow = tiles == 1 ? unit : unit / tiles;
  int64_t c0 = (tiles == 1 ? 0 : (unit - brow * tiles) * G * V) + l * V;
  const bool stores = member && c0 < N;
  if (c0 >= N) c0 = N - V;  // a lane past the last column repeats it and stores nothing
  int start = 0, n = 0;
  if (member) {
    start = __ldg(brp + brow);
    n = __ldg(brp + brow + 1) - start;
  }
  float *stages = ring + (warp * groups + group) * (2 * WORDS);
  auto request = [&](int left, int at) {  // the next chunk of the block row's last `left` blocks into a stage
    if (left > 0) {
      const int have = left < CHUNK ? left : CHUNK, first = start + (n - left);
      float *dst = stages + at;
      const float *src = bv + (int64_t)first * BLOCK;
      if constexpr (WIDE) {
#pragma unroll 2
        for (int i = l; i < have * (BLOCK / 4); i += G) copy_async<16>(dst + 4 * i, src + 4 * i);
      } else {
#pragma unroll 2
        for (int i = l; i < have * BLOCK; i += G) copy_async<4>(dst + i, src + i);
      }
#pragma unroll 1
      for (int i = l; i < have; i += G) copy_async<4>(dst + CHUNK * BLOCK + i, bci + first + i);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[BS][V];
  Pair sum[BS][P > 0 ? P : 1];
  const Pair mz = pair(minus_zero, minus_zero);
#pragma unroll
  for (int r = 0; r < BS; ++r) {
#pragma unroll
    for (int v = 0; v < V; ++v) acc[r][v] = 0.0f;
#pragma unroll
    for (int v = 0; v < P; ++v) sum[r][v] = 0;
  }
  const Offset pitch = (Offset)N * 4, slab = pitch * BS, lane_at = (Offset)c0 * 4;
  const char *base = reinterpret_cast<const char *>(B);
  const int most = __reduce_max_sync(0xffffffffu, n);
  request(n, 0);
  int at = 0;
  for (int done = 0, left = n; done < most; left -= CHUNK) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();  // everyone's copies of this chunk; and everyone is through with the chunk before
    request(left - CHUNK, WORDS - at);
    const float *a = stages + at;
    const int *column = reinterpret_cast<const int *>(a + CHUNK * BLOCK);
    at = WORDS - at;
    const int rest = most - done < CHUNK ? most - done : CHUNK;
    done += rest;
#pragma unroll 1
    for (int j0 = 0; j0 < rest; j0 += U, a += U * BLOCK, column += U) {
      float b[U][BS][V];
#pragma unroll
      for (int j = 0; j < U; ++j) {
        if (j0 + j < left) {
          const Offset o = (Offset)column[j] * slab + lane_at;
#pragma unroll
          for (int k = 0; k < BS; ++k) load<V>(b[j][k], reinterpret_cast<const float *>(base + (o + k * pitch)));
        }
      }
#pragma unroll
      for (int j = 0; j < U; ++j) {
        if (j0 + j < left) {
#pragma unroll
          for (int k0 = 0; k0 < BS; k0 += 4) {
            constexpr int K = 4;
            float w[BS][K];
#pragma unroll
            for (int r = 0; r < BS; ++r) {
              const float4 t = *reinterpret_cast<const float4 *>(a + j * BLOCK + r * BS + k0);
              w[r][0] = t.x; w[r][1] = t.y; w[r][2] = t.z; w[r][3] = t.w;
            }
#pragma unroll
            for (int k = 0; k < K; ++k) {
              if constexpr (P > 0) {
                Pair bb[P];
#pragma unroll
                for (int v = 0; v < P; ++v) bb[v] = pair(b[j][k0 + k][2 * v], b[j][k0 + k][2 * v + 1]);
#pragma unroll
                for (int r = 0; r < BS; ++r) {
                  const Pair ww = pair(w[r][k], w[r][k]);
#pragma unroll
                  for (int v = 0; v < P; ++v) sum[r][v] = add_pair(sum[r][v], mul_pair(ww, bb[v], mz));
                }
              } else {
#pragma unroll
                for (int r = 0; r < BS; ++r)
#pragma unroll
                  for (int v = 0; v < V; ++v) acc[r][v] = add(acc[r][v], mul(w[r][k], b[j][k0 + k][v]));
              }
            }
          }
        }
      }
    }
  }
  if (stores) {
    float *out = C + brow * BS * N + c0;
#pragma unroll
    for (int r = 0; r < BS; ++r) {
      if constexpr (P > 0) {
#pragma unroll
        for (int v = 0; v < P; ++v)
          asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[r][2 * v]), "=f"(acc[r][2 * v + 1]) : "l"(sum[r][v]));
      }
      store<V>(out + r * N, acc[r]);
    }
  }
}

template <int BS, int V>
cudaError_t launch_groups(const BsrSpmmArgs &a, cudaStream_t s) {
  // Tiles of at least eight lanes that leave few of a warp's lanes idle (34 lanes' worth of columns: two tiles of 17 would
  // use 17 of 32 lanes, four of nine 27).
  const int64_t runs = a.n_rhs / V;
  int64_t tiles = ceil_div(runs, 32);
  double most = 0;
  for (int64_t t = tiles, end = tiles + 5; t < end && ceil_div(runs, t) >= 8; ++t) {
    const int64_t g = ceil_div(runs, t);
    const double used = (double)runs / (double)(t * g) * (double)(32 / g * g) / 32;
    if (used > most + 0.05) { most = used; tiles = t; }
  }
  const int G = (int)ceil_div(runs, tiles), groups = GROUP_THREADS / 32 * (32 / G);
  tiles = ceil_div(runs, G);
  const int64_t units = a.rows / BS * tiles;
  unsigned grid = 0;  // refused, not truncated, beyond the CUDA grid limit
  if (tiles > 2147483647LL || !grid_dim(ceil_div(units, groups), &grid)) return cudaErrorInvalidConfiguration;
  const bool wide = reinterpret_cast<uintptr_t>(a.block_values) % 16 == 0;
  const bool small = a.cols * a.n_rhs < (1LL << 30);
  const size_t smem = (size_t)groups * 2 * group_stage_words(BS) * sizeof(float);
#define SWB_BSR(WIDE, OFFSET)                                                                                       \
  launch_chained(bsr_spmm_row_group_kernel<BS, V, WIDE, OFFSET>, grid, GROUP_THREADS, smem, s, units, a.n_rhs,  \
                 (int)tiles, G, -0.0f, a.block_row_ptr, a.block_col_idx, static_cast<const float *>(a.block_values), \
                 static_cast<const float *>(a.B), static_cast<float *>(a.C))
  if (!wide) SWB_BSR(false, uint64_t);
  else if (small) SWB_BSR(true, uint32_t);
  else SWB_BSR(true, uint64_t);
#undef SWB_BSR
  return cudaGetLastError();
}

// V: the columns per lane that B and C are aligned for.  Four where that leaves 24 warps for every one of 148 SMs, 32 warps with up
// to 64 columns, whose warps hold several block rows and run as long as the longest; two above 45,000 lanes, one above 20,000
// (time with four columns against two, over 100 sizes of 6 to 24 blocks a row: up to 64 columns 1.02 to 1.25 below 120,000 lanes,
// 1.03 at 131,072 (16,384 of 24 of 4 x 4, N = 32: 30.8 and 30.0 us), 0.93 to 1.01 from 160,000 on; more columns 0.85 to 1.15 from
// 90,000 to 110,000, 0.86 to 1.04 at 115,000, 0.73 to 0.94 above; two and one: 2,081 of 53, N = 32 18 and 17 us, 1,476 of 20, N =
// 448 28 and 38).  With fewer lanes, threads that read their operands themselves, two rows each, start sooner (204 block rows of 40
// of 8 x 8, N = 88: 15.9 us, here 21.9; 374 of 13 of 4 x 4, N = 16: 5.1, here 6.2).  Groups below eight lanes would crowd shared
// memory.
template <int BS>
bool try_groups(const BsrSpmmArgs &a, int V, cudaStream_t s, cudaError_t *e) {
  const int64_t brows = a.rows / BS, n = a.n_rhs;
  if (n < 8 || brows * n < 20000) return false;
  if (V == 4 && n >= 32 && brows * (n / 4) >= 148 * 32 * (n <= 64 ? 32 : 24)) *e = launch_groups<BS, 4>(a, s);
  else if (V >= 2 && n >= 16 && brows * (n / 2) >= 45000) *e = launch_groups<BS, 2>(a, s);
  else *e = launch_groups<BS, 1>(a, s);
  return true;
}
