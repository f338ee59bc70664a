// BSR SpMM for 8x8, 16x16 and 32x32 bf16 blocks with warp-level MMAs, operands from global memory straight into their
// fragments: any number of columns, any alignment, few block rows as well as many (arithmetic as in bsr_tcgen05.cu).
//
// A warp owns a block row and 16 T columns and forms the product transposed, so that one instruction shape fits all block
// sizes: mma.sync.m16n8k16 with m = 16 columns of B, n = 8 rows of a block, k = 16 local columns (a step: two 8 x 8 blocks, one
// 16 x 16 block, half of a 32 x 32 block).  Which local column is which k, and which column of B which m, is free as long as
// both operands agree.  Lane (g, q) = (lane / 4, lane % 4) takes adjacent local columns 4 q .. 4 q + 3 of a step and
// adjacent columns 2 T g .. 2 T g + 2 T - 1: its share of the block values is one load per 8 rows, its share of a row of B one
// load of up to 16 bytes, and its results are adjacent columns of C.  Pairs of rows of B are interleaved by byte permutes.
// The next steps' loads are in flight during this step's MMAs, block columns are held 32 at a time by the warp's lanes.
//
// Every output is added up over its block row's steps in storage order, so that a part of a matrix has the bits of the whole,
// whichever kernel takes either: as one chain of MMAs or (bsr_chain_sums) as f32 sums of steps or, 32 x 32 blocks, of segments of
// two, four or eight blocks by the block row's length, each of which is a chain of its own.  Where block rows are few, a team of
// up to eight warps shares one all the same.  Its members take segments in turn and add up each other's sums, in order, for their tiles of
// 8 rows; or they load the steps in turn and hand them over in shared memory, and each of the first members adds up its share of
// the block row's rows.
//
// What bounds it: launch and latency on small calls, L1 on large ones (eight lanes of a load touch four lines, some 64 lookups
// for 2 KB of B; ncu: L1 data pipe 67 %, tensor pipe 18 % on 1,024 block rows of 51, N = 512), which bsr_tcgen05.cu then takes.
// Tried: the same loads through a ring in shared memory (178 us against 134 on that size).  Before, on the CUDA cores or with
// tcgen05 at any size: 123 block rows of 61 blocks of 32 x 32, N = 2 138 -> 7.6 us; 382 of 27, N = 29 109 -> 15.9; 1,438 of 15
// blocks of 8 x 8, N = 80 30.0 -> 10.0; 90 of 36 blocks of 16 x 16, N = 88 17.5 -> 7.9.  A fixed order of sums has its price
// where few warps have much to add up: a block row in as many parts as there are warps, added up at the end, took 5.8, 12.8, 10.4
// and 5.8 us.  With operands handed over the two sizes of 32 x 32 took 11.7 and 20.4, and 107 of 1 to 63 and odd numbers of columns
// 1.19 times the time of segments.  Segments for the smaller blocks too: 1.06 and 1.04 times the time (8 x 8, 16 x 16; where a
// warp has whole block rows 1.09 and 1.14).  Tried for teams that hand over operands: two rounds' loads in flight (spills; 1.09
// times the time over 170 sizes), a barrier per step (1.13), sums of steps in place of operands (1.00 to 1.2).
#include <cuda_bf16.h>

#include "swb_chain.cuh"
#include "swb_index.h"
#include "swb_kernels.h"

namespace swb {
namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int MMA_WARPS = 8;
// Steps in hand (one being multiplied, the others' loads in flight) and CTAs per SM that registers are kept for.  Narrow B leaves
// registers for more of both: 2,970 block rows of 52 blocks of 16 x 16, N = 8 36.9 -> 30.4 us with three steps and CTAs (37.6
// with four CTAs of two steps, 37.1 with two of four).  8 x 8 blocks then need no more than 64 registers, which is four CTAs.
constexpr int mma_depth(int bs, int T) { return bs == 32 || T > 1 ? 2 : 3; }
// Steps that each member of a team has in flight and hands over at a time: 48 KB of shared memory for eight members.
constexpr int team_steps(int bs, int T) { return T == 4 ? 2 : bs == 32 && T == 2 ? 3 : 4; }
constexpr int mma_ctas(int bs, int T, int V) { return bs < 32 && T == 1 ? 3 : bs == 16 && T == 2 && V > 1 ? 3 : 2; }

// H: a lane's share of one step (1) or of both of a 32 x 32 block (2), which lie 16 rows of B and local columns apart.
template <int BS, int T, int V, int H>
struct Fragments {
  static constexpr int TILES = BS / 8;  // n8 tiles of block rows
  uint32_t slab[H][4][T + (V == 0)];    // four rows of B, 2 T adjacent columns each (V = 0: the words that hold them)
  uint32_t block[H][TILES][2];          // block row 8 u + g, four local columns
};
// Words per lane of a step as its MMAs take it: four for every 16 columns of B, two for every 8 rows of blocks.
constexpr int step_words(int bs, int T) { return 4 * T + bs / 4; }

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
// A step's 16 products added to the sums: by the tensor core, or (its sums are cut off, not rounded) as a sum of their own that
// is then added, rounded to nearest.
template <bool CHAIN>
__device__ __forceinline__ void add_step(float (&sum)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (CHAIN) {
    mma(sum, a[0], a[1], a[2], a[3], b0, b1);
  } else {
    float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    mma(d, a[0], a[1], a[2], a[3], b0, b1);
#pragma unroll
    for (int i = 0; i < 4; ++i) sum[i] += d[i];
  }
}

// V: elements per load of a row of B, or 0: N is odd and B starts at a word, so that rows in turn start at a word and in the
// middle of one.  WIDE: block values are aligned for loads of a lane's share of a row.  TEAM: several warps share a unit, 2, 4 or 8 but
// no fewer than there are tiles of 8 rows in a block.
template <int BS, int T, int V, bool WIDE, bool TEAM, bool CHAIN>
__device__ __forceinline__ void add_in_order(int64_t units, int tiles, int team_warps, int64_t N, const int32_t *__restrict__ brp,
                                             const int32_t *__restrict__ bci, const __nv_bfloat16 *__restrict__ bv,
                                             const __nv_bfloat16 *__restrict__ B, __nv_bfloat16 *__restrict__ C) {
  constexpr int H = BS == 32 && !TEAM ? 2 : 1;
  using F = Fragments<BS, T, V, H>;
  // Steps of this kernel per two blocks, and those whose block columns the warp holds.
  constexpr int PER_TWO = BS == 8 ? 1 : BS == 16 || H == 2 ? 2 : 4, BATCH = 16 * PER_TWO;
  constexpr int DEPTH = TEAM ? team_steps(BS, T) : mma_depth(BS, T);
  constexpr int WORDS = step_words(BS, T);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  const int split = TEAM ? team_warps : 1, team = warp / split, member = warp % split;
  const int64_t unit = (int64_t)blockIdx.x * (MMA_WARPS / split) + team;
  const bool active = unit < units;
  const int64_t brow = active ? unit / tiles : 0;
  const int64_t col0 = (active ? unit - brow * tiles : 0) * (16 * T) + g * (2 * T);
  const int valid = N - col0 >= 2 * T ? 2 * T : N > col0 ? (int)(N - col0) : 0;
  int start = 0, end = 0;
  if (active) {
    start = brp[brow];
    end = brp[brow + 1];
  }
  const int steps = BS == 8 ? (end - start + 1) / 2 : (end - start) * (PER_TWO / 2);

  constexpr int SUMS = TEAM ? 1 : F::TILES;  // tiles of 8 rows that the warp adds up: all, or (the first warps of a team) one
  float acc[SUMS][T][4];
#pragma unroll
  for (int u = 0; u < SUMS; ++u)
#pragma unroll
    for (int t = 0; t < T; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[u][t][i] = 0.0f;

  const int local = BS == 8 ? 4 * (q & 1) : 4 * q;  // the lane's first local column of a step
  const int second = BS == 8 ? q >> 1 : 0;          // which of a step's two blocks it reads
  const __nv_bfloat16 *Bt = B + col0 + (int64_t)local * N;
  auto block_of = [&](int k) { return PER_TWO == 1 ? 2 * k : PER_TWO == 2 ? k : k >> 1; };
  auto column = [&](int k) {  // block columns of the steps from k on
    const int p = start + block_of(k) + lane;
    return p < end ? __ldg(bci + p) : 0;
  };
  int here = column(0), ahead = column(BATCH);
  auto load = [&](F &f, int k) {  // called for k = member, member + split, ... (a batch is a multiple of every split)
    const int i = k % BATCH;
    if (i == member && k != member) { here = ahead; ahead = column(k - i + BATCH); }
    const int bc = __shfl_sync(FULL, here, block_of(i) + second);
    const int p = start + block_of(k) + second;
    const int from = PER_TWO == 4 ? 16 * (k & 1) : 0;
    const bool in = BS != 8 || p < end;  // the second block of a last step may be missing: zeros
    const __nv_bfloat16 *b = Bt + ((int64_t)bc * BS + from) * N;
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if constexpr (V == 0) load_words<T>(f.slab[h][r], b + (16 * h + r) * N, r & 1, in ? valid : 0);
        else load_row<T, V>(f.slab[h][r], b + (16 * h + r) * N, in ? valid : 0);
      }
    const __nv_bfloat16 *a = bv + (int64_t)p * (BS * BS) + g * BS + from + local;
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
      for (int u = 0; u < F::TILES; ++u) load_row<2, WIDE ? 4 : 1>(f.block[h][u], a + u * 8 * BS + 16 * h, in ? 4 : 0);
  };
  auto columns_of = [&](const F &f, int h, int t, uint32_t (&a)[4]) {  // the MMA's operand of columns 2 t and 2 t + 1
    uint32_t x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if constexpr (V == 0) x[i] = i & 1 ? __byte_perm(f.slab[h][i][t], f.slab[h][i][t + 1], 0x5432) : f.slab[h][i][t];
      else x[i] = f.slab[h][i][t];
    }
    a[0] = __byte_perm(x[0], x[1], 0x5410); a[1] = __byte_perm(x[0], x[1], 0x7632);
    a[2] = __byte_perm(x[2], x[3], 0x5410); a[3] = __byte_perm(x[2], x[3], 0x7632);
  };
  F f[DEPTH];
  if constexpr (!TEAM) {
#pragma unroll
    for (int d = 0; d < DEPTH - 1; ++d)
      if (d < steps) load(f[d], d);
    for (int k = 0; k < steps;) {
#pragma unroll
      for (int d = 0; d < DEPTH; ++d) {
        if (k + DEPTH - 1 < steps) load(f[(d + DEPTH - 1) % DEPTH], k + DEPTH - 1);
#pragma unroll
        for (int h = 0; h < H; ++h)
#pragma unroll
          for (int t = 0; t < T; ++t) {
            uint32_t a[4];
            columns_of(f[d], h, t, a);
#pragma unroll
            for (int u = 0; u < F::TILES; ++u) add_step<CHAIN>(acc[u][t], a, f[d].block[h][u][0], f[d].block[h][u][1]);
          }
        if (++k >= steps) break;
      }
    }
  } else {
    // A round: each member puts its steps, every split-th one, into the team's shared memory; behind a barrier the first members
    // add them up, in order, for a tile of 8 rows each, while the next round's loads are in flight.
    extern __shared__ __align__(16) uint4 handed[];
    constexpr int STEP = WORDS * 8;  // quads
    uint4 *steps_of_team = handed + team * split * (DEPTH * STEP);
    auto meet = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(32 * split) : "memory"); };
    auto load_round = [&](int k) {
#pragma unroll
      for (int d = 0; d < DEPTH; ++d)
        if (k + d * split < steps) load(f[d], k + d * split);
    };
    load_round(member);
    for (int first = 0; first < steps; first += DEPTH * split) {
#pragma unroll
      for (int d = 0; d < DEPTH; ++d) {
        if (first + d * split + member < steps) {
          uint4 *mine = steps_of_team + (d * split + member) * STEP;
#pragma unroll
          for (int t = 0; t < T; ++t) {
            uint32_t a[4];
            columns_of(f[d], 0, t, a);
            mine[t * 32 + lane] = make_uint4(a[0], a[1], a[2], a[3]);
          }
          uint2 *blocks = reinterpret_cast<uint2 *>(mine + T * 32);
#pragma unroll
          for (int u = 0; u < F::TILES; ++u) blocks[u * 32 + lane] = make_uint2(f[d].block[0][u][0], f[d].block[0][u][1]);
        }
      }
      meet();
      load_round(first + DEPTH * split + member);
      if (member < F::TILES) {
        const int n = steps - first < DEPTH * split ? steps - first : DEPTH * split;
        const uint4 *step = steps_of_team;
#pragma unroll CHAIN || T < 4 ? 4 : 2
        for (int j = 0; j < n; ++j, step += STEP) {
          const uint2 v = reinterpret_cast<const uint2 *>(step + T * 32)[member * 32 + lane];
#pragma unroll
          for (int t = 0; t < T; ++t) {
            const uint4 w = step[t * 32 + lane];
            const uint32_t a[4] = {w.x, w.y, w.z, w.w};
            add_step<CHAIN>(acc[0][t], a, v.x, v.y);
          }
        }
      }
      if (first + DEPTH * split < steps) meet();
    }
  }
  if (!active || (TEAM && member >= F::TILES)) return;
#pragma unroll
  for (int u = 0; u < SUMS; ++u) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      uint32_t w[T];
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(acc[u][t][r], acc[u][t][2 + r]);
        w[t] = *reinterpret_cast<const uint32_t *>(&h);
      }
      store_row<T, V ? V : 1>(C + (brow * BS + 8 * (TEAM ? member : u) + 2 * q + r) * N + col0, w, valid);
    }
  }
}

// 32 x 32 blocks as sums of segments.  A step is a block, of which lane (g, q) takes local columns 8 q .. 8 q + 7.
template <int T, int V>
struct SegmentFragments {
  uint32_t slab[8][T + (V == 0)];  // eight rows of B, 2 T adjacent columns each (V = 0: the words that hold them)
  uint32_t block[4][4];            // block row 8 u + g, eight local columns
};
// Blocks of a segment: by the block row's length alone.  A chain of L MMAs is off by some 1.5e-8 L of its size, sums rounded one by
// one by 8e-9 times the root of their number, hence longer segments on longer rows only.
__device__ __forceinline__ int segment_log2_length(int blocks) { return blocks <= 16 ? 1 : blocks <= 64 ? 2 : 3; }
// Tiles of 8 rows whose sums a warp adds up, and whether it does so in registers.
constexpr int share_of_sums(bool team) { return team ? 2 : 4; }
constexpr bool sums_in_registers(int T) { return T == 1; }
// Segments that a member of a team sums before they are handed over, and shared memory, of which the default 48 KB are the limit.
constexpr int segments_at_once(int T) { return T == 1 ? 3 : 1; }
constexpr int segment_smem(int T, bool team) {
  return MMA_WARPS * T * 512 * ((sums_in_registers(T) ? 0 : share_of_sums(team)) + (team ? 4 * segments_at_once(T) : 0));
}
__device__ __forceinline__ void add4(float4 &a, const float4 &b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }

template <int T, int V, bool WIDE, bool TEAM>
__device__ __forceinline__ void add_in_segments(int64_t units, int tiles, int team_warps, int64_t N,
                                                const int32_t *__restrict__ brp, const int32_t *__restrict__ bci,
                                                const __nv_bfloat16 *__restrict__ bv, const __nv_bfloat16 *__restrict__ B,
                                                __nv_bfloat16 *__restrict__ C) {
  using F = SegmentFragments<T, V>;
  constexpr int BS = 32, TILES = BS / 8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  const int split = TEAM ? team_warps : 1, team = warp / split, member = warp % split;
  const int64_t unit = (int64_t)blockIdx.x * (MMA_WARPS / split) + team;
  const bool active = unit < units;
  const int64_t brow = active ? unit / tiles : 0;
  const int64_t col0 = (active ? unit - brow * tiles : 0) * (16 * T) + g * (2 * T);
  const int valid = N - col0 >= 2 * T ? 2 * T : N > col0 ? (int)(N - col0) : 0;
  int start = 0, end = 0;
  if (active) {
    start = brp[brow];
    end = brp[brow + 1];
  }
  const int steps = end - start;
  const int log2_length = segment_log2_length(steps), length = 1 << log2_length;
  const int segments = (steps + length - 1) >> log2_length;
  auto own = [&](int j) { return ((((j >> log2_length) * split) + member) << log2_length) | (j & (length - 1)); };  // the j-th step

  float acc[TILES][T][4];  // the segment's sums
#pragma unroll
  for (int u = 0; u < TILES; ++u)
#pragma unroll
    for (int t = 0; t < T; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[u][t][i] = 0.0f;
  // The block row's: all of its rows, or a team member's share of the tiles of 8 rows.  In registers, where there are any left.
  constexpr int SUMS = share_of_sums(TEAM);
  constexpr bool KEPT = sums_in_registers(T);
  extern __shared__ __align__(16) uint4 handed[];
  float4 *shared_sums = reinterpret_cast<float4 *>(handed) + warp * (SUMS * T * 32) + lane;
  float4 sum[KEPT ? SUMS : 1][KEPT ? T : 1];
#pragma unroll
  for (int u = 0; u < SUMS; ++u)
#pragma unroll
    for (int t = 0; t < T; ++t) {
      if constexpr (KEPT) sum[u][t] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      else shared_sums[(u * T + t) * 32] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  auto of_sums = [&](int u, int t) -> float4 & {
    if constexpr (KEPT) return sum[u][t];
    else return shared_sums[(u * T + t) * 32];
  };

  const __nv_bfloat16 *Bt = B + col0 + (int64_t)(8 * q) * N;
  auto column = [&](int k) {  // block columns of the steps from k on
    const int p = start + k + lane;
    return p < end ? __ldg(bci + p) : 0;
  };
  // Held: 32 of them, or (a member of a team on a longer row) a segment's, and those behind them.
  const bool whole = steps <= 32;
  int held = TEAM && !whole ? own(0) : 0;
  int here = column(held), ahead = whole ? 0 : column(held + (TEAM ? split << log2_length : 32));
  auto load = [&](F &f, int k) {
    if (!whole && k != held && (k & (TEAM ? length - 1 : 31)) == 0) {
      held = k;
      here = ahead;
      ahead = column(k + (TEAM ? split << log2_length : 32));
    }
    const int bc = __shfl_sync(FULL, here, k - held);
    const __nv_bfloat16 *b = Bt + (int64_t)bc * BS * N;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if constexpr (V == 0) load_words<T>(f.slab[r], b + r * N, r & 1, valid);
      else load_row<T, V>(f.slab[r], b + r * N, valid);
    }
    const __nv_bfloat16 *a = bv + (int64_t)(start + k) * (BS * BS) + g * BS + 8 * q;
#pragma unroll
    for (int u = 0; u < TILES; ++u) load_row<4, WIDE ? 8 : 1>(f.block[u], a + u * 8 * BS, 8);
  };
  auto compute = [&](const F &f) {
#pragma unroll
    for (int r = 0; r < 8; r += 4)
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
        for (int u = 0; u < TILES; ++u) mma(acc[u][t], a0, a1, a2, a3, f.block[u][r / 2], f.block[u][r / 2 + 1]);
      }
  };
  // The end of a segment: its sums are added to the block row's.  The members of a team put theirs into shared memory and add up
  // an exchange's, in order, for their tiles of 8 rows.
  constexpr int SLOT = TILES * T * 32, AT_ONCE = segments_at_once(T);
  float4 *slots = reinterpret_cast<float4 *>(handed) + (KEPT ? 0 : MMA_WARPS * SUMS * T * 32) + (warp - member) * (AT_ONCE * SLOT) +
                  lane;
  int first = 0;  // segment of the exchange
  auto meet = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(32 * split) : "memory"); };
  auto exchange = [&] {
    meet();
    const int n = segments - first < AT_ONCE * split ? segments - first : AT_ONCE * split;
#pragma unroll
    for (int i = 0; i < SUMS; ++i) {
      const int u = member + i * split;
      if (u < TILES) {
#pragma unroll
        for (int t = 0; t < T; ++t) {
          float4 w = of_sums(i, t);
#pragma unroll 4
          for (int m = 0; m < n; ++m) add4(w, slots[m * SLOT + (u * T + t) * 32]);
          of_sums(i, t) = w;
        }
      }
    }
    first += AT_ONCE * split;
    if (first < segments) meet();
  };
  auto end_segment = [&](int segment) {
#pragma unroll
    for (int u = 0; u < TILES; ++u)
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const float4 w = make_float4(acc[u][t][0], acc[u][t][1], acc[u][t][2], acc[u][t][3]);
        if constexpr (TEAM) slots[(segment - first) * SLOT + (u * T + t) * 32] = w;
        else add4(of_sums(u, t), w);
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[u][t][i] = 0.0f;
      }
    if (TEAM && segment - first >= (AT_ONCE - 1) * split) exchange();
  };
  F f[2];
  int last = -1;  // segment
  if (own(0) < steps) load(f[0], own(0));
  // Segments have an even number of blocks, but for the block row's last one, which ends behind the loop.
  for (int j = 0; own(j) < steps;) {
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      if (own(j + 1) < steps) load(f[1 - d], own(j + 1));
      compute(f[d]);
      last = own(j) >> log2_length;
      if (own(++j) >= steps) break;
      if (d == 1 && (j & (length - 1)) == 0) end_segment(last);
    }
  }
  if (last >= 0) end_segment(last);
  if constexpr (TEAM)
    while (first < segments) exchange();
  if (!active) return;
#pragma unroll
  for (int i = 0; i < SUMS; ++i) {
    const int u = TEAM ? member + i * split : i;
    if (u >= TILES) break;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      uint32_t w[T];
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const float4 v = of_sums(i, t);
        const __nv_bfloat162 h = r == 0 ? __floats2bfloat162_rn(v.x, v.z) : __floats2bfloat162_rn(v.y, v.w);
        w[t] = *reinterpret_cast<const uint32_t *>(&h);
      }
      store_row<T, V ? V : 1>(C + (brow * BS + 8 * u + 2 * q + r) * N + col0, w, valid);
    }
  }
}

template <int BS, int T, int V, bool WIDE, bool TEAM, bool CHAIN>
__global__ void __launch_bounds__(32 * MMA_WARPS, TEAM ? 2 : mma_ctas(BS, T, V))
    bsr_spmm_mma_kernel(int64_t units, int tiles, int team_warps, int64_t N, const int32_t *__restrict__ brp,
                        const int32_t *__restrict__ bci, const __nv_bfloat16 *__restrict__ bv,
                        const __nv_bfloat16 *__restrict__ B, __nv_bfloat16 *__restrict__ C) {
  after_previous_kernel();
  if constexpr (BS == 32 && !CHAIN) add_in_segments<T, V, WIDE, TEAM>(units, tiles, team_warps, N, brp, bci, bv, B, C);
  else add_in_order<BS, T, V, WIDE, TEAM, CHAIN>(units, tiles, team_warps, N, brp, bci, bv, B, C);
}

template <int BS, int T, int V, bool WIDE, bool CHAIN = false>
cudaError_t launch_mma(const BsrSpmmArgs &a, int sm_count, cudaStream_t s) {
  const int64_t tiles = ceil_div(a.n_rhs, 16 * T), units = a.rows / BS * tiles;
  // Warps of a block row: more while the GPU has no more than ten per SM and each has a step (16 x 16, N = 8, us with 1, 2, 4 and
  // 8 warps: 80 block rows of 30 9.9, 7.0, 4.9, 3.9; 300 of 20 8.3, 5.4, 4.4, 4.8; 600 of 12 6.6, 4.8, 5.4, 6.1; 2,000 of 20 11.0,
  // 11.4, 13.9, 17.5).  Blocks of 32 x 32 have four tiles of rows for four adding warps, up to 20 warps per SM, and four others
  // that only load, up to 18 (measured on narrow B, which has segments since, 1, 4 and 8 warps: 300 of 20, N = 8 12.2, 9.7, 7.9; 80 of
  // 30, N = 48 19.8, 13.6, 11.1; 300 of 20, N = 48 18.0, 16.6, 18.9; 382 of 27, N = 29 31.3, 20.1, -; 1,000 of 20, N = 48 23.4, 40.7,
  // 43.0).  With segments twice as many while there are fewer than ten per SM and each has two blocks (16 per SM: 1.02 times the time).
  int split = 1;
  if (BS == 32 && !CHAIN) {
    while (split < MMA_WARPS && units * split < 10 * (int64_t)sm_count && a.nnzb * BS >= split * 2 * a.rows) split *= 2;
  }
  for (int more = BS == 32 ? 4 : 2; more <= MMA_WARPS && (BS != 32 || CHAIN); more *= 2)
    if (units * more <= (int64_t)sm_count * (BS != 32 ? 10 : more == 4 ? 20 : 18) && a.nnzb * BS * BS >= more * 8 * a.rows) split = more;
  unsigned grid = 0;
  if (!grid_dim(ceil_div(units * split, MMA_WARPS), &grid)) return cudaErrorInvalidConfiguration;
  const size_t smem = BS == 32 && !CHAIN ? segment_smem(T, split > 1)  // at most 48 KB
                      : split > 1 ? MMA_WARPS * team_steps(BS, T) * step_words(BS, T) * 32 * 4 : 0;
  launch_chained(split > 1 ? bsr_spmm_mma_kernel<BS, T, V, WIDE, true, CHAIN> : bsr_spmm_mma_kernel<BS, T, V, WIDE, false, CHAIN>,
                 grid, 32 * MMA_WARPS, smem, s, units, (int)tiles, split, a.n_rhs, a.block_row_ptr, a.block_col_idx,
                 static_cast<const __nv_bfloat16 *>(a.block_values), static_cast<const __nv_bfloat16 *>(a.B),
                 static_cast<__nv_bfloat16 *>(a.C));
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
  if (bsr_chain_sums(a) && reinterpret_cast<uintptr_t>(a.C) % 16 == 0)  // 64 columns and more, all aligned
    return launch_mma<BS, BS == 32 ? 2 : 4, BS == 32 ? 4 : 8, true, true>(a, sm_count, s);
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
