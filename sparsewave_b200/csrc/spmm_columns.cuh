// Runs of V adjacent columns held by a lane (included by spmm_kernels.cu inside namespace swb::{anonymous}).
//
// A lane's position may lie outside its row (the ends of a 16-byte quad of positions).  Loads and sums of such a
// position are predicated instructions, written as such: an `if` around them compiles to branches, which cost four
// times the instructions of the work itself.
#pragma once

template <int V> struct Columns { float f[V]; };

template <int V>
__device__ __forceinline__ void load_if(Columns<V> &b, const void *p, int k, int n);
template <>
__device__ __forceinline__ void load_if<1>(Columns<1> &b, const void *p, int k, int n) {
  asm("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %2, %3;\n\t@p ld.global.nc.f32 %0, [%1];\n\t}"
      : "=f"(b.f[0]) : "l"(p), "r"(k), "r"(n));
}
template <>
__device__ __forceinline__ void load_if<2>(Columns<2> &b, const void *p, int k, int n) {
  asm("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %3, %4;\n\t@p ld.global.nc.v2.f32 {%0, %1}, [%2];\n\t}"
      : "=f"(b.f[0]), "=f"(b.f[1]) : "l"(p), "r"(k), "r"(n));
}
template <>
__device__ __forceinline__ void load_if<4>(Columns<4> &b, const void *p, int k, int n) {
  asm("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %5, %6;\n\t@p ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
      : "=f"(b.f[0]), "=f"(b.f[1]), "=f"(b.f[2]), "=f"(b.f[3]) : "l"(p), "r"(k), "r"(n));
}

// acc += v * b where k < n: the product is rounded on its own, like everywhere in this library.
template <int V>
__device__ __forceinline__ void add_if(Columns<V> &acc, float v, const Columns<V> &b, int k, int n) {
#pragma unroll
  for (int j = 0; j < V; ++j)
    asm("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %2, %3;\n\t@p add.rn.f32 %0, %0, %1;\n\t}"
        : "+f"(acc.f[j]) : "f"(mul(v, b.f[j])), "r"(k), "r"(n));
}

template <int V>
__device__ __forceinline__ void store_columns(float *p, const Columns<V> &a);
template <>
__device__ __forceinline__ void store_columns<1>(float *p, const Columns<1> &a) { *p = a.f[0]; }
template <>
__device__ __forceinline__ void store_columns<2>(float *p, const Columns<2> &a) {
  *reinterpret_cast<float2 *>(p) = make_float2(a.f[0], a.f[1]);
}
template <>
__device__ __forceinline__ void store_columns<4>(float *p, const Columns<4> &a) {
  *reinterpret_cast<float4 *>(p) = make_float4(a.f[0], a.f[1], a.f[2], a.f[3]);
}
