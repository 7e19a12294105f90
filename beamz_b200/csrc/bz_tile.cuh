// Parts shared by the temporally blocked 2D kernels (forward steps and their adjoint):
// tiles of 64 columns whose lanes own two adjacent columns as one packed operand.
#pragma once

#include "bz_stencil.cuh"

namespace bz {

constexpr unsigned FULL = 0xffffffffu;
constexpr int TBW = 64;  // tile columns

// Pairs of neighbouring cells: float pairs stay packed in one 64-bit register through the
// whole launch (unpacking and packing again would cost more than the arithmetic).
typedef unsigned long long f32pair;
template <typename T>
struct PairOf;
template <>
struct PairOf<float> {
  typedef f32pair type;
};
template <>
struct PairOf<double> {
  typedef double2 type;
};

__device__ __forceinline__ f32pair mk2(float a, float b) {
  f32pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float lo2(f32pair v) {
  return __uint_as_float((unsigned)v);
}
__device__ __forceinline__ float hi2(f32pair v) {
  return __uint_as_float((unsigned)(v >> 32));
}
__device__ __forceinline__ f32pair mul2(f32pair a, f32pair b) {
  f32pair r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32pair fma2(f32pair a, f32pair b, f32pair c) {
  f32pair r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// a - b as one fused multiply-add with -1: a single rounding, as the subtraction's
__device__ __forceinline__ f32pair sub2(f32pair a, f32pair b) { return fma2(b, mk2(-1.f, -1.f), a); }
__device__ __forceinline__ bool nonzero2(f32pair v) { return v != 0ull; }

__device__ __forceinline__ double2 mk2(double a, double b) { return make_double2(a, b); }
__device__ __forceinline__ double lo2(double2 v) { return v.x; }
__device__ __forceinline__ double hi2(double2 v) { return v.y; }
__device__ __forceinline__ double2 mul2(double2 a, double2 b) { return make_double2(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)); }
__device__ __forceinline__ double2 fma2(double2 a, double2 b, double2 c) {
  return make_double2(__fma_rn(a.x, b.x, c.x), __fma_rn(a.y, b.y, c.y));
}
__device__ __forceinline__ double2 sub2(double2 a, double2 b) { return make_double2(__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y)); }
__device__ __forceinline__ bool nonzero2(double2 v) { return v.x != 0.0 || v.y != 0.0; }

template <typename T>
__device__ __forceinline__ typename PairOf<T>::type ldg2(const T* p) {
  return __ldg(reinterpret_cast<const typename PairOf<T>::type*>(p));
}
// The same with the cells that exist (e0, e1) and arrays that may be aligned to T only.
template <typename T>
__device__ __forceinline__ typename PairOf<T>::type ld_pair(const T* p, bool e0, bool e1) {
  return mk2(e0 ? __ldg(p) : T(0), e1 ? __ldg(p + 1) : T(0));
}

// The operations of this warp's rows are one range of the sorted list; the lanes read it
// side by side (row by row, or by searching, would chain dependent loads). Calls
// f(row, column, k, single) for the first operation of each cell in columns [c0, c1) of
// the tile; single: no other operation on the cell. Returns the rows that have any.
template <typename F>
__device__ __forceinline__ unsigned scan_ops(const int* __restrict__ cells, int k0, int k1, int nx, int yb, int X0,
                                             int c0, int c1, int lane, F f) {
  unsigned rows = 0u;
  for (int k = k0 + lane; k < k1; k += 32) {
    const int c = __ldg(cells + k), prev = k > k0 ? __ldg(cells + k - 1) : -1, next = k + 1 < k1 ? __ldg(cells + k + 1) : -1;
    const int y = c / nx, x = c - y * nx;
    if (c == prev || x < c0 || x >= c1) continue;
    f(y - yb, x - X0, k, c != next);
    rows |= 1u << (y - yb);
  }
  return __reduce_or_sync(FULL, rows);
}

}  // namespace bz
