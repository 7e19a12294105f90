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

// Asks for the tile that starts at column X and row Y of five arrays to be brought into L2:
// the lanes of a warp take the arrays' 128-byte lines of one row (pitch and rows are
// multiples of a line).
template <typename T, int TH, int NW>
__device__ __forceinline__ void prefetch_tile(const T* const (&arr)[5], int X, int Y, int ny, int pitch, int warp, int lane) {
  constexpr int PER = 128 / (int)sizeof(T), LINES = TBW / PER + 1;  // a tile row starts anywhere in a line
  static_assert(5 * LINES <= 32, "one lane a line");
  const int a = lane / LINES, col = (max(X, 0) & ~(PER - 1)) + (lane - a * LINES) * PER;
  if (a >= 5 || col >= pitch) return;
  const T* p = a == 0 ? arr[0] : a == 1 ? arr[1] : a == 2 ? arr[2] : a == 3 ? arr[3] : arr[4];
  for (int r = warp; r < TH; r += NW) {
    const int y = Y + r;
    if (y >= 0 && y < ny) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + (long long)y * pitch + col));
  }
}

// Blocks between a tile and the one to prefetch, where the arrays do not stay in L2 from one
// launch to the next (and there is more than one such distance); 0: no prefetch. The distance
// is a wave of two blocks an SM, the large float tiles' (64 designs of 600 x 400: forward
// launch 297 -> 288 us, 1500 reverse steps 98 -> 93 ms). Kernels of one block an SM
// (double, power, seven and nine reverse steps) fetch two waves ahead with it, the 64 x 32
// float tile, of three, two thirds of one; neither was tuned apart.
inline int prefetch_distance(long long bytes, long long blocks) {
  constexpr long long WAVE = 2 * 148;
  return bytes > (100LL << 20) && blocks > 2 * WAVE ? (int)WAVE : 0;
}

}  // namespace bz
