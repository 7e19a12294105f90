// 2D Ez-mode Yee time step, fused: H update, E update (PEC ring), source
// injection, optional |S|^2 accumulation, monitor sampling.
//
// Reference semantics (beamz project paths):
//   H update  beamz/simulation/backends/numpy_backend.py:34-61
//   E update  beamz/simulation/backends/numpy_backend.py:63-88
//   sources   beamz/simulation/helper.py:5-118 (applied after the E update)
//   power     beamz/simulation/helper.py:152-187
//   monitors  beamz/simulation/helper.py:245-256, beamz/devices/monitors.py:279-315
//
// Data layout: every field is [design][component][ny][pitch] with x contiguous.
// Ping-pong: the launch reads the *_in copies and writes the *_out copies, so
// blocks never see a neighbour's half-updated values. One thread owns one column
// x of a tile of RB rows and marches along y, carrying Ez(y) and the new Hy(y-1)
// in registers; Ez(y, x+1) and the new Hx(y, x-1) come from the neighbouring
// lanes by warp shuffles (warp-edge lanes read/recompute them from global
// memory). The row loop is fully unrolled so the loads of later rows issue
// before the arithmetic of earlier ones.
//
// After the tile is written, the block applies the source and monitor
// operations that fall inside it, spread over all its threads.
#include "bz_tile.cuh"

namespace bz {
namespace {

constexpr int BX = 128;  // threads (columns) per block

template <typename T>
struct Geo2D {
  int nx, ny, pitch, n_designs, n_mat;
  long long plane;  // ny * pitch
  T chx, chy, qy, inv_kd2, one;  // one = 1, kept out of the compiler's sight
};

template <typename T>
struct Ops2D {
  int n_src, src_steps;
  const int* src_row;
  const int* src_cell;
  const T* src_mul;
  const T* src_w;
  long long w_stride;
  const int* src_sig;
  const T* signals;
  int n_mon, ring_len;
  const int* mon_row;
  const int* mon_cell;
  const int* mon_point;
  T* record;
  long long rec_step0;
  int n_rec;
  T* ring;
  T* region;
  int rx0, ry0, rw, rh, n_reg;
  long long reg_step0;
};

template <typename T>
__device__ __forceinline__ double sq_pow(const T* ez, const T* hx, const T* hy, int nc) {
  // |S|^2 with Sx = -sum_c Ez*Hy, Sy = sum_c Ez*Hx (helper.py:171-179)
  double sx = 0.0, sy = 0.0;
  for (int c = 0; c < nc; ++c) {
    sx -= (double)ez[c] * (double)hy[c];
    sy += (double)ez[c] * (double)hx[c];
  }
  return sx * sx + sy * sy;
}

template <typename T, int NC, bool PWR, int RB>
__global__ void __launch_bounds__(BX) step2d_kernel(
    const T* __restrict__ ez_in, const T* __restrict__ hx_in, const T* __restrict__ hy_in,
    T* __restrict__ ez_out, T* __restrict__ hx_out, T* __restrict__ hy_out,
    const T* __restrict__ ce, const T* __restrict__ loss, double* __restrict__ pwr,
    Geo2D<T> g, Ops2D<T> o, long long step_base, const long long* __restrict__ d_step) {
  const long long step = d_step ? (__ldg(d_step) + step_base) : step_base;
  const int nx = g.nx, ny = g.ny, pitch = g.pitch;
  const int x = blockIdx.x * BX + threadIdx.x;
  const int wl = threadIdx.x & 31;
  const int d = blockIdx.z;
  const int y0 = blockIdx.y * RB;
  const int nrows = min(RB, ny - y0);
  const bool xin = x < nx;
  const long long fb = (long long)d * NC * g.plane;
  const long long mb = (g.n_mat > 1 ? (long long)d : 0LL) * g.plane;
  const T* __restrict__ cep = ce + mb;
  const T* __restrict__ lsp = loss + mb;

  T ezc[NC], hyp[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    ezc[c] = xin ? __ldg(ez_in + fb + c * g.plane + (long long)y0 * pitch + x) : T(0);
    hyp[c] = T(0);
  }
  if (y0 >= 1) {
    // New Hy(y0-1, x): needed by the E update of row y0, owned by the tile above.
    const long long r = (long long)(y0 - 1) * pitch + x;
    T fh, cx, cy;
    h_coeffs(xin ? __ldg(lsp + r) : T(0), g.chx, g.chy, fh, cx, cy);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const long long off = fb + c * g.plane + r;
      const T ezm = xin ? __ldg(ez_in + off) : T(0);
      const T hy = xin ? __ldg(hy_in + off) : T(0);
      hyp[c] = hy_update(fh, hy, cy, ezc[c], ezm);
    }
  }

#pragma unroll
  for (int i = 0; i < RB; ++i) {
    const int y = y0 + i;
    if (i < nrows) {  // uniform across the block
      const long long r = (long long)y * pitch + x;
      const T a = xin ? __ldg(lsp + r) : T(0);
      const T cec = xin ? __ldg(cep + r) : T(0);
      T fh, cx, cy;
      h_coeffs(a, g.chx, g.chy, fh, cx, cy);
      // Warp-edge lane 0 recomputes the new Hx(y, x-1) of the lane to its left.
      const bool left_fix = (wl == 0) && xin && x >= 1;
      T fhl = T(0), cxl = T(0), cyl;
      if (left_fix) h_coeffs(__ldg(lsp + r - 1), g.chx, g.chy, fhl, cxl, cyl);
      const bool interior = (x >= 1) && (x <= nx - 2) && (y >= 1) && (y <= ny - 2);
      const T fe = sub_rn(T(1), mul_rn(mul_rn(a, cec), g.inv_kd2));
      T ezo[NC], hxo[NC], hyo[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const T* __restrict__ E = ez_in + fb + c * g.plane;
        const T ezn = (xin && y + 1 < ny) ? __ldg(E + r + pitch) : T(0);
        T ezr = __shfl_down_sync(FULL, ezc[c], 1);
        if (wl == 31) ezr = (x + 1 < nx) ? __ldg(E + r + 1) : T(0);
        const T hx0 = xin ? __ldg(hx_in + fb + c * g.plane + r) : T(0);
        const T hy0 = xin ? __ldg(hy_in + fb + c * g.plane + r) : T(0);
        const T hxn = hx_update(fh, hx0, cx, ezr, ezc[c]);
        const T hyn = hy_update(fh, hy0, cy, ezn, ezc[c]);
        T hxl = __shfl_up_sync(FULL, hxn, 1);
        if (left_fix) {
          const T hxl0 = __ldg(hx_in + fb + c * g.plane + r - 1);
          hxl = hx_update(fhl, hxl0, cxl, ezc[c], __ldg(E + r - 1));
        }
        T ez_new = ezc[c];
        if (interior) ez_new = ez_update(fe, ezc[c], cec, g.qy, hxn, hxl, hyn, hyp[c]);
        ezo[c] = ez_new;
        hxo[c] = (x < nx - 1) ? hxn : T(0);
        hyo[c] = (y < ny - 1) ? hyn : T(0);
        if (xin) {
          const long long off = fb + c * g.plane + r;
          ez_out[off] = ez_new;
          if (x < nx - 1) hx_out[off] = hxn;
          if (y < ny - 1) hy_out[off] = hyn;
        }
        ezc[c] = ezn;
        hyp[c] = hyn;
      }
      if (PWR && xin) pwr[(long long)d * g.plane + r] += sq_pow<T>(ezo, hxo, hyo, NC);
      if (o.region != nullptr) {  // Ez after this step inside the capture box
        const long long slot = step + 1 - o.reg_step0;
        const int rx = x - o.rx0, ry = y - o.ry0;
        if (slot >= 1 && slot < o.n_reg && rx >= 0 && rx < o.rw && ry >= 0 && ry < o.rh) {
#pragma unroll
          for (int c = 0; c < NC; ++c)
            o.region[(((slot * g.n_designs + d) * NC + c) * o.rh + ry) * (long long)o.rw + rx] = ezo[c];
        }
      }
    }
  }

  if (o.n_src == 0 && o.n_mon == 0) return;  // uniform across the grid
  // ---- post phase: operations on cells of this block's tile -----------------
  __shared__ int s_k0[RB], s_pre[RB + 1];
  const int xlo = blockIdx.x * BX;
  const int xhi = min(xlo + BX, nx);
  __syncthreads();  // this block's field writes are now visible to all its threads
  if (o.n_src > 0) {
    const int total = block_op_ranges(o.src_row, o.src_cell, y0, nrows, nx, xlo, xhi, s_k0, s_pre);
    for (int i = threadIdx.x; i < total; i += BX) {
      int t;
      const int k = op_at(i, nrows, s_k0, s_pre, t);
      const int cell = __ldg(o.src_cell + k);
      if (i > s_pre[t] && __ldg(o.src_cell + k - 1) == cell) continue;  // not first of its cell's run
      const int y = y0 + t;
      const long long rr = (long long)y * pitch + (cell - y * nx);
      T e[NC], hx[NC], hy[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        e[c] = ez_out[fb + c * g.plane + rr];
        hx[c] = hx_out[fb + c * g.plane + rr];
        hy[c] = hy_out[fb + c * g.plane + rr];
      }
      double p_old = 0.0;
      if (PWR) p_old = sq_pow<T>(e, hx, hy, NC);
      for (int kk = k; kk < o.n_src && __ldg(o.src_cell + kk) == cell; ++kk) {
        const T m = __ldg(o.src_mul + kk);
        const int sg = __ldg(o.src_sig + kk);
        const T s = (step < o.src_steps) ? __ldg(o.signals + (long long)sg * o.src_steps + step) : T(0);
#pragma unroll
        for (int c = 0; c < NC; ++c) e[c] = fma_rn(m, e[c], mul_rn(__ldg(o.src_w + d * o.w_stride + (long long)kk * NC + c), s));
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) ez_out[fb + c * g.plane + rr] = e[c];
      if (PWR) {
        double* pp = pwr + (long long)d * g.plane + rr;
        *pp = (*pp - p_old) + sq_pow<T>(e, hx, hy, NC);
      }
    }
    __syncthreads();
  }
  if (o.n_mon > 0) {
    const int total = block_op_ranges(o.mon_row, o.mon_cell, y0, nrows, nx, xlo, xhi, s_k0, s_pre);
    const bool rec = o.record != nullptr && step >= o.rec_step0 && step < o.rec_step0 + o.n_rec;
    const long long slot = o.ring != nullptr ? step % o.ring_len : 0;
    for (int i = threadIdx.x; i < total; i += BX) {
      int t;
      const int k = op_at(i, nrows, s_k0, s_pre, t);
      const int cell = __ldg(o.mon_cell + k);
      const int p = __ldg(o.mon_point + k);
      const int y = y0 + t;
      const int xx = cell - y * nx;
      const long long rr = (long long)y * pitch + xx;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const long long off = fb + c * g.plane + rr;
        const T ez = ez_out[off];
        const T hx = hx_out[off];
        const T hy = hy_out[off];
        if (rec) {
          T* dst = o.record + ((((step - o.rec_step0) * g.n_designs + d) * NC + c) * (long long)o.n_mon + p) * 3;
          dst[0] = ez;
          dst[1] = hx;
          dst[2] = hy;
        }
        if (o.ring) {
          // The new Hx(x-1) and Hy(y-1) may belong to another block of this launch, so
          // they are recomputed from the step's inputs (same arithmetic as their owner).
          const T* __restrict__ E = ez_in + fb + c * g.plane;
          T hxl = T(0), hyu = T(0);
          if (xx >= 1) {
            T fh, cx, cy;
            h_coeffs(__ldg(lsp + rr - 1), g.chx, g.chy, fh, cx, cy);
            hxl = hx_update(fh, __ldg(hx_in + off - 1), cx, __ldg(E + rr), __ldg(E + rr - 1));
          }
          if (y >= 1) {
            T fh, cx, cy;
            h_coeffs(__ldg(lsp + rr - pitch), g.chx, g.chy, fh, cx, cy);
            hyu = hy_update(fh, __ldg(hy_in + off - pitch), cy, __ldg(E + rr), __ldg(E + rr - pitch));
          }
          T* q = o.ring + (((slot * g.n_designs + d) * NC + c) * (long long)o.n_mon + p) * 5;
          q[0] = ez;
          q[1] = hx;
          q[2] = hxl;
          q[3] = hy;
          q[4] = hyu;
        }
      }
    }
  }
}

// ---- temporal blocking ---------------------------------------------------------
// step2d_tb_kernel advances TS (odd) steps per launch. A block holds a tile of 64
// columns x NW*R rows in registers: lane l of warp w owns columns X0+2l, X0+2l+1 of
// rows Y0+w*R .. Y0+w*R+R-1. Each sub-step is the single-step update restricted to
// the tile; the values next to the tile's edges go stale by one cell per sub-step, so
// after TS sub-steps the tile minus a halo (TS+1 columns, TS rows a side) is exact, and
// only it is stored. Reads copy (step & 1) and writes the other, like TS single steps.
//
// What bounds it is issue and latency, not memory (the grid stays in L2 for TS steps):
//  * The two columns of a lane are one packed operand (add/mul/fma.f32x2: the same
//    rounding per element), one shuffle a row and field moves the x neighbour.
//  * A tile without loss and off the grid's edge (most tiles) needs no factor but ce
//    (fh = fe = 1 exactly), so a cell costs four registers and two blocks share an SM:
//    one loads while the other computes. Other tiles keep fh, cx, cy and fe in shared
//    memory.
//  * One block barrier a sub-step: a warp receives Ez of the rows above and below it
//    and carries the new Hy of the row above itself (one redundant row of updates).
//  * Every lane looks up its own cells' operations (a shared-memory map filled once per
//    launch), so the points of a line along x are handled by the lanes in parallel.
// Components of a complex field are independent real fields (real coefficients) and
// run as separate blocks.
//
// Measured against the same tile with five factors a cell in registers, two barriers a
// sub-step and the operations walked one by one (us a launch, before -> after): 2000 x
// 1000 cells with a line source and three lines of points, 7 steps, 57.5 -> 35.0; 400 x
// 400 with four recorded edge lines, 9 steps, 49.3 -> 16.5; two components of 1000 x 501,
// 7 steps, 34.9 -> 26.7; 64 designs of 600 x 400, 7 steps, 481 -> 297; float64 601 x 397,
// 9 steps, 32.9 -> 25.1. A sub-step of two co-resident tiles clear of loss takes about
// 900 cycles, of which the packed arithmetic fills about 730; the tile's loads take 3000
// to 6000 cycles a launch. Measured slower: all shuffles of a pass ahead of its
// arithmetic (1070 cycles; more registers live), x differences as single subtractions
// instead of packed ones (1150).
template <typename T>
__device__ __forceinline__ void put3(T* p, T a, T b, T c) {
  p[0] = a;
  p[1] = b;
  p[2] = c;
}
template <typename T>
__device__ __forceinline__ void put5(T* p, T a, T b, T c, T d, T e) {
  p[0] = a;
  p[1] = b;
  p[2] = c;
  p[3] = d;
  p[4] = e;
}

// Shared memory of a block: factors of the tiles that need them, the rows exchanged
// between warps (two buffers), per cell the operation on it, and the operations' values.
constexpr int TB_POOL = 160;  // source operations of a tile held on chip; further ones are read from memory
constexpr int TB_REC = 256;     // pairs of cells staged for monitor points each sub-step
constexpr int TB_POINTS = 256;  // monitor points of a tile written from the staged cells
template <typename T, int TS, int R, int NW>
struct TbSmem {
  static constexpr int TH = NW * R;
  static constexpr int FAC = 4 * TH * TBW * (int)sizeof(T);
  static constexpr int EXCH = 2 * 2 * NW * TBW * (int)sizeof(T);
  static constexpr int POOL = (TS + 1) * TB_POOL * (int)sizeof(T);
  static constexpr int MAP = TH * TBW * (int)sizeof(short);
  static constexpr int REC = 2 * TB_REC * 10 * (int)sizeof(T);
  static constexpr int LIST = 2 * TB_POINTS * (int)sizeof(int);
  static constexpr int BYTES = FAC + EXCH + POOL + REC + LIST + MAP + 16;
};

template <typename T, int TS, int R, int NW, int MINB, bool PWR>
__global__ void __launch_bounds__(32 * NW, MINB) step2d_tb_kernel(
    const T* __restrict__ ez_in, const T* __restrict__ hx_in, const T* __restrict__ hy_in,
    T* __restrict__ ez_out, T* __restrict__ hx_out, T* __restrict__ hy_out,
    const T* __restrict__ ce, const T* __restrict__ loss, double* __restrict__ pwr, Geo2D<T> g, Ops2D<T> o,
    int n_comp, int plane0,
    int n_planes, int ahead, bool vec, long long step_base, const long long* __restrict__ d_step) {
  typedef typename PairOf<T>::type V;
  typedef TbSmem<T, TS, R, NW> S;
  constexpr int TH = S::TH, HX = TS + 1;
  constexpr int OW = TBW - 2 * HX, OH = TH - 2 * TS;
  static_assert(TS % 2 == 1 && OW > 0 && OH > 0 && R <= 16, "bad temporal tile");
  extern __shared__ __align__(16) unsigned char tb_smem[];
  V* s_fac = reinterpret_cast<V*>(tb_smem);                              // [4][TH][32]: fh, -cx, cy, fe
  V* s_ex = reinterpret_cast<V*>(tb_smem + S::FAC);                      // [2][2][NW][32]: first, last rows' Ez
  T* s_pool = reinterpret_cast<T*>(tb_smem + S::FAC + S::EXCH);          // [TS + 1][TB_POOL]: addends, factor
  T* s_rec = s_pool + (TS + 1) * TB_POOL;                                // [2][TB_REC][10]: staged cells
  int2* s_list = reinterpret_cast<int2*>(tb_smem + S::FAC + S::EXCH + S::POOL + S::REC);  // (staged cell, point)
  int* s_used = reinterpret_cast<int*>(s_list + TB_POINTS);              // slots taken: sources, points, staged cells
  short* s_map = reinterpret_cast<short*>(s_used + 4);                   // [TH][64]: sources

  const long long step0 = d_step ? (__ldg(d_step) + step_base) : step_base;
  const int nx = g.nx, ny = g.ny, pitch = g.pitch;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int dc = plane0 + blockIdx.z, d = dc / n_comp, comp = dc - d * n_comp;  // one component per block
  const int X0 = (int)blockIdx.x * OW - HX, Y0 = (int)blockIdx.y * OH - TS;
  const int yb = Y0 + w * R, xa = X0 + 2 * lane, tr0 = w * R;
  const long long fb = (long long)dc * g.plane + (long long)yb * pitch + xa;  // the thread's first cell
  const long long mb = (g.n_mat > 1 ? (long long)d : 0LL) * g.plane + (long long)yb * pitch + xa;
  // tiles whose every cell is an interior one of the grid skip all bounds
  const bool inner = X0 >= 1 && X0 + TBW - 1 <= nx - 2 && Y0 >= 1 && Y0 + TH - 1 <= ny - 2;

  // the operations' list ranges first: their latency overlaps the tile's loads
  int sk0 = 0, sk1 = 0, mk0 = 0, mk1 = 0;
  const int mlo = max(Y0 + TS, max(yb, 0)), mhi = min(min(Y0 + TH - TS, ny), yb + R);
  if (o.n_src > 0 && max(yb, 0) < min(yb + R, ny)) {
    sk0 = __ldg(o.src_row + max(yb, 0));
    sk1 = __ldg(o.src_row + min(yb + R, ny));
  }
  if (o.n_mon > 0 && mlo < mhi) {
    mk0 = __ldg(o.mon_row + mlo);
    mk1 = __ldg(o.mon_row + mhi);
  }
  if (threadIdx.x < 3) s_used[threadIdx.x] = 0;

  V ez[R], hx[R], hy[R], cc[R], ls[R];
  V hyu;  // Hy of the row above the warp's first; stale, as all halo rows, for warp 0
  if (inner && vec) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = i * pitch;
      ls[i] = ldg2(loss + mb + r);
      ez[i] = ldg2(ez_in + fb + r);
      hx[i] = ldg2(hx_in + fb + r);
      hy[i] = ldg2(hy_in + fb + r);
      cc[i] = ldg2(ce + mb + r);
    }
    hyu = ldg2(hy_in + fb - pitch);  // inside the grid also for warp 0, whose copy is never used as exact
  } else {
    const bool in0 = xa >= 0 && xa < nx, in1 = xa >= 0 && xa + 1 < nx;
    const bool inm0 = in0 && xa < nx - 1, inm1 = in1 && xa + 1 < nx - 1;  // columns of Hx
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int y = yb + i, r = i * pitch;
      const bool iny = y >= 0 && y < ny, inh = y >= 0 && y < ny - 1;
      ls[i] = ld_pair(loss + mb + r, in0 && iny, in1 && iny);
      ez[i] = ld_pair(ez_in + fb + r, in0 && iny, in1 && iny);
      hx[i] = ld_pair(hx_in + fb + r, inm0 && iny, inm1 && iny);
      hy[i] = ld_pair(hy_in + fb + r, in0 && inh, in1 && inh);
      cc[i] = ld_pair(ce + mb + r, in0 && iny, in1 && iny);
    }
    hyu = ld_pair(hy_in + fb - pitch, in0 && yb >= 1 && yb < ny, in1 && yb >= 1 && yb < ny);
  }
  if (ahead > 0) {  // the tile that a block of the next wave will load
    const long long next = ((long long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x + ahead;
    const int bz = (int)(next / ((long long)gridDim.x * gridDim.y));
    if (bz < (int)gridDim.z) {
      const int rem = (int)(next - (long long)bz * gridDim.x * gridDim.y), by = rem / (int)gridDim.x, bx = rem - by * (int)gridDim.x;
      const long long pf = (long long)(plane0 + bz) * g.plane;
      const long long pm = (g.n_mat > 1 ? (long long)((plane0 + bz) / n_comp) : 0LL) * g.plane;
      const T* const arr[5] = {ez_in + pf, hx_in + pf, hy_in + pf, ce + pm, loss + pm};
      prefetch_tile<T, TH, NW>(arr, bx * OW - HX, by * OH - TS, ny, pitch, w, lane);
    }
  }
  __syncthreads();  // the pools' counters are set

  // Sources act on every tile cell (halo cells evolve like the real ones). A cell's map
  // entry is the pool slot of its only operation, -1 for none, -2 - n for several (or no
  // slot left), found from the warp's n-th list entry on.
  unsigned src_rows = 0u, mon_rows = 0u, mon_lanes = 0u;
  bool src_many = false, mon_staged = false, mon_direct = false;
  int rec0 = 0;  // the warp's first staged pair
  short* const w_src = s_map + tr0 * TBW;
  if (sk0 < sk1) {
    for (int i = lane; i < R * TBW; i += 32) w_src[i] = -1;
    __syncwarp();
    src_rows = scan_ops(o.src_cell, sk0, sk1, nx, yb, X0, max(X0, 0), min(X0 + TBW, nx), lane,
                        [&](int i, int col, int k, bool single) {
      int slot = single ? atomicAdd(s_used, 1) : TB_POOL;
      if (slot < TB_POOL) {
        const T wv = __ldg(o.src_w + d * o.w_stride + (long long)k * n_comp + comp);
        const T* sg = o.signals + (long long)__ldg(o.src_sig + k) * o.src_steps + step0;
        s_pool[TS * TB_POOL + slot] = __ldg(o.src_mul + k);
#pragma unroll
        for (int s = 0; s < TS; ++s)
          s_pool[s * TB_POOL + slot] = mul_rn(wv, step0 + s < o.src_steps ? __ldg(sg + s) : T(0));
      } else {
        slot = -2 - min(k - sk0, 32000);
        src_many = true;
      }
      w_src[i * TBW + col] = (short)slot;
    });
  }
  // Monitors sample owned cells: the warp stages the lanes x rows that hold its points each
  // sub-step (record 10 values a pair of cells), and the block writes the points from there.
  // A warp whose points spread over more cells than it can stage (a tile crossed by eight or
  // more adjacent lines) writes row by row: every lane searches the row's points for its two
  // cells. (400 x 400 cells, 9 steps a launch, us a step, walking the warp's whole list for each
  // row -> searching: 8 adjacent lines 470 -> 8.6, 64 lines 529 -> 12.3, 16 lines along y 30.8 ->
  // 7.2; 4 lines, staged, 2.6. A map of the cells' first points in the staged cells' place takes
  // 5.0, 6.3 and 3.3, but 64 x 64 tiles that never use it ran 3 to 14 % slower beside that code.)
  if (mk0 < mk1) {
    const int c0 = X0 + HX, c1 = min(X0 + TBW - HX, nx);
    for (int k = mk0 + lane; k < mk1; k += 32) {
      const int c = __ldg(o.mon_cell + k), y = c / nx, x = c - y * nx;
      if (x < c0 || x >= c1) continue;
      mon_rows |= 1u << (y - yb);
      mon_lanes |= 1u << ((x - X0) >> 1);
    }
    mon_rows = __reduce_or_sync(FULL, mon_rows);
    mon_lanes = __reduce_or_sync(FULL, mon_lanes);
    const int n_rec = __popc(mon_rows) * __popc(mon_lanes);
    if (lane == 0 && n_rec > 0) rec0 = atomicAdd(s_used + 2, n_rec);
    rec0 = __shfl_sync(FULL, rec0, 0);
    mon_staged = n_rec > 0 && rec0 + n_rec <= TB_REC;
    mon_direct = n_rec > 0 && !mon_staged;
    for (int k = mk0 + lane; k < mk1 && mon_staged; k += 32) {
      const int c = __ldg(o.mon_cell + k), y = c / nx, x = c - y * nx;
      if (x < c0 || x >= c1) continue;
      const int slot = atomicAdd(s_used + 1, 1), ln = (x - X0) >> 1;
      const int rec = __popc(mon_rows & ((1u << (y - yb)) - 1u)) * __popc(mon_lanes) + __popc(mon_lanes & ((1u << ln) - 1u));
      if (slot < TB_POINTS) s_list[slot] = make_int2((rec0 + rec) * 10 + ((x - X0) & 1), __ldg(o.mon_point + k));
      else mon_direct = true;  // the list is full: the warp's points are also written row by row
    }
    mon_direct = __any_sync(FULL, mon_direct);
  }
  src_many = __any_sync(FULL, src_many);
  const bool own = lane >= HX / 2 && lane < 32 - HX / 2 && xa < nx;
  // owned cells inside the capture box: bit 2*i + column
  unsigned cap = 0u;
  if (o.region != nullptr && own) {
    const int rx = xa - o.rx0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int tr = tr0 + i, y = yb + i, ry = y - o.ry0;
      if (tr < TS || tr >= TH - TS || y >= ny || ry < 0 || ry >= o.rh) continue;
      if (rx >= 0 && rx < o.rw) cap |= 1u << (2 * i);
      if (xa + 1 < nx && rx + 1 >= 0 && rx + 1 < o.rw) cap |= 2u << (2 * i);
    }
  }

  // |S|^2 sums of the owned cells (one component), added to every sub-step in step order
  double pw[PWR ? R : 1][2];
  if (PWR && own) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int tr = tr0 + i;
      const bool in = tr >= TS && tr < TH - TS && yb + i < ny;
      pw[i][0] = in ? pwr[fb + i * pitch] : 0.0;
      pw[i][1] = in && xa + 1 < nx ? pwr[fb + i * pitch + 1] : 0.0;
    }
  }

  // Factors, where any tile cell has loss or lies on or outside the grid's edge. Cells
  // whose H or E the reference never changes (Hx in the last column, Hy in the last
  // row, E on the PEC ring, everything outside) get factors that keep the value.
  bool lossy = !inner;
#pragma unroll
  for (int i = 0; i < R; ++i) lossy = lossy || nonzero2(ls[i]);
  lossy = __syncthreads_or(lossy);
  if (lossy) {
    const bool in0 = xa >= 0 && xa < nx, in1 = xa >= 0 && xa + 1 < nx;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int y = yb + i;
      const bool iny = y >= 0 && y < ny, inh = y >= 0 && y < ny - 1, inty = y >= 1 && y <= ny - 2;
      const bool i0 = inty && xa >= 1 && xa <= nx - 2, i1 = inty && xa + 1 >= 1 && xa + 1 <= nx - 2;
      T fh0, fh1, cx0, cx1, cy0, cy1;
      h_coeffs(lo2(ls[i]), g.chx, g.chy, fh0, cx0, cy0);
      h_coeffs(hi2(ls[i]), g.chx, g.chy, fh1, cx1, cy1);
      const T fe0 = i0 ? sub_rn(T(1), mul_rn(mul_rn(lo2(ls[i]), lo2(cc[i])), g.inv_kd2)) : T(1);
      const T fe1 = i1 ? sub_rn(T(1), mul_rn(mul_rn(hi2(ls[i]), hi2(cc[i])), g.inv_kd2)) : T(1);
      cc[i] = mk2(i0 ? lo2(cc[i]) : T(0), i1 ? hi2(cc[i]) : T(0));
      V* q = s_fac + (tr0 + i) * 32 + lane;
      q[0] = mk2(fh0, fh1);
      q[TH * 32] = mk2(iny && in0 && xa < nx - 1 ? -cx0 : T(0), iny && in1 && xa + 1 < nx - 1 ? -cx1 : T(0));
      q[2 * TH * 32] = mk2(inh && in0 ? cy0 : T(0), inh && in1 ? cy1 : T(0));
      q[3 * TH * 32] = mk2(fe0, fe1);
    }
  }
  // one = 1 in a register the compiler cannot see through: x + y as fma(1, x, y), so that a
  // product y is rounded before the sum, as in every other kernel of this update
  const V one = mk2(g.one, g.one), mcx = mk2(-g.chx, -g.chx), pcy = mk2(g.chy, g.chy), qy = mk2(g.qy, g.qy);
  const V zero = mk2(T(0), T(0));
  const int n_list = min(s_used[1], TB_POINTS);  // after the barrier above: every warp has added its points
  int ring_slot = o.n_mon > 0 && o.ring ? (int)(step0 % o.ring_len) : 0;  // of step0, then of each sub-step
  // Writes point p of the cell at q (pairs of Ez, Hx, Hy, Hy of the row above; Hx left of the
  // pair) to the record and the DFT ring.
  auto write_point = [&](const T* q, int j, long long p, long long step, int slot) {
    if (o.record != nullptr && step >= o.rec_step0 && step < o.rec_step0 + o.n_rec)
      put3(o.record + (((step - o.rec_step0) * n_planes + dc) * o.n_mon + p) * 3, q[j], q[2 + j], q[4 + j]);
    if (o.ring)
      put5(o.ring + (((long long)slot * n_planes + dc) * o.n_mon + p) * 5, q[j], q[2 + j], j ? q[2] : q[8], q[4 + j],
           q[6 + j]);
  };
  auto write_list = [&](int s) {  // the staged points of sub-step s, one a thread
    const T* q = s_rec + (s & 1) * TB_REC * 10;
    for (int i = threadIdx.x; i < n_list; i += 32 * NW) {
      const int2 e = s_list[i];
      const int j = e.x & 1;
      write_point(q + e.x - j, j, e.y, step0 + s, ring_slot);
    }
  };

#pragma unroll 1
  for (int s = 0; s < TS; ++s) {
    V* ex = s_ex + (s & 1) * (2 * NW * 32) + lane;
    ex[w * 32] = ez[0];
    ex[(NW + w) * 32] = ez[R - 1];
    __syncthreads();  // also orders the factors before their first use, and the staged samples
    if (n_list > 0 && s > 0) write_list(s - 1);
    if (s > 0 && ++ring_slot == o.ring_len) ring_slot = 0;  // now the slot of sub-step s
    const V ez_dn = w + 1 < NW ? ex[(w + 1) * 32] : zero;
    const V ez_up = w > 0 ? ex[(NW + w - 1) * 32] : zero;
    V hu;  // new Hy of the row above the current one
    if (!lossy) {
      hyu = fma2(one, hyu, mul2(pcy, sub2(ez[0], ez_up)));
      hu = hyu;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const V down = i + 1 < R ? ez[i + 1 < R ? i + 1 : i] : ez_dn;
        const V er = mk2(hi2(ez[i]), __shfl_down_sync(FULL, lo2(ez[i]), 1));  // lane 31: stale halo
        hx[i] = fma2(one, hx[i], mul2(mcx, sub2(er, ez[i])));
        hy[i] = fma2(one, hy[i], mul2(pcy, sub2(down, ez[i])));
        const V hl = mk2(__shfl_up_sync(FULL, hi2(hx[i]), 1), lo2(hx[i]));  // lane 0: stale halo
        ez[i] = fma2(one, ez[i], mul2(cc[i], fma2(qy, sub2(hy[i], hu), sub2(hl, hx[i]))));
        hu = hy[i];
      }
    } else {
      const V* q = s_fac + tr0 * 32 + lane;
      if (w > 0) hyu = fma2(q[-32], hyu, mul2(q[2 * TH * 32 - 32], sub2(ez[0], ez_up)));
      hu = hyu;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const V fh = q[i * 32], cx = q[(TH + i) * 32], cy = q[(2 * TH + i) * 32], fe = q[(3 * TH + i) * 32];
        const V down = i + 1 < R ? ez[i + 1 < R ? i + 1 : i] : ez_dn;
        const V er = mk2(hi2(ez[i]), __shfl_down_sync(FULL, lo2(ez[i]), 1));
        hx[i] = fma2(fh, hx[i], mul2(cx, sub2(er, ez[i])));
        hy[i] = fma2(fh, hy[i], mul2(cy, sub2(down, ez[i])));
        const V hl = mk2(__shfl_up_sync(FULL, hi2(hx[i]), 1), lo2(hx[i]));
        ez[i] = fma2(fe, ez[i], mul2(cc[i], fma2(qy, sub2(hy[i], hu), sub2(hl, hx[i]))));
        hu = hy[i];
      }
    }
    if (!PWR && !(src_rows | mon_rows | cap)) continue;
    const long long step = step0 + s;
    // Sources (helper.py:5-118), in operation order per cell
    if (src_rows) {
      const T* add = s_pool + s * TB_POOL;
      const T* fac = s_pool + TS * TB_POOL;
#pragma unroll
      for (int i = 0; i < R; ++i) {  // no branches: rows without sources have empty maps
        const short2 e = *reinterpret_cast<const short2*>(w_src + i * TBW + 2 * lane);
        const int e0 = max((int)e.x, 0), e1 = max((int)e.y, 0);
        const T v0 = lo2(ez[i]), v1 = hi2(ez[i]);
        const T n0 = fma_rn(fac[e0], v0, add[e0]), n1 = fma_rn(fac[e1], v1, add[e1]);
        ez[i] = mk2(e.x >= 0 ? n0 : v0, e.y >= 0 ? n1 : v1);
      }
      if (src_many) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
          if (!(src_rows & (1u << i))) continue;
          T v[2] = {lo2(ez[i]), hi2(ez[i])};
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int e = w_src[i * TBW + 2 * lane + j], cell = (yb + i) * nx + xa + j;
            if (e >= -1) continue;
            int k = sk0 + (-2 - e);
            while (__ldg(o.src_cell + k) != cell) ++k;
            do {
              const T sv = step < o.src_steps ? __ldg(o.signals + (long long)__ldg(o.src_sig + k) * o.src_steps + step) : T(0);
              v[j] = fma_rn(__ldg(o.src_mul + k), v[j],
                            mul_rn(__ldg(o.src_w + d * o.w_stride + (long long)k * n_comp + comp), sv));
              ++k;
            } while (k < sk1 && __ldg(o.src_cell + k) == cell);
          }
          ez[i] = mk2(v[0], v[1]);
        }
      }
    }
    if (PWR) {
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const T e[2] = {lo2(ez[i]), hi2(ez[i])}, h0[2] = {lo2(hx[i]), hi2(hx[i])}, h1[2] = {lo2(hy[i]), hi2(hy[i])};
#pragma unroll
        for (int j = 0; j < 2; ++j) pw[i][j] += sq_pow<T>(e + j, h0 + j, h1 + j, 1);
      }
    }
    // Ez after this sub-step inside the capture box (the box holds no sources)
    if (cap) {
      const long long slot = step + 1 - o.reg_step0;
      if (slot >= 1 && slot < o.n_reg) {
        T* q = o.region + ((slot * n_planes + dc) * o.rh + (yb - o.ry0)) * (long long)o.rw + (xa - o.rx0);
#pragma unroll
        for (int i = 0; i < R; ++i) {
          if (cap & (1u << (2 * i))) q[i * o.rw] = lo2(ez[i]);
          if (cap & (2u << (2 * i))) q[i * o.rw + 1] = hi2(ez[i]);
        }
      }
    }
    // Monitor samples of owned cells, with Hx left of each pair
    if (mon_rows) {
      T side[R];
#pragma unroll
      for (int i = 0; i < R; ++i) side[i] = __shfl_up_sync(FULL, hi2(hx[i]), 1);
      if (mon_staged && (mon_lanes >> lane & 1u)) {
        T* q = s_rec + ((s & 1) * TB_REC + rec0 + __popc(mon_lanes & ((1u << lane) - 1u))) * 10;
#pragma unroll
        for (int i = 0; i < R; ++i) {
          if (!(mon_rows & (1u << i))) continue;  // uniform across the warp
          V* v = reinterpret_cast<V*>(q);
          v[0] = ez[i];
          v[1] = hx[i];
          v[2] = hy[i];
          v[3] = yb + i < 1 ? zero : (i > 0 ? hy[i > 0 ? i - 1 : 0] : hyu);
          q[8] = xa >= 1 ? side[i] : T(0);
          q += __popc(mon_lanes) * 10;
        }
      }
      if (mon_direct) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
          if (!(mon_rows & (1u << i))) continue;
          const V up = yb + i < 1 ? zero : (i > 0 ? hy[i > 0 ? i - 1 : 0] : hyu);
          const T hl = xa >= 1 ? side[i] : T(0);
          const int base = (yb + i) * nx;
          int k = mk1, k1 = mk1;
          if (own) {  // the owner writes
            k1 = __ldg(o.mon_row + yb + i + 1);
            k = lower_bound_i(o.mon_cell, __ldg(o.mon_row + yb + i), k1, base + xa);
          }
          for (; k < k1; ++k) {
            const int x = __ldg(o.mon_cell + k) - base;
            if (x > xa + 1) break;
            const T q[9] = {lo2(ez[i]), hi2(ez[i]), lo2(hx[i]), hi2(hx[i]), lo2(hy[i]), hi2(hy[i]), lo2(up), hi2(up), hl};
            if (x == xa) write_point(q, 0, __ldg(o.mon_point + k), step, ring_slot);
            else write_point(q, 1, __ldg(o.mon_point + k), step, ring_slot);
          }
        }
      }
    }
  }
  if (n_list > 0) {  // uniform across the block
    __syncthreads();
    write_list(TS - 1);
  }
  // Store the owned box
  if (!own) return;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int tr = tr0 + i, y = yb + i;
    if (tr < TS || tr >= TH - TS || y >= ny) continue;
    const long long off = fb + i * pitch;
    if (PWR) {
      pwr[off] = pw[i][0];
      if (xa + 1 < nx) pwr[off + 1] = pw[i][1];
    }
    if (vec && xa + 1 < nx - 1) {  // both columns exist in every component
      *reinterpret_cast<V*>(ez_out + off) = ez[i];
      *reinterpret_cast<V*>(hx_out + off) = hx[i];
      if (y < ny - 1) *reinterpret_cast<V*>(hy_out + off) = hy[i];
    } else {
      const bool in1 = xa + 1 < nx;
      ez_out[off] = lo2(ez[i]);
      if (in1) ez_out[off + 1] = hi2(ez[i]);
      if (xa < nx - 1) hx_out[off] = lo2(hx[i]);
      if (xa + 1 < nx - 1) hx_out[off + 1] = hi2(hx[i]);
      if (y < ny - 1) {
        hy_out[off] = lo2(hy[i]);
        if (in1) hy_out[off + 1] = hi2(hy[i]);
      }
    }
  }
}

template <typename T>
Geo2D<T> make_geo(const bz_grid2d* gd) {
  Geo2D<T> g;
  g.nx = gd->nx;
  g.ny = gd->ny;
  g.pitch = gd->pitch;
  g.n_designs = gd->n_designs;
  g.n_mat = gd->n_mat;
  g.plane = (long long)gd->ny * gd->pitch;
  g.chx = (T)gd->chx;
  g.chy = (T)gd->chy;
  g.qy = (T)gd->qy;
  g.inv_kd2 = (T)gd->inv_kd2;
  g.one = (T)1;
  return g;
}

template <typename T>
Ops2D<T> make_ops(const bz_source_ops* s, const bz_monitor_ops* m) {
  Ops2D<T> o = {};
  if (s && s->n_ops > 0) {
    o.n_src = s->n_ops;
    o.src_steps = s->n_steps;
    o.src_row = s->row_ptr;
    o.src_cell = s->cell;
    o.src_mul = (const T*)s->mul;
    o.src_w = (const T*)s->weight;
    o.w_stride = s->weight_stride;
    o.src_sig = s->sig;
    o.signals = (const T*)s->signals;
  }
  if (m && m->n_points > 0 && (m->record || m->ring)) {
    o.n_mon = m->n_points;
    o.ring_len = m->ring_len;
    o.mon_row = m->row_ptr;
    o.mon_cell = m->cell;
    o.mon_point = m->point;
    o.record = (T*)m->record;
    o.rec_step0 = m->rec_step0;
    o.n_rec = m->n_rec;
    o.ring = (T*)m->ring;
  }
  return o;
}

template <typename T, int TS, int R, int NW, int MINB, bool PWR = false>
int launch_tb(const bz_grid2d* gd, const bz_fields2d* f, const bz_source_ops* s, const bz_monitor_ops* m,
              int64_t step, const int64_t* d_step, cudaStream_t st) {
  constexpr int OW = TBW - 2 * (TS + 1), OH = NW * R - 2 * TS;
  constexpr int SMEM = TbSmem<T, TS, R, NW>::BYTES;
  const auto kernel = step2d_tb_kernel<T, TS, R, NW, MINB, PWR>;
  static std::atomic<unsigned long long> devices{0ull};
  if (!raise_smem_limit((const void*)kernel, SMEM, devices))
    return fail(BZ_ERR_CUDA, "bz_step2d_multi: cannot configure the kernel's shared memory");
  const Geo2D<T> g = make_geo<T>(gd);
  Ops2D<T> o = make_ops<T>(s, m);
  if (m && m->region && m->n_reg > 1) {
    o.region = (T*)m->region;
    o.rx0 = m->rx0;
    o.ry0 = m->ry0;
    o.rw = m->rw;
    o.rh = m->rh;
    o.n_reg = m->n_reg;
    o.reg_step0 = m->reg_step0;
  }
  uintptr_t bits = (uintptr_t)f->ce | (uintptr_t)f->loss;
  for (int i = 0; i < 2; ++i) bits |= (uintptr_t)f->ez[i] | (uintptr_t)f->hx[i] | (uintptr_t)f->hy[i];
  const bool vec = bits % (2 * sizeof(T)) == 0;  // pairs start at even columns and the pitch is even
  const int src = (int)(step & 1);
  const int n_planes = gd->n_designs * gd->n_comp;
  const int ahead = prefetch_distance((long long)sizeof(T) * g.plane * (6LL * n_planes + 2LL * gd->n_mat),
                                      ceil_div(gd->nx, OW) * ceil_div(gd->ny, OH) * (long long)n_planes);
  for (int p0 = 0; p0 < n_planes; p0 += 65535) {  // the z extent of a grid is at most 65535
    dim3 grid((unsigned)ceil_div(gd->nx, OW), (unsigned)ceil_div(gd->ny, OH),
              (unsigned)(n_planes - p0 < 65535 ? n_planes - p0 : 65535));
    kernel<<<grid, 32 * NW, SMEM, st>>>(
        (const T*)f->ez[src], (const T*)f->hx[src], (const T*)f->hy[src], (T*)f->ez[src ^ 1], (T*)f->hx[src ^ 1],
        (T*)f->hy[src ^ 1], (const T*)f->ce, (const T*)f->loss, f->power, g, o, gd->n_comp, p0, n_planes,
        ahead, vec,
        (long long)step, (const long long*)d_step);
  }
  return check_launch("bz_step2d_multi");
}

// Tile shapes (rows a warp x warps) for float: 0, 2 and 5 = 8 x 8, 1 = 4 x 8, 3 = 2 x 16,
// 4 = 4 x 12; three steps a launch always take 4 x 8 (a shape costs little
// there). Double takes 4 x 16, or 2 x 16 for tiles 1 and 3.
template <typename T, int TS>
int tb_by_tile(const bz_grid2d* g, const bz_fields2d* f, const bz_source_ops* s, const bz_monitor_ops* m,
               int64_t step, int32_t tile, const int64_t* d_step, cudaStream_t st) {
  if constexpr (sizeof(T) == 4 && TS == 3) {
    return launch_tb<T, TS, 4, 8, 3>(g, f, s, m, step, d_step, st);
  } else if constexpr (sizeof(T) == 4) {
    switch (tile) {
      case 1: return launch_tb<T, TS, 4, 8, 3>(g, f, s, m, step, d_step, st);
      case 3: return launch_tb<T, TS, 2, 16, 2>(g, f, s, m, step, d_step, st);
      case 4: return launch_tb<T, TS, 4, 12, 2>(g, f, s, m, step, d_step, st);
      default: return launch_tb<T, TS, 8, 8, 2>(g, f, s, m, step, d_step, st);
    }
  } else {
    if (tile == 1 || tile == 3) return launch_tb<T, TS, 2, 16, 1>(g, f, s, m, step, d_step, st);
    return launch_tb<T, TS, 4, 16, 1>(g, f, s, m, step, d_step, st);
  }
}

template <typename T>
int tb_by_steps(const bz_grid2d* g, const bz_fields2d* f, const bz_source_ops* s, const bz_monitor_ops* m,
                int64_t step, int32_t n_sub, int32_t tile, const int64_t* d_step, cudaStream_t st) {
  switch (n_sub) {
    case 3: return tb_by_tile<T, 3>(g, f, s, m, step, tile, d_step, st);
    case 7: return tb_by_tile<T, 7>(g, f, s, m, step, tile, d_step, st);
    case 9: return tb_by_tile<T, 9>(g, f, s, m, step, tile, d_step, st);
    default: return tb_by_tile<T, 5>(g, f, s, m, step, tile, d_step, st);
  }
}

template <typename T, int NC, bool PWR, int RB>
int launch(const bz_grid2d* gd, const bz_fields2d* f, const bz_source_ops* s, const bz_monitor_ops* m,
           int64_t step, const int64_t* d_step, cudaStream_t st) {
  const Geo2D<T> g = make_geo<T>(gd);
  Ops2D<T> o = make_ops<T>(s, m);
  if (m && m->region && m->n_reg > 1) {
    o.region = (T*)m->region;
    o.rx0 = m->rx0;
    o.ry0 = m->ry0;
    o.rw = m->rw;
    o.rh = m->rh;
    o.n_reg = m->n_reg;
    o.reg_step0 = m->reg_step0;
  }
  const int src = (int)(step & 1);  // copy read by this launch: parity of the host-side step argument
  dim3 grid((unsigned)ceil_div(gd->nx, BX), (unsigned)ceil_div(gd->ny, RB), (unsigned)gd->n_designs);
  step2d_kernel<T, NC, PWR, RB><<<grid, BX, 0, st>>>(
      (const T*)f->ez[src], (const T*)f->hx[src], (const T*)f->hy[src], (T*)f->ez[src ^ 1], (T*)f->hx[src ^ 1],
      (T*)f->hy[src ^ 1], (const T*)f->ce, (const T*)f->loss, f->power, g, o, (long long)step,
      (const long long*)d_step);
  return check_launch("bz_step2d");
}

template <typename T, int NC, bool PWR>
int by_rows(const bz_grid2d* g, const bz_fields2d* f, const bz_source_ops* s, const bz_monitor_ops* m,
            int64_t step, const int64_t* d_step, cudaStream_t st) {
  switch (g->tile_rows) {
    case 4: return launch<T, NC, PWR, 4>(g, f, s, m, step, d_step, st);
    case 8: return launch<T, NC, PWR, 8>(g, f, s, m, step, d_step, st);
    case 32: return launch<T, NC, PWR, 32>(g, f, s, m, step, d_step, st);
    default: return launch<T, NC, PWR, 16>(g, f, s, m, step, d_step, st);
  }
}

template <typename T>
int dispatch(const bz_grid2d* g, const bz_fields2d* f, const bz_source_ops* s, const bz_monitor_ops* m,
             int64_t step, const int64_t* d_step, cudaStream_t st) {
  const bool pw = f->power != nullptr;
  if (g->n_comp == 1) return pw ? by_rows<T, 1, true>(g, f, s, m, step, d_step, st) : by_rows<T, 1, false>(g, f, s, m, step, d_step, st);
  return pw ? by_rows<T, 2, true>(g, f, s, m, step, d_step, st) : by_rows<T, 2, false>(g, f, s, m, step, d_step, st);
}

}  // namespace
}  // namespace bz

namespace bz {
namespace {

int check_step_args(const char* who, const bz_grid2d* g, const bz_fields2d* f, const bz_source_ops* s,
                    const bz_monitor_ops* m, int64_t step) {
  BZ_REQUIRE(g && f, "%s: grid or fields is NULL", who);
  BZ_REQUIRE(g->nx >= 2 && g->ny >= 2, "%s: grid must be at least 2x2 (got %d x %d)", who, g->nx, g->ny);
  BZ_REQUIRE(g->pitch >= g->nx && g->pitch % 32 == 0, "%s: pitch %d must be >= nx and a multiple of 32", who,
             g->pitch);
  BZ_REQUIRE(g->n_designs >= 1 && g->n_designs <= 65535, "%s: n_designs %d out of range", who, g->n_designs);
  BZ_REQUIRE(g->n_comp == 1 || g->n_comp == 2, "%s: n_comp must be 1 or 2 (got %d)", who, g->n_comp);
  BZ_REQUIRE(g->n_mat == 1 || g->n_mat == g->n_designs, "%s: n_mat must be 1 or n_designs", who);
  BZ_REQUIRE(g->dtype == BZ_F32 || g->dtype == BZ_F64, "%s: unknown dtype %d", who, g->dtype);
  for (int i = 0; i < 2; ++i) BZ_REQUIRE(f->ez[i] && f->hx[i] && f->hy[i], "%s: field buffer %d is NULL", who, i);
  BZ_REQUIRE(f->ce && f->loss, "%s: coefficient arrays are NULL", who);
  BZ_REQUIRE(step >= 0, "%s: negative step", who);
  if (s && s->n_ops > 0)
    BZ_REQUIRE(s->row_ptr && s->cell && s->mul && s->weight && s->sig && s->signals && s->n_steps >= 0,
               "%s: incomplete source ops", who);
  if (m && m->region) BZ_REQUIRE(m->rw >= 1 && m->rh >= 1 && m->n_reg >= 1, "%s: bad capture box", who);
  if (m && m->n_points > 0) {
    BZ_REQUIRE(m->row_ptr && m->cell && m->point, "%s: incomplete monitor ops", who);
    BZ_REQUIRE(m->ring == nullptr || m->ring_len >= 1, "%s: ring without length", who);
    BZ_REQUIRE(m->record == nullptr || m->n_rec >= 0, "%s: bad record length", who);
  }
  return BZ_OK;
}

}  // namespace
}  // namespace bz

extern "C" int bz_step2d(const bz_grid2d* g, const bz_fields2d* f, const bz_source_ops* s,
                         const bz_monitor_ops* m, int64_t step, const int64_t* d_step, void* stream) {
  const int rc = bz::check_step_args("bz_step2d", g, f, s, m, step);
  if (rc != BZ_OK) return rc;
  BZ_REQUIRE(g->tile_rows == 0 || g->tile_rows == 4 || g->tile_rows == 8 || g->tile_rows == 16 || g->tile_rows == 32,
             "bz_step2d: tile_rows must be 0, 4, 8, 16 or 32 (got %d)", g->tile_rows);
  cudaStream_t st = bz::as_stream(stream);
  return g->dtype == BZ_F32 ? bz::dispatch<float>(g, f, s, m, step, d_step, st)
                            : bz::dispatch<double>(g, f, s, m, step, d_step, st);
}

extern "C" int bz_step2d_multi(const bz_grid2d* g, const bz_fields2d* f, const bz_source_ops* s,
                               const bz_monitor_ops* m, int64_t step, int32_t n_sub, int32_t tile,
                               const int64_t* d_step, void* stream) {
  const int rc = bz::check_step_args("bz_step2d_multi", g, f, s, m, step);
  if (rc != BZ_OK) return rc;
  BZ_REQUIRE(n_sub == 1 || n_sub == 3 || n_sub == 5 || n_sub == 7 || n_sub == 9,
             "bz_step2d_multi: n_sub must be 1, 3, 5, 7 or 9 (got %d)",
             n_sub);
  BZ_REQUIRE(tile >= 0 && tile <= 5, "bz_step2d_multi: tile must be 0..5 (got %d)", tile);
  if (n_sub == 1) return bz_step2d(g, f, s, m, step, d_step, stream);
  if (f->power != nullptr)
    return bz::fail(BZ_ERR_UNSUPPORTED, "bz_step2d_multi: power accumulation needs bz_step2d or bz_step2d_multi_power");
  cudaStream_t st = bz::as_stream(stream);
  return g->dtype == BZ_F32 ? bz::tb_by_steps<float>(g, f, s, m, step, n_sub, tile, d_step, st)
                            : bz::tb_by_steps<double>(g, f, s, m, step, n_sub, tile, d_step, st);
}

extern "C" int bz_step2d_multi_power(const bz_grid2d* g, const bz_fields2d* f, const bz_source_ops* s,
                                     const bz_monitor_ops* m, int64_t step, const int64_t* d_step, void* stream) {
  const int rc = bz::check_step_args("bz_step2d_multi_power", g, f, s, m, step);
  if (rc != BZ_OK) return rc;
  BZ_REQUIRE(f->power != nullptr, "bz_step2d_multi_power: power is NULL");
  BZ_REQUIRE(g->n_comp == 1, "bz_step2d_multi_power: one component only (the power of two mixes them)");
  cudaStream_t st = bz::as_stream(stream);
  // The sums take 16 bytes of registers a cell: 64 x 48 tiles, one block an SM. 500 x 300
  // cells with four recorded edge lines: 16.0 us a launch of seven steps, against 23.7 us
  // a step in bz_step2d.
  if (g->dtype == BZ_F32) return bz::launch_tb<float, 7, 4, 12, 1, true>(g, f, s, m, step, d_step, st);
  return bz::launch_tb<double, 7, 2, 16, 1, true>(g, f, s, m, step, d_step, st);
}
