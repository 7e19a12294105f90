// Exact discrete adjoint of the 2D step (bz_step2d), one time step backwards.
//
// Forward step n (coefficients per cell from ce, loss; interior mask I):
//   Hx' = fh*Hx - cx*(E(x+1) - E(x))        Hy' = fh*Hy + cy*(E(y+1) - E(y))
//   Et  = Fe*E + Ce*((Hx'(x-1) - Hx'(x)) - qy*(Hy'(y-1) - Hy'(y)))    Fe = I?fe:1, Ce = I?ce:0
//   E_{n+1} = mul*Et + sources,   J reads E_{n+1} at monitor cells.
// Reverse mode with e = dJ/dEt (already multiplied by mul and fed the objective's
// dJ/dE_{n+1}), and carried adjoints hx, hy of H' from later steps:
//   U   = Ce*e
//   hx' = hx + U(x+1) - U(x)                hy' = hy - qy*(U(y+1) - U(y))
//   wx  = cx*hx',  wy = cy*hy'   (zero where Hx, Hy do not exist)
//   dJ/dE_n = Fe*e - (wx(x-1) - wx(x)) + (wy(y-1) - wy(y))
//   carried: hx <- fh*hx', hy <- fh*hy'
// The data flow mirrors the forward kernel (an H-like pass reading +1 neighbours,
// then an E-like pass reading -1 neighbours), so the same column-march layout is
// used. In the design region (no conductivity) dEt/d eps_r = -(Et - E_n)/eps_r, and
// the kernel accumulates grad += -e*(E_{n+1} - E_n)/eps_r from captured forward
// fields. The post phase then prepares the input of step n-1:
//   e_{n-1} = mul*(dJ/dE_n + objective term), through the same source operations.
#include "bz_tile.cuh"

namespace bz {
namespace {

constexpr int BX = 128;
constexpr int RB = 16;

template <typename T>
struct AdjArgs {
  const T* e_in;
  const T* hx_in;
  const T* hy_in;
  T* e_out;
  T* hx_out;
  T* hy_out;
  const T* ce;
  const T* loss;
  int nx, ny, pitch, n_designs, n_mat;
  long long plane;
  T chx, chy, qy, inv_kd2;
  // gradient
  double* grad;
  const double* eps_region;
  const T* fwd;
  int rx0, ry0, rw, rh, n_fwd;
  long long fwd_step0;
  // operations preparing step n-1
  int n_src, src_steps;
  const int* src_row;
  const int* src_cell;
  const T* src_mul;
  const T* src_w;
  long long w_stride;
  const int* src_sig;
  const T* signals;
};

template <typename T>
__device__ __forceinline__ void cell_coeffs(const AdjArgs<T>& a, const T* lsp, const T* cep, long long r, int x,
                                            int y, T& fh, T& cx, T& cy, T& Fe, T& Ce) {
  const T ls = __ldg(lsp + r), c = __ldg(cep + r);
  h_coeffs(ls, a.chx, a.chy, fh, cx, cy);
  const bool interior = x >= 1 && x <= a.nx - 2 && y >= 1 && y <= a.ny - 2;
  Fe = interior ? T(1) - ls * c * a.inv_kd2 : T(1);
  Ce = interior ? c : T(0);
}

template <typename T>
__global__ void __launch_bounds__(BX) adjoint2d_kernel(AdjArgs<T> a, long long step) {
  const int nx = a.nx, ny = a.ny, pitch = a.pitch;
  const int x = blockIdx.x * BX + threadIdx.x;
  const int wl = threadIdx.x & 31;
  const int d = blockIdx.z;
  const int y0 = blockIdx.y * RB;
  const int nrows = min(RB, ny - y0);
  const bool xin = x < nx;
  const long long fb = (long long)d * a.plane;
  const long long mb = (a.n_mat > 1 ? (long long)d : 0LL) * a.plane;
  const T* lsp = a.loss + mb;
  const T* cep = a.ce + mb;
  const T* E = a.e_in + fb;

  // U(y0, x) and the carried wy(y0-1, x) of the row above the tile
  T fh, cx, cy, Fe, Ce;
  T Uc = T(0), wy_up = T(0);
  if (xin) {
    cell_coeffs(a, lsp, cep, (long long)y0 * pitch + x, x, y0, fh, cx, cy, Fe, Ce);
    Uc = Ce * __ldg(E + (long long)y0 * pitch + x);
    if (y0 >= 1) {
      const long long r = (long long)(y0 - 1) * pitch + x;
      T fhm, cxm, cym, Fem, Cem;
      cell_coeffs(a, lsp, cep, r, x, y0 - 1, fhm, cxm, cym, Fem, Cem);
      const T Um = Cem * __ldg(E + r);
      const T hyp = __ldg(a.hy_in + fb + r) - a.qy * (Uc - Um);
      wy_up = cym * hyp;
    }
  }
  for (int i = 0; i < RB; ++i) {
    const int y = y0 + i;
    if (i >= nrows) break;  // uniform across the block
    const long long r = (long long)y * pitch + x;
    T e = T(0);
    if (xin) {
      cell_coeffs(a, lsp, cep, r, x, y, fh, cx, cy, Fe, Ce);
      e = __ldg(E + r);
    }
    T Un = T(0);  // U(y+1, x)
    if (xin && y + 1 < ny) {
      T fh1, cx1, cy1, Fe1, Ce1;
      cell_coeffs(a, lsp, cep, r + pitch, x, y + 1, fh1, cx1, cy1, Fe1, Ce1);
      Un = Ce1 * __ldg(E + r + pitch);
    }
    T Ur = __shfl_down_sync(FULL, Uc, 1);  // U(y, x+1)
    if (wl == 31) {
      Ur = T(0);
      if (x + 1 < nx) {
        T f1, c1, c2, Fe1, Ce1;
        cell_coeffs(a, lsp, cep, r + 1, x + 1, y, f1, c1, c2, Fe1, Ce1);
        Ur = Ce1 * __ldg(E + r + 1);
      }
    }
    const T hx0 = xin ? __ldg(a.hx_in + fb + r) : T(0);
    const T hy0 = xin ? __ldg(a.hy_in + fb + r) : T(0);
    const T hxp = hx0 + (Ur - Uc);
    const T hyp = hy0 - a.qy * (Un - Uc);
    const T wx = (x < nx - 1) ? cx * hxp : T(0);
    const T wy = (y < ny - 1) ? cy * hyp : T(0);
    T wx_left = __shfl_up_sync(FULL, wx, 1);
    if (wl == 0) {
      wx_left = T(0);
      if (xin && x >= 1) {  // recompute wx(y, x-1) of the lane to the left
        T fl, cxl, cyl, Fel, Cel;
        cell_coeffs(a, lsp, cep, r - 1, x - 1, y, fl, cxl, cyl, Fel, Cel);
        const T Ul = Cel * __ldg(E + r - 1);
        wx_left = cxl * (__ldg(a.hx_in + fb + r - 1) + (Uc - Ul));
      }
    }
    if (xin) {
      const T e_prev = Fe * e - (wx_left - wx) + (wy_up - wy);
      a.e_out[fb + r] = e_prev;
      if (x < nx - 1) a.hx_out[fb + r] = fh * hxp;
      if (y < ny - 1) a.hy_out[fb + r] = fh * hyp;
      if (a.grad != nullptr) {
        const int rx = x - a.rx0, ry = y - a.ry0;
        const long long s1 = step + 1 - a.fwd_step0;
        if (rx >= 0 && rx < a.rw && ry >= 0 && ry < a.rh && s1 >= 1 && s1 < a.n_fwd) {
          const long long cell = (long long)ry * a.rw + rx;
          const long long per = (long long)a.n_designs * a.rh * a.rw;
          const double en1 = (double)a.fwd[s1 * per + (long long)d * a.rh * a.rw + cell];
          const double en0 = (double)a.fwd[(s1 - 1) * per + (long long)d * a.rh * a.rw + cell];
          const double er = a.eps_region[(a.n_mat > 1 ? (long long)d : 0LL) * a.rh * a.rw + cell];
          a.grad[(long long)d * a.rh * a.rw + cell] -= (double)e * (en1 - en0) / er;
        }
      }
    }
    Uc = Un;
    wy_up = wy;
  }

  if (a.n_src == 0 || step == 0) return;
  // ---- post phase: e_{n-1} = mul * (dJ/dE_n + objective term at step n-1) ---------
  __shared__ int s_k0[RB], s_pre[RB + 1];
  const int xlo = blockIdx.x * BX;
  const int xhi = min(xlo + BX, nx);
  __syncthreads();
  const int total = block_op_ranges(a.src_row, a.src_cell, y0, nrows, nx, xlo, xhi, s_k0, s_pre);
  const long long sstep = step - 1;
  for (int i = threadIdx.x; i < total; i += BX) {
    int t;
    const int k = op_at(i, nrows, s_k0, s_pre, t);
    const int cell = __ldg(a.src_cell + k);
    if (i > s_pre[t] && __ldg(a.src_cell + k - 1) == cell) continue;
    const int y = y0 + t;
    const long long rr = fb + (long long)y * pitch + (cell - y * nx);
    T v = a.e_out[rr];
    for (int kk = k; kk < a.n_src && __ldg(a.src_cell + kk) == cell; ++kk) {
      const T s = sstep < a.src_steps ? __ldg(a.signals + (long long)__ldg(a.src_sig + kk) * a.src_steps + sstep) : T(0);
      v = __ldg(a.src_mul + kk) * v + __ldg(a.src_w + d * a.w_stride + kk) * s;
    }
    a.e_out[rr] = v;
  }
}


// ---- several reverse steps per launch (temporal blocking) ---------------------------
// The register tile of the blocked forward kernel (bz_step2d.cu: two adjacent columns a
// lane as one packed operand, R rows a warp, halo of TS+1 columns and TS rows a side),
// run backwards: TS reverse steps m = step, step-1, ..., each the single-step adjoint
// above. Per sub-step a warp receives U = Ce*e of the rows above and below it (one block
// barrier) and carries hy' of the row above itself. Tiles clear of loss and off the
// grid's edge need no factor but Ce; there the E-like pass takes the constant factors out
// of the differences (cx*(hx'(x) - hx'(x-1))). Other tiles read fh, cx, cy and Fe from
// shared memory; boundary rules enter the factors (Ce = 0, Fe = 1 off the interior;
// cx = 0 in the last column and outside, cy = 0 in the last row and outside).
//
// Design-box cells keep each sub-step's incoming e in shared memory ([TS][R][thread]
// pairs); their gradient terms are applied after the last sub-step, off the
// barrier-paced loop. The history and the factors share one region, so that two float
// blocks of five steps fit an SM; a tile that needs both (the box next to the absorber)
// recomputes its factors from the loss each sub-step instead.
//
// Bound by issue and latency like the forward kernel, and by the tile loads, which two
// blocks an SM hide only in part. 64 designs of 600 x 400 with a 120 x 120 box, 1500
// reverse steps: 98 ms in launches of five (two blocks an SM), 124 ms in launches of seven
// (one block: the history takes 115 KB); 114 ms before, with seven factors and fields a
// cell in registers and two barriers a sub-step.
constexpr int ADJ_POOL = 160;  // cells with operations held on chip; further ones are read from memory
template <typename T, int TS, int R, int NW>
struct AdjSmem {
  static constexpr int TH = NW * R;
  static constexpr int FAC = 4 * TH * TBW * (int)sizeof(T), HIST = TS * TH * TBW * (int)sizeof(T);
  static constexpr int SHARED = FAC > HIST ? FAC : HIST;
  static constexpr int EXCH = 2 * 2 * NW * TBW * (int)sizeof(T);
  static constexpr int POOL = (TS + 1) * ADJ_POOL * (int)sizeof(T);
  static constexpr int MAP = TH * TBW * (int)sizeof(short);
  static constexpr int BYTES = SHARED + EXCH + POOL + MAP + 16;
};

// The operations of one cell (sorted list entries k .. until another cell) at the N steps
// sstep, sstep-1, ...: v <- fac * v + add[i].
template <int N, typename T>
__device__ __forceinline__ void adj_run(const AdjArgs<T>& a, int d, int k, int k1, long long sstep, T& fac, T (&add)[N]) {
  const int cell = __ldg(a.src_cell + k);
  fac = T(1);
#pragma unroll
  for (int i = 0; i < N; ++i) add[i] = T(0);
  do {
    const T m = __ldg(a.src_mul + k), wv = __ldg(a.src_w + d * a.w_stride + k);
    const T* sg = a.signals + (long long)__ldg(a.src_sig + k) * a.src_steps + sstep;
    fac *= m;
#pragma unroll
    for (int i = 0; i < N; ++i)
      add[i] = m * add[i] + wv * (sstep - i >= 0 && sstep - i < a.src_steps ? __ldg(sg - i) : T(0));
    ++k;
  } while (k < k1 && __ldg(a.src_cell + k) == cell);
}

template <typename T, int TS, int R, int NW, int MINB>
__global__ void __launch_bounds__(32 * NW, MINB) adjoint2d_tb_kernel(AdjArgs<T> a, int ahead, bool vec, long long step0) {
  typedef typename PairOf<T>::type V;
  typedef AdjSmem<T, TS, R, NW> S;
  constexpr int TH = S::TH, HX = TS + 1, OW = TBW - 2 * HX, OH = TH - 2 * TS, NT = 32 * NW;
  static_assert(TS % 2 == 1 && OW > 0 && OH > 0 && R <= 16, "bad temporal tile");
  extern __shared__ __align__(16) unsigned char adj_smem[];
  V* s_fac = reinterpret_cast<V*>(adj_smem);   // [4][TH][32]: fh, cx, cy, Fe
  V* s_hist = s_fac;                           // or [TS][R][NT]: incoming e of design-box cells
  V* s_ex = reinterpret_cast<V*>(adj_smem + S::SHARED);                 // [2][2][NW][32]: first, last rows' U
  T* s_pool = reinterpret_cast<T*>(adj_smem + S::SHARED + S::EXCH);     // [TS + 1][ADJ_POOL]: addends, factor
  int* s_used = reinterpret_cast<int*>(s_pool + (TS + 1) * ADJ_POOL);
  short* s_map = reinterpret_cast<short*>(s_used + 4);                  // [TH][64]

  const int nx = a.nx, ny = a.ny, pitch = a.pitch;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, d = blockIdx.z;
  const int X0 = (int)blockIdx.x * OW - HX, Y0 = (int)blockIdx.y * OH - TS;
  const int yb = Y0 + w * R, xa = X0 + 2 * lane, tr0 = w * R;
  const long long fb = (long long)d * a.plane + (long long)yb * pitch + xa;  // the thread's first cell
  const long long mb = (a.n_mat > 1 ? (long long)d : 0LL) * a.plane + (long long)yb * pitch + xa;
  const bool inner = X0 >= 1 && X0 + TBW - 1 <= nx - 2 && Y0 >= 1 && Y0 + TH - 1 <= ny - 2;
  const bool in0 = xa >= 0 && xa < nx, in1 = xa >= 0 && xa + 1 < nx;

  int sk0 = 0, sk1 = 0;  // the operations of the warp's rows
  if (a.n_src > 0 && max(yb, 0) < min(yb + R, ny)) {
    sk0 = __ldg(a.src_row + max(yb, 0));
    sk1 = __ldg(a.src_row + min(yb + R, ny));
  }
  if (threadIdx.x == 0) *s_used = 0;

  V e[R], hx[R], hy[R], cc[R], ls[R];
  V hyu;  // hy of the row above the warp's first; stale, as all halo rows, for warp 0
  if (inner && vec) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = i * pitch;
      ls[i] = ldg2(a.loss + mb + r);
      e[i] = ldg2(a.e_in + fb + r);
      hx[i] = ldg2(a.hx_in + fb + r);
      hy[i] = ldg2(a.hy_in + fb + r);
      cc[i] = ldg2(a.ce + mb + r);
    }
    hyu = ldg2(a.hy_in + fb - pitch);
  } else {
    const bool inm0 = in0 && xa < nx - 1, inm1 = in1 && xa + 1 < nx - 1;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int y = yb + i, r = i * pitch;
      const bool iny = y >= 0 && y < ny, inh = y >= 0 && y < ny - 1;
      ls[i] = ld_pair(a.loss + mb + r, in0 && iny, in1 && iny);
      e[i] = ld_pair(a.e_in + fb + r, in0 && iny, in1 && iny);
      hx[i] = ld_pair(a.hx_in + fb + r, inm0 && iny, inm1 && iny);
      hy[i] = ld_pair(a.hy_in + fb + r, in0 && inh, in1 && inh);
      cc[i] = ld_pair(a.ce + mb + r, in0 && iny, in1 && iny);
    }
    hyu = ld_pair(a.hy_in + fb - pitch, in0 && yb >= 1 && yb < ny, in1 && yb >= 1 && yb < ny);
  }
  if (ahead > 0) {  // the tile that a block of the next wave will load
    const long long next = ((long long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x + ahead;
    const int bz = (int)(next / ((long long)gridDim.x * gridDim.y));
    if (bz < (int)gridDim.z) {
      const int rem = (int)(next - (long long)bz * gridDim.x * gridDim.y), by = rem / (int)gridDim.x, bx = rem - by * (int)gridDim.x;
      const long long pf = (long long)bz * a.plane, pm = a.n_mat > 1 ? pf : 0LL;
      const T* const arr[5] = {a.e_in + pf, a.hx_in + pf, a.hy_in + pf, a.ce + pm, a.loss + pm};
      prefetch_tile<T, TH, NW>(arr, bx * OW - HX, by * OH - TS, ny, pitch, w, lane);
    }
  }
  __syncthreads();  // the pool's counter is set

  // Operations on every tile cell: a map cell -> pool slot, -1 for none, -2 - n for a cell
  // beyond the pool, found from the warp's n-th list entry on.
  unsigned src_rows = 0u;
  bool src_many = false;
  short* const w_src = s_map + tr0 * TBW;
  if (sk0 < sk1) {
    for (int i = lane; i < R * TBW; i += 32) w_src[i] = -1;
    __syncwarp();
    src_rows = scan_ops(a.src_cell, sk0, sk1, nx, yb, X0, max(X0, 0), min(X0 + TBW, nx), lane,
                        [&](int i, int col, int k, bool) {
      int slot = atomicAdd(s_used, 1);
      if (slot < ADJ_POOL) {
        T fac, add[TS];
        adj_run<TS>(a, d, k, sk1, step0 - 1, fac, add);
#pragma unroll
        for (int s = 0; s < TS; ++s) s_pool[s * ADJ_POOL + slot] = add[s];
        s_pool[TS * ADJ_POOL + slot] = fac;
      } else {
        slot = -2 - min(k - sk0, 32000);
        src_many = true;
      }
      w_src[i * TBW + col] = (short)slot;
    });
  }
  src_many = __any_sync(FULL, src_many);
  const bool own = lane >= HX / 2 && lane < 32 - HX / 2 && xa < nx;
  unsigned gbits = 0u;  // owned design-box cells: bit 2*i + column
  if (a.grad != nullptr && own) {
    const int rx = xa - a.rx0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int tr = tr0 + i, y = yb + i, ry = y - a.ry0;
      if (tr < TS || tr >= TH - TS || y >= ny || ry < 0 || ry >= a.rh) continue;
      if (rx >= 0 && rx < a.rw) gbits |= 1u << (2 * i);
      if (xa + 1 < nx && rx + 1 >= 0 && rx + 1 < a.rw) gbits |= 2u << (2 * i);
    }
  }

  bool lossy = !inner;
#pragma unroll
  for (int i = 0; i < R; ++i) lossy = lossy || nonzero2(ls[i]);
  lossy = __syncthreads_or(lossy);
  const bool boxed = __syncthreads_or(gbits != 0u);
  // factors of row yb + i (i = -1: the row above, fh and cy only); Ce of the row given
  auto factors = [&](int i, V c, V l, V& fh, V& cx, V& cy, V& fe) {
    const int y = yb + i;
    const bool iny = y >= 0 && y < ny, inh = y >= 0 && y < ny - 1;
    T fh0, fh1, cx0, cx1, cy0, cy1;
    h_coeffs(lo2(l), a.chx, a.chy, fh0, cx0, cy0);
    h_coeffs(hi2(l), a.chx, a.chy, fh1, cx1, cy1);
    fh = mk2(fh0, fh1);
    cx = mk2(iny && in0 && xa < nx - 1 ? cx0 : T(0), iny && in1 && xa + 1 < nx - 1 ? cx1 : T(0));
    cy = mk2(inh && in0 ? cy0 : T(0), inh && in1 ? cy1 : T(0));
    fe = mk2(T(1) - lo2(l) * lo2(c) * a.inv_kd2, T(1) - hi2(l) * hi2(c) * a.inv_kd2);  // 1 where c = 0
  };
  if (lossy) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int y = yb + i;
      const bool inty = y >= 1 && y <= ny - 2;
      cc[i] = mk2(inty && xa >= 1 && xa <= nx - 2 ? lo2(cc[i]) : T(0),
                  inty && xa + 1 >= 1 && xa + 1 <= nx - 2 ? hi2(cc[i]) : T(0));
      if (!boxed) {
        V fh, cx, cy, fe;
        factors(i, cc[i], ls[i], fh, cx, cy, fe);
        V* q = s_fac + (tr0 + i) * 32 + lane;
        q[0] = fh;
        q[TH * 32] = cx;
        q[2 * TH * 32] = cy;
        q[3 * TH * 32] = fe;
      }
    }
  }
  const V one = mk2(T(1), T(1)), qy = mk2(a.qy, a.qy), mqy = mk2(-a.qy, -a.qy), zero = mk2(T(0), T(0));
  const V pcx = mk2(a.chx, a.chx), pcy = mk2(a.chy, a.chy);

#pragma unroll 1
  for (int s = 0; s < TS; ++s) {
    if (gbits) {
#pragma unroll
      for (int i = 0; i < R; ++i) s_hist[(s * R + i) * NT + threadIdx.x] = e[i];
    }
    V* ex = s_ex + (s & 1) * (2 * NW * 32) + lane;
    V U = mul2(cc[0], e[0]);
    ex[w * 32] = U;
    ex[(NW + w) * 32] = mul2(cc[R - 1], e[R - 1]);
    __syncthreads();  // also orders the factors before their first use
    const V u_dn = w + 1 < NW ? ex[(w + 1) * 32] : zero;
    const V u_up = w > 0 ? ex[(NW + w - 1) * 32] : zero;
    if (!lossy) {
      hyu = fma2(mqy, sub2(U, u_up), hyu);
      V hu = hyu;  // hy' of the row above
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const V un = i + 1 < R ? mul2(cc[i + 1 < R ? i + 1 : i], e[i + 1 < R ? i + 1 : i]) : u_dn;
        const V ur = mk2(hi2(U), __shfl_down_sync(FULL, lo2(U), 1));  // lane 31: stale halo
        hx[i] = fma2(one, hx[i], sub2(ur, U));
        hy[i] = fma2(mqy, sub2(un, U), hy[i]);
        const V hl = mk2(__shfl_up_sync(FULL, hi2(hx[i]), 1), lo2(hx[i]));  // lane 0: stale halo
        e[i] = fma2(pcx, sub2(hx[i], hl), fma2(pcy, sub2(hu, hy[i]), e[i]));
        hu = hy[i];
        U = un;
      }
    } else {
      const V* q = s_fac + tr0 * 32 + lane;
      V wu = zero;  // cy * hy' of the row above
      if (w > 0) {
        V fh, cx, cy, fe;
        if (boxed) {
          factors(-1, zero, ld_pair(a.loss + mb - pitch, in0 && yb >= 1 && yb <= ny, in1 && yb >= 1 && yb <= ny), fh, cx, cy, fe);
        } else {
          fh = q[-32];
          cy = q[2 * TH * 32 - 32];
        }
        hyu = fma2(mqy, sub2(U, u_up), hyu);
        wu = mul2(cy, hyu);
        hyu = mul2(fh, hyu);
      }
#pragma unroll
      for (int i = 0; i < R; ++i) {
        V fh, cx, cy, fe;
        if (boxed) {
          const bool iny = yb + i >= 0 && yb + i < ny;
          factors(i, cc[i], ld_pair(a.loss + mb + i * pitch, in0 && iny, in1 && iny), fh, cx, cy, fe);
        } else {
          fh = q[i * 32];
          cx = q[(TH + i) * 32];
          cy = q[(2 * TH + i) * 32];
          fe = q[(3 * TH + i) * 32];
        }
        const V un = i + 1 < R ? mul2(cc[i + 1 < R ? i + 1 : i], e[i + 1 < R ? i + 1 : i]) : u_dn;
        const V ur = mk2(hi2(U), __shfl_down_sync(FULL, lo2(U), 1));
        const V hxp = fma2(one, hx[i], sub2(ur, U)), hyp = fma2(mqy, sub2(un, U), hy[i]);
        const V wx = mul2(cx, hxp), wy = mul2(cy, hyp);
        const V wl = mk2(__shfl_up_sync(FULL, hi2(wx), 1), lo2(wx));
        e[i] = fma2(one, fma2(fe, e[i], sub2(wx, wl)), sub2(wu, wy));
        hx[i] = mul2(fh, hxp);
        hy[i] = mul2(fh, hyp);
        wu = wy;
        U = un;
      }
    }
    // operations preparing step m-1 (none after step 0)
    if (src_rows && step0 - s >= 1) {
      const T* add = s_pool + s * ADJ_POOL;
      const T* fac = s_pool + TS * ADJ_POOL;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        if (!(src_rows & (1u << i))) continue;  // uniform across the warp
        const short2 m = *reinterpret_cast<const short2*>(w_src + i * TBW + 2 * lane);
        const int m0 = max((int)m.x, 0), m1 = max((int)m.y, 0);
        T v0 = lo2(e[i]), v1 = hi2(e[i]);
        if (m.x >= 0) v0 = fac[m0] * v0 + add[m0];
        if (m.y >= 0) v1 = fac[m1] * v1 + add[m1];
        if (src_many) {
          const int cell = (yb + i) * nx + xa;
          T f, ad[1];
          if (m.x < -1) {
            int k = sk0 - 2 - m.x;
            while (__ldg(a.src_cell + k) != cell) ++k;
            adj_run<1>(a, d, k, sk1, step0 - s - 1, f, ad);
            v0 = f * v0 + ad[0];
          }
          if (m.y < -1) {
            int k = sk0 - 2 - m.y;
            while (__ldg(a.src_cell + k) != cell + 1) ++k;
            adj_run<1>(a, d, k, sk1, step0 - s - 1, f, ad);
            v1 = f * v1 + ad[0];
          }
        }
        e[i] = mk2(v0, v1);
      }
    }
  }
  if (!own) return;
  // store the owned box
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int tr = tr0 + i, y = yb + i;
    if (tr < TS || tr >= TH - TS || y >= ny) continue;
    const long long off = fb + i * pitch;
    if (vec && xa + 1 < nx - 1) {  // both columns exist in every component
      *reinterpret_cast<V*>(a.e_out + off) = e[i];
      *reinterpret_cast<V*>(a.hx_out + off) = hx[i];
      if (y < ny - 1) *reinterpret_cast<V*>(a.hy_out + off) = hy[i];
    } else {
      a.e_out[off] = lo2(e[i]);
      if (in1) a.e_out[off + 1] = hi2(e[i]);
      if (xa < nx - 1) a.hx_out[off] = lo2(hx[i]);
      if (xa + 1 < nx - 1) a.hx_out[off + 1] = hi2(hx[i]);
      if (y < ny - 1) {
        a.hy_out[off] = lo2(hy[i]);
        if (in1) a.hy_out[off + 1] = hi2(hy[i]);
      }
    }
  }
  // grad -= sum over the sub-steps' reverse steps m of e_m * (E_{m+1} - E_m), over
  // eps_r, on the owned design-box cells (no other block writes them)
  if (gbits) {
    const long long per = (long long)a.n_designs * a.rh * a.rw, db = (long long)d * a.rh * a.rw;
    const long long eb = (a.n_mat > 1 ? (long long)d : 0LL) * a.rh * a.rw;
    const long long p0 = step0 + 1 - a.fwd_step0;  // captured plane E_{m+1} of sub-step 0
    const bool all = p0 < a.n_fwd && p0 - TS >= 0;  // every plane the sub-steps need was captured
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (!(gbits >> (2 * i) & 3u)) continue;
      const long long cell = (long long)(yb + i - a.ry0) * a.rw + (xa - a.rx0);
      const bool g0 = gbits >> (2 * i) & 1u, g1 = gbits >> (2 * i) & 2u;
      const T* f = a.fwd + p0 * per + db + cell;
      T f0[TS + 1], f1[TS + 1];  // planes p0, p0-1, ..., p0-TS, all loads issued before the sums
#pragma unroll
      for (int k = 0; k <= TS; ++k) {
        const bool ok = all || (p0 - k >= 0 && p0 - k < a.n_fwd);
        f0[k] = ok && g0 ? __ldg(f - k * per) : T(0);
        f1[k] = ok && g1 ? __ldg(f - k * per + 1) : T(0);
      }
      T acc0 = T(0), acc1 = T(0);  // the block's terms in the fields' precision (e and the planes are T)
#pragma unroll
      for (int s = 0; s < TS; ++s)
        if (p0 - s >= 1 && p0 - s < a.n_fwd) {
          const V h = s_hist[(s * R + i) * NT + threadIdx.x];
          acc0 += lo2(h) * (f0[s] - f0[s + 1]);
          acc1 += hi2(h) * (f1[s] - f1[s + 1]);
        }
      if (g0) a.grad[db + cell] -= (double)acc0 / a.eps_region[eb + cell];
      if (g1) a.grad[db + cell + 1] -= (double)acc1 / a.eps_region[eb + cell + 1];
    }
  }
}

template <typename T>
AdjArgs<T> adj_args(const bz_grid2d* g, const bz_adjoint2d* s, const bz_source_ops* ops, int32_t phase) {
  AdjArgs<T> a = {};
  const int src = phase & 1;
  a.e_in = (const T*)s->e[src];
  a.hx_in = (const T*)s->hx[src];
  a.hy_in = (const T*)s->hy[src];
  a.e_out = (T*)s->e[src ^ 1];
  a.hx_out = (T*)s->hx[src ^ 1];
  a.hy_out = (T*)s->hy[src ^ 1];
  a.ce = (const T*)s->ce;
  a.loss = (const T*)s->loss;
  a.nx = g->nx;
  a.ny = g->ny;
  a.pitch = g->pitch;
  a.n_designs = g->n_designs;
  a.n_mat = g->n_mat;
  a.plane = (long long)g->ny * g->pitch;
  a.chx = (T)g->chx;
  a.chy = (T)g->chy;
  a.qy = (T)g->qy;
  a.inv_kd2 = (T)g->inv_kd2;
  a.grad = s->grad;
  a.eps_region = s->eps_region;
  a.fwd = (const T*)s->fwd_region;
  a.rx0 = s->rx0;
  a.ry0 = s->ry0;
  a.rw = s->rw;
  a.rh = s->rh;
  a.n_fwd = s->n_fwd;
  a.fwd_step0 = s->fwd_step0;
  if (ops && ops->n_ops > 0) {
    a.n_src = ops->n_ops;
    a.src_steps = ops->n_steps;
    a.src_row = ops->row_ptr;
    a.src_cell = ops->cell;
    a.src_mul = (const T*)ops->mul;
    a.src_w = (const T*)ops->weight;
    a.w_stride = ops->weight_stride;
    a.src_sig = ops->sig;
    a.signals = (const T*)ops->signals;
  }
  return a;
}

template <typename T>
int launch_adj(const bz_grid2d* g, const bz_adjoint2d* s, const bz_source_ops* ops, int64_t step, int32_t phase,
               cudaStream_t st) {
  const AdjArgs<T> a = adj_args<T>(g, s, ops, phase);
  dim3 grid((unsigned)ceil_div(g->nx, BX), (unsigned)ceil_div(g->ny, RB), (unsigned)g->n_designs);
  adjoint2d_kernel<T><<<grid, BX, 0, st>>>(a, (long long)step);
  return check_launch("bz_adjoint_step2d");
}

template <typename T, int TS, int R, int NW, int MINB>
int launch_adj_tile(const bz_grid2d* g, const bz_adjoint2d* s, const bz_source_ops* ops, int64_t step, int32_t phase,
                    cudaStream_t st) {
  constexpr int SMEM = AdjSmem<T, TS, R, NW>::BYTES;
  const auto kernel = adjoint2d_tb_kernel<T, TS, R, NW, MINB>;
  const AdjArgs<T> a = adj_args<T>(g, s, ops, phase);
  static std::atomic<unsigned long long> devices{0ull};
  if (!raise_smem_limit((const void*)kernel, SMEM, devices))
    return fail(BZ_ERR_CUDA, "bz_adjoint_step2d_multi: cannot configure the kernel's shared memory");
  uintptr_t bits = (uintptr_t)s->ce | (uintptr_t)s->loss;
  for (int i = 0; i < 2; ++i) bits |= (uintptr_t)s->e[i] | (uintptr_t)s->hx[i] | (uintptr_t)s->hy[i];
  const bool vec = bits % (2 * sizeof(T)) == 0;
  dim3 grid((unsigned)ceil_div(g->nx, TBW - 2 * (TS + 1)), (unsigned)ceil_div(g->ny, NW * R - 2 * TS),
            (unsigned)g->n_designs);
  const int ahead = prefetch_distance((long long)sizeof(T) * a.plane * (6LL * g->n_designs + 2LL * g->n_mat),
                                      (long long)grid.x * grid.y * grid.z);
  kernel<<<grid, 32 * NW, SMEM, st>>>(a, ahead, vec, (long long)step);
  return check_launch("bz_adjoint_step2d_multi");
}

// float: 64 x 64 tiles, two blocks an SM up to five steps; where those leave SMs idle, 64 x
// 32 tiles of two rows a warp, whose sub-steps are shorter (300 x 200 cells, one design,
// nine steps a launch: 800 reverse steps 3.6 -> 2.2 ms). double: 64 x 32.
template <typename T, int TS>
int launch_adj_tb(const bz_grid2d* g, const bz_adjoint2d* s, const bz_source_ops* ops, int64_t step, int32_t phase,
                  cudaStream_t st) {
  if constexpr (sizeof(T) == 4) {
    const long long tiles = ceil_div(g->nx, TBW - 2 * (TS + 1)) * ceil_div(g->ny, 64 - 2 * TS) * (long long)g->n_designs;
    if (tiles >= 148) return launch_adj_tile<T, TS, 8, 8, 2>(g, s, ops, step, phase, st);
  }
  return launch_adj_tile<T, TS, 2, 16, 1>(g, s, ops, step, phase, st);
}

}  // namespace
}  // namespace bz

namespace bz {
namespace {
int check_adj(const char* who, const bz_grid2d* g, const bz_adjoint2d* s, const bz_source_ops* ops, int64_t step) {
  BZ_REQUIRE(g && s, "%s: grid or state is NULL", who);
  BZ_REQUIRE(g->n_comp == 1, "%s: only real fields (n_comp = 1)", who);
  BZ_REQUIRE(g->nx >= 2 && g->ny >= 2 && g->pitch >= g->nx && g->pitch % 32 == 0, "%s: bad grid", who);
  BZ_REQUIRE(g->n_mat == 1 || g->n_mat == g->n_designs, "%s: n_mat must be 1 or n_designs", who);
  for (int i = 0; i < 2; ++i) BZ_REQUIRE(s->e[i] && s->hx[i] && s->hy[i], "%s: NULL state buffer", who);
  BZ_REQUIRE(s->ce && s->loss, "%s: NULL coefficients", who);
  if (s->grad) BZ_REQUIRE(s->eps_region && s->fwd_region && s->rw >= 1 && s->rh >= 1, "%s: bad grad box", who);
  if (ops && ops->n_ops > 0)
    BZ_REQUIRE(ops->row_ptr && ops->cell && ops->mul && ops->weight && ops->sig && ops->signals,
               "%s: incomplete ops", who);
  BZ_REQUIRE(step >= 0, "%s: negative step", who);
  BZ_REQUIRE(g->dtype == BZ_F32 || g->dtype == BZ_F64, "%s: unknown dtype %d", who, g->dtype);
  return BZ_OK;
}
}  // namespace
}  // namespace bz

extern "C" int bz_adjoint_step2d_multi(const bz_grid2d* g, const bz_adjoint2d* s, const bz_source_ops* ops,
                                       int64_t step, int32_t n_sub, int32_t phase, void* stream) {
  const int rc = bz::check_adj("bz_adjoint_step2d_multi", g, s, ops, step);
  if (rc != BZ_OK) return rc;
  BZ_REQUIRE(n_sub == 1 || n_sub == 3 || n_sub == 5 || n_sub == 7 || n_sub == 9,
             "bz_adjoint_step2d_multi: n_sub must be 1, 3, 5, 7 or 9 (got %d)", n_sub);
  BZ_REQUIRE(step + 1 >= n_sub, "bz_adjoint_step2d_multi: %d reverse steps from step %lld pass step 0", n_sub,
             (long long)step);
  if (n_sub == 1) return bz_adjoint_step2d(g, s, ops, step, phase, stream);
  cudaStream_t st = bz::as_stream(stream);
  if (g->dtype == BZ_F32) {
    switch (n_sub) {
      case 3: return bz::launch_adj_tb<float, 3>(g, s, ops, step, phase, st);
      case 5: return bz::launch_adj_tb<float, 5>(g, s, ops, step, phase, st);
      case 9: return bz::launch_adj_tb<float, 9>(g, s, ops, step, phase, st);
      default: return bz::launch_adj_tb<float, 7>(g, s, ops, step, phase, st);
    }
  }
  switch (n_sub) {
    case 3: return bz::launch_adj_tb<double, 3>(g, s, ops, step, phase, st);
    case 5: return bz::launch_adj_tb<double, 5>(g, s, ops, step, phase, st);
    case 9: return bz::launch_adj_tb<double, 9>(g, s, ops, step, phase, st);
    default: return bz::launch_adj_tb<double, 7>(g, s, ops, step, phase, st);
  }
}

extern "C" int bz_adjoint_step2d(const bz_grid2d* g, const bz_adjoint2d* s, const bz_source_ops* ops, int64_t step,
                                 int32_t phase, void* stream) {
  BZ_REQUIRE(g && s, "bz_adjoint_step2d: grid or state is NULL");
  BZ_REQUIRE(g->n_comp == 1, "bz_adjoint_step2d: only real fields (n_comp = 1)");
  BZ_REQUIRE(g->nx >= 2 && g->ny >= 2 && g->pitch >= g->nx && g->pitch % 32 == 0, "bz_adjoint_step2d: bad grid");
  BZ_REQUIRE(g->n_mat == 1 || g->n_mat == g->n_designs, "bz_adjoint_step2d: n_mat must be 1 or n_designs");
  for (int i = 0; i < 2; ++i) BZ_REQUIRE(s->e[i] && s->hx[i] && s->hy[i], "bz_adjoint_step2d: NULL state buffer");
  BZ_REQUIRE(s->ce && s->loss, "bz_adjoint_step2d: NULL coefficients");
  if (s->grad) BZ_REQUIRE(s->eps_region && s->fwd_region && s->rw >= 1 && s->rh >= 1, "bz_adjoint_step2d: bad grad box");
  if (ops && ops->n_ops > 0)
    BZ_REQUIRE(ops->row_ptr && ops->cell && ops->mul && ops->weight && ops->sig && ops->signals,
               "bz_adjoint_step2d: incomplete ops");
  BZ_REQUIRE(step >= 0, "bz_adjoint_step2d: negative step");
  cudaStream_t st = bz::as_stream(stream);
  if (g->dtype == BZ_F32) return bz::launch_adj<float>(g, s, ops, step, phase, st);
  if (g->dtype == BZ_F64) return bz::launch_adj<double>(g, s, ops, step, phase, st);
  return bz::fail(BZ_ERR_INVALID, "bz_adjoint_step2d: unknown dtype %d", g->dtype);
}
