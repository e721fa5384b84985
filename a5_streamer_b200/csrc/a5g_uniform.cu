// a5g -- the field solve of a large uniformly refined Cartesian run (grid
// mode) on dense levels.
//
// Where every level of the tree is a complete rectangular grid, the solve of
// compute_fld needs no box lists, ghost recipes or refinement boundaries: a
// level is one dense array split by colour (all cells with even x + y,
// 0-based, then the odd ones, nx / 2 values per row). A red-black half-sweep
// reads one colour and one colour of the right-hand side and writes the other
// colour in place, unit stride, one kernel per half-sweep; the levels of at
// most UCOARSE cells run in one block in shared memory. The launches of a
// solve are captured once and replayed as a graph.
//
// Measured on the level-6 mesh of the 8 mm case (1,048,576 cells, 148
// blocks): behind the grid barriers of one cooperative launch a half-sweep
// took 3.2 us on average (0.5M cells over 75,776 threads, box records and
// ghost recipes through L2), and the solves 2.6 ms of a 3.2 ms step.
//
// The values are those of the box phases (a5g_phases.cuh), expression by
// expression, in FP64 and in the mixed form's FP32 correction solve.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "a5_uniform.h"

namespace {

constexpr int UMAXLV = 16, UCOARSE = 4096, UTHR = 512, UWARP = 64;
constexpr int UNC = 8, USLOT = 100, UFSLOT = 72;  // box_size and slots on levels >= 1
enum { I_ELEC = 0, I_PION = 1, I_PHI = 4, I_FLD = 5, I_RHS = 6, I_EPS = 8 };
constexpr double UC_EPS0 = 8.8541878176e-12, UC_ELEM_CHARGE = 1.6022e-19;

// One level: nx2 cells per row and colour, ny rows; magic numbers of the
// divisions by nx2 and by nx2 / V.
struct ULv {
  int nx2, ny, half;
  unsigned m_nx, m_nxv;
  int off;  // first cell in the arrays of all levels
  double dx2, inv_dx2, inv_dr;
};
// t / d through the high product: exact for t (m d - 2^32) < 2^32, m = ceil(2^32 / d); m 0 for d = 1
__device__ __forceinline__ unsigned udiv(unsigned t, unsigned m) { return m ? __umulhi(t, m) : t; }
unsigned magic(long long d) { return d <= 1 ? 0u : (unsigned)(((1ULL << 32) + d - 1) / d); }

template <class T, int V>
struct alignas(sizeof(T) * V) Vec {
  T v[V];
};
template <class T, int V>
__device__ __forceinline__ Vec<T, V> ldv(const T *p) { return *reinterpret_cast<const Vec<T, V> *>(p); }

// V consecutive cells of one colour: first index, parity of the row, walls
struct Group {
  int b;
  unsigned fl;
};
enum { GF_ODD = 1, GF_XL = 2, GF_XH = 4, GF_YL = 8, GF_YH = 16 };
template <int V>
__device__ __forceinline__ Group group_of(const ULv &L, int xv, int y) {
  return Group{y * L.nx2 + xv, (unsigned)(y & 1) | (xv == 0 ? GF_XL : 0) | (xv + V == L.nx2 ? GF_XH : 0) |
                                   (y == 0 ? GF_YL : 0) | (y == L.ny - 1 ? GF_YH : 0)};
}
// Places of a group's neighbours from the start of its level. Beyond a wall
// its own values are mirrored (sides_bc_pot, src/streamer_2d.f90:620-638:
// Neumann on x, -own at low y, 2 V - own at high y).
struct Places {
  int own, m, e, ym, yp;
  unsigned fl;
};
template <int V>
__device__ __forceinline__ Places places_of(const ULv &L, int c, const Group &g) {
  const int own = c * L.half + g.b, a = (1 - c) * L.half + g.b;
  const bool q = ((g.fl ^ c) & GF_ODD) != 0;  // x parity of the group's cells
  Places w;
  w.own = own;
  w.m = a;
  w.e = q ? ((g.fl & GF_XH) ? own + V - 1 : a + V) : ((g.fl & GF_XL) ? own : a - 1);
  w.ym = (g.fl & GF_YL) ? own : a - L.nx2;
  w.yp = (g.fl & GF_YH) ? own : a + L.nx2;
  w.fl = (g.fl & ~(unsigned)GF_ODD) | (q ? GF_ODD : 0);
  return w;
}
template <class T, int V>
struct Nbr {
  Vec<T, V> xm, xp, ym, yp;
};
template <class T, int V>
__device__ __forceinline__ Nbr<T, V> neighbours(const T *P, const Places &w, T v2) {
  Nbr<T, V> n;
  const Vec<T, V> m = ldv<T, V>(P + w.m);
  const T e = P[w.e];
  n.ym = ldv<T, V>(P + w.ym);
  n.yp = ldv<T, V>(P + w.yp);
  const bool q = w.fl & GF_ODD;
#pragma unroll
  for (int k = 0; k < V; k++) {
    n.xm.v[k] = q ? m.v[k] : (k == 0 ? e : m.v[k > 0 ? k - 1 : 0]);
    n.xp.v[k] = q ? (k == V - 1 ? e : m.v[k < V - 1 ? k + 1 : 0]) : m.v[k];
    if (w.fl & GF_YL) n.ym.v[k] = -n.ym.v[k];
    if (w.fl & GF_YH) n.yp.v[k] = v2 - n.yp.v[k];
  }
  return n;
}
// box_lpl (afivo/src/m_aX_mg.f90:662-680), box_gsrb_lpl (:636-659)
template <class T>
__device__ __forceinline__ T lap(T xm, T xp, T ym, T yp, T own, T inv) {
  return inv * (xm + xp + ym + yp - T(4) * own);
}
template <class T, int V>
__device__ __forceinline__ T lap_of(const Nbr<T, V> &n, int k, T own, T inv) {
  return lap(n.xm.v[k], n.xp.v[k], n.ym.v[k], n.yp.v[k], own, inv);
}
template <class T, int V>
__device__ __forceinline__ T gsrb_of(const Nbr<T, V> &n, int k, T dx2f) {
  return T(0.25) * (n.xp.v[k] + n.xm.v[k] + n.yp.v[k] + n.ym.v[k] - dx2f);
}

// One group of a half-sweep of colour c (1 on odd half-sweeps: i + j odd,
// 1-based). FIRST: the restriction has just reached the level, F holds the
// restricted residual and F = lpl(O) + F first, O being P before the visit.
template <class T, int V, bool FIRST>
__global__ void __launch_bounds__(256) u_sweep(ULv L, T *P, T *F, const T *O, int c, T v2) {
  const unsigned t = blockIdx.x * 256u + threadIdx.x;
  if (t >= (unsigned)(L.half / V)) return;
  const int nv = L.nx2 / V, y = udiv(t, L.m_nxv);
  const Places w = places_of<V>(L, c, group_of<V>(L, (t - y * nv) * V, y));
  Vec<T, V> f = ldv<T, V>(F + w.own);
  const Nbr<T, V> n = neighbours<T, V>(P, w, v2);
  if (FIRST) {
    const Vec<T, V> o = ldv<T, V>(O + w.own);
    const Nbr<T, V> n0 = neighbours<T, V>(O, w, v2);
#pragma unroll
    for (int k = 0; k < V; k++) f.v[k] = lap_of<T, V>(n0, k, o.v[k], T(L.inv_dx2)) + f.v[k];
    *reinterpret_cast<Vec<T, V> *>(F + w.own) = f;
  }
  Vec<T, V> r;
#pragma unroll
  for (int k = 0; k < V; k++) r.v[k] = gsrb_of<T, V>(n, k, T(L.dx2) * f.v[k]);
  *reinterpret_cast<Vec<T, V> *>(P + w.own) = r;
}

__device__ __forceinline__ int didx(const ULv &L, int x, int y) { return ((x + y) & 1) * L.half + y * L.nx2 + (x >> 1); }

// The 2 x 2 fine cells under cell (X, Y) of the coarser level and what
// surrounds them: w, f and the operator a per cell in the order of
// box_rstr_lpl (i fastest)
template <class T>
struct Quad {
  T w[4], f[4], a[4];
  int at[4];
};
template <class T>
__device__ __forceinline__ Quad<T> quad(const ULv &L, const T *P, const T *F, int X, int Y, T v2) {
  Quad<T> q;
  const int x0 = 2 * X, y0 = 2 * Y, b = y0 * L.nx2 + X;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int dx = k & 1, dy = k >> 1;
    q.at[k] = ((dx + dy) & 1) * L.half + b + dy * L.nx2;
    q.w[k] = P[q.at[k]];
    q.f[k] = F[q.at[k]];
  }
  T xl[2], xh[2], yl[2], yh[2];
#pragma unroll
  for (int d = 0; d < 2; d++) {
    const int row = b + d * L.nx2;
    xl[d] = X > 0 ? P[((1 + d) & 1) * L.half + row - 1] : q.w[2 * d];
    xh[d] = x0 + 2 < 2 * L.nx2 ? P[(d & 1) * L.half + row + 1] : q.w[1 + 2 * d];
    yl[d] = Y > 0 ? P[((d + 1) & 1) * L.half + b - L.nx2] : -q.w[d];
    yh[d] = y0 + 2 < L.ny ? P[(d & 1) * L.half + b + 2 * L.nx2] : v2 - q.w[d + 2];
  }
  const T inv = T(L.inv_dx2);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int dx = k & 1, dy = k >> 1;
    q.a[k] = lap(dx ? q.w[k - 1] : xl[dy], dx ? xh[dy] : q.w[k + 1], dy ? q.w[k - 2] : yl[dx], dy ? yh[dx] : q.w[k + 2],
                 q.w[k], inv);
  }
  return q;
}
template <class T>
__device__ __forceinline__ T quarter(T a, T b, T c, T d) { return T(0.25) * (a + b + c + d); }

// Residual and phi restricted under one coarse cell (p_fr). SETUP: the fine
// level's F still holds the restricted residual: F = lpl(P) + F first.
template <class T, bool SETUP>
__device__ __forceinline__ void restrict_at(const ULv &L, const ULv &C, const T *P, T *F, T *Pc, T *Fc, T *Oc,
                                            unsigned t, T v2) {
  const int nx = 2 * C.nx2, Y = udiv(t >> 1, C.m_nx), X = (int)t - Y * nx;
  Quad<T> q = quad<T>(L, P, F, X, Y, v2);
  T r[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if (SETUP) {
      q.f[k] = q.a[k] + q.f[k];
      F[q.at[k]] = q.f[k];
    }
    r[k] = q.f[k] - q.a[k];
  }
  const int i = didx(C, X, Y);
  const T p = quarter(q.w[0], q.w[1], q.w[2], q.w[3]);
  Fc[i] = quarter(r[0], r[1], r[2], r[3]);
  Pc[i] = p;
  Oc[i] = p;
}
template <class T, bool SETUP>
__global__ void __launch_bounds__(128) u_restrict(ULv L, ULv C, const T *P, T *F, T *Pc, T *Fc, T *Oc, T v2) {
  const unsigned t = blockIdx.x * 128u + threadIdx.x;
  if (t < (unsigned)(2 * C.half)) restrict_at<T, SETUP>(L, C, P, F, Pc, Fc, Oc, t, v2);
}

// correct_children (:319-341) with box_corr_lpl (:605-633) for the pair of
// fine cells (2 X, y), (2 X + 1, y) under coarse cell (X, Y): phi += 0.5 c1 +
// 0.25 (c2x + c2y), the correction P - O of the coarser level; its ghost
// values from the walls' rule for both.
template <class T>
__device__ __forceinline__ void correct_at(const ULv &L, const ULv &C, T *P, const T *Pc, const T *Oc, unsigned t, T v2) {
  const int y = udiv(t, L.m_nx), X = (int)t - y * L.nx2, Y = y >> 1, Y2 = (y & 1) ? Y + 1 : Y - 1;
  const int i0 = didx(C, X, Y);
  const T p0 = Pc[i0], o0 = Oc[i0], c1 = p0 - o0;
  auto cv = [&](int x, int yy) {
    const int i = didx(C, x, yy);
    return Pc[i] - Oc[i];
  };
  const T cl = X > 0 ? cv(X - 1, Y) : c1, ch = X < 2 * C.nx2 - 1 ? cv(X + 1, Y) : c1;
  const T cy = Y2 < 0 ? (-p0) - (-o0) : (Y2 >= C.ny ? (v2 - p0) - (v2 - o0) : cv(X, Y2));
  const int b = y * L.nx2 + X, il = (y & 1) * L.half + b, ih = (1 - (y & 1)) * L.half + b;
  const T a = P[il], h = P[ih];
  P[il] = a + T(0.5) * c1 + T(0.25) * (cl + cy);
  P[ih] = h + T(0.5) * c1 + T(0.25) * (ch + cy);
}
template <class T>
__global__ void __launch_bounds__(128) u_correct(ULv L, ULv C, T *P, const T *Pc, const T *Oc, T v2) {
  const unsigned t = blockIdx.x * 128u + threadIdx.x;
  if (t < (unsigned)L.half) correct_at<T>(L, C, P, Pc, Oc, t, v2);
}

// F = lpl(P) + F on one cell per thread
template <class T>
__device__ __forceinline__ void add_lap_at(const ULv &L, const T *P, T *F, unsigned t, T v2) {
  const int c = t >= (unsigned)L.half, b = (int)t - c * L.half, y = udiv(b, L.m_nx);
  const Nbr<T, 1> n = neighbours<T, 1>(P, places_of<1>(L, c, group_of<1>(L, b - y * L.nx2, y)), v2);
  F[t] = lap_of<T, 1>(n, 0, P[t], T(L.inv_dx2)) + F[t];
}
template <class T>
__global__ void __launch_bounds__(128) u_add_lap(ULv L, const T *P, T *F, T v2) {
  const unsigned t = blockIdx.x * 128u + threadIdx.x;
  if (t < (unsigned)(2 * L.half)) add_lap_at<T>(L, P, F, t, v2);
}

// The mixed form's set-up (p_mx_residual): on the finest level (RES) the FP64
// residual, else the FP32 one of the coarser set-up; its 2 x 2 means, formed
// in FP64, and those of P and F to the coarser level.
template <bool RES>
__device__ __forceinline__ void mx_down_at(const ULv &L, const ULv &C, const double *P, const double *F, float *R,
                                           double *Pc, double *Fc, float *Rc, unsigned t, double v2) {
  const int nx = 2 * C.nx2, Y = udiv(t >> 1, C.m_nx), X = (int)t - Y * nx;
  double r[4], w[4], f[4];
  if (RES) {
    const Quad<double> q = quad<double>(L, P, F, X, Y, v2);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      r[k] = q.f[k] - q.a[k];
      w[k] = q.w[k];
      f[k] = q.f[k];
      R[q.at[k]] = (float)r[k];
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int i = didx(L, 2 * X + (k & 1), 2 * Y + (k >> 1));
      r[k] = (double)R[i];
      w[k] = P[i];
      f[k] = F[i];
    }
  }
  const int i = didx(C, X, Y);
  Rc[i] = (float)quarter(r[0], r[1], r[2], r[3]);
  Pc[i] = quarter(w[0], w[1], w[2], w[3]);
  Fc[i] = quarter(f[0], f[1], f[2], f[3]);
}
template <bool RES>
__global__ void __launch_bounds__(128) u_mx_down(ULv L, ULv C, const double *P, const double *F, float *R, double *Pc,
                                                 double *Fc, float *Rc, double v2) {
  const unsigned t = blockIdx.x * 128u + threadIdx.x;
  if (t < (unsigned)(2 * C.half)) mx_down_at<RES>(L, C, P, F, R, Pc, Fc, Rc, t, v2);
}
__global__ void __launch_bounds__(256) u_mx_acc(double *P, const float *c, int n) {
  for (int k = blockIdx.x * 256 + threadIdx.x; k < n; k += gridDim.x * 256) P[k] = P[k] + (double)c[k];
}

// ---------------------------------------------------------------------------
// The coarsest levels in one block, their arrays in shared memory. A chain of
// dependent phases: a level visit keeps its places in registers, the levels
// of at most UWARP cells per colour run in one warp, and the phases are out
// of line so that the section fits the instruction cache.
struct UCoarse {
  ULv lv[8];       // off: first cell in shared memory
  int goff[8];     // first cell in the global arrays
  int n, nwarp, cells;
  int down, up, base;
};
enum { CU_FMG = 0, CU_FMG_GIVEN, CU_VCYCLE };
struct Team {
  int tid, n;
  bool warp;
  __device__ __forceinline__ void sync() const {
    if (warp) __syncwarp();
    else __syncthreads();
  }
};
template <class T, int V, int K>
__device__ __forceinline__ void cu_visit(const ULv &L, T *P, T *F, int cycles, bool first, T v2, const Team &g) {
  const int n = L.half / V, nv = L.nx2 / V;
  const T dx2 = T(L.dx2), inv = T(L.inv_dx2);
  Places w[2][K];
  Vec<T, V> df[2][K];
#pragma unroll
  for (int k = 0; k < K; k++) {
    const int t = g.tid + k * g.n;
    if (t < n) {
      const int y = udiv(t, V == 1 ? L.m_nx : L.m_nxv);
      const Group gr = group_of<V>(L, (t - y * nv) * V, y);
#pragma unroll
      for (int c = 0; c < 2; c++) {
        w[c][k] = places_of<V>(L, c, gr);
        Vec<T, V> f = ldv<T, V>(F + w[c][k].own);
        if (first) {  // F = lpl(P) + F, before any cell of P changes
          const Nbr<T, V> nb = neighbours<T, V>(P, w[c][k], v2);
          const Vec<T, V> o = ldv<T, V>(P + w[c][k].own);
#pragma unroll
          for (int v = 0; v < V; v++) f.v[v] = lap_of<T, V>(nb, v, o.v[v], inv) + f.v[v];
          *reinterpret_cast<Vec<T, V> *>(F + w[c][k].own) = f;
        }
#pragma unroll
        for (int v = 0; v < V; v++) df[c][k].v[v] = dx2 * f.v[v];
      }
    }
  }
  if (first) g.sync();
#pragma unroll 1
  for (int it = 0; it < cycles; it++) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int c = 1 - h;  // odd half-sweeps first
#pragma unroll
      for (int k = 0; k < K; k++) {
        if (g.tid + k * g.n < n) {
          const Nbr<T, V> nb = neighbours<T, V>(P, w[c][k], v2);
          Vec<T, V> o;
#pragma unroll
          for (int v = 0; v < V; v++) o.v[v] = gsrb_of<T, V>(nb, v, df[c][k].v[v]);
          *reinterpret_cast<Vec<T, V> *>(P + w[c][k].own) = o;
        }
      }
      g.sync();
    }
  }
}
template <class T>
__device__ __noinline__ void cu_gsrb(const ULv &L, T *P, T *F, int cycles, bool first, T v2, const Team &g) {
  if (g.warp) {
    if (L.half <= 32) cu_visit<T, 1, 1>(L, P, F, cycles, first, v2, g);
    else cu_visit<T, 1, UWARP / 32>(L, P, F, cycles, first, v2, g);
  } else if (L.nx2 & 1) {
    cu_visit<T, 1, UCOARSE / 2 / UTHR>(L, P, F, cycles, first, v2, g);
  } else {
    cu_visit<T, 2, UCOARSE / 4 / UTHR>(L, P, F, cycles, first, v2, g);
  }
}
// the residual of level l restricted (p_fr), and the correction to level l
template <class T>
__device__ __noinline__ void cu_down(const UCoarse &D, int l, T *P, T *F, T *O, bool setup, T v2, const Team &g) {
  const ULv &L = D.lv[l], &C = D.lv[l - 1];
  for (int t = g.tid; t < 2 * C.half; t += g.n) {
    if (setup) restrict_at<T, true>(L, C, P + L.off, F + L.off, P + C.off, F + C.off, O + C.off, t, v2);
    else restrict_at<T, false>(L, C, P + L.off, F + L.off, P + C.off, F + C.off, O + C.off, t, v2);
  }
  g.sync();
}
template <class T>
__device__ __noinline__ void cu_up(const UCoarse &D, int l, T *P, const T *O, T v2, const Team &g) {
  const ULv &L = D.lv[l], &C = D.lv[l - 1];
  for (int t = g.tid; t < L.half; t += g.n) correct_at<T>(L, C, P + L.off, P + C.off, O + C.off, t, v2);
  g.sync();
}
// A V-cycle over levels 0..q (mg2_fas_vcycle, :208-254); first: level q has
// just been reached by the restriction.
template <class T>
__device__ __noinline__ void cu_vcycle(const UCoarse &D, T *P, T *F, T *O, int q, bool first, T v2) {
  const Team g{(int)threadIdx.x, UTHR, false}, w{(int)threadIdx.x, 32, true};
  bool fst = first;
  int l = q;
  for (; l >= 1 && l >= D.nwarp; l--) {
    cu_gsrb<T>(D.lv[l], P + D.lv[l].off, F + D.lv[l].off, D.down, fst, v2, g);
    cu_down<T>(D, l, P, F, O, false, v2, g);
    fst = true;
  }
  const int lw = l;
  if (D.nwarp > 0) {
    if (threadIdx.x < 32) {
      for (; l >= 1; l--) {
        cu_gsrb<T>(D.lv[l], P + D.lv[l].off, F + D.lv[l].off, D.down, fst, v2, w);
        cu_down<T>(D, l, P, F, O, false, v2, w);
        fst = true;
      }
      cu_gsrb<T>(D.lv[0], P + D.lv[0].off, F + D.lv[0].off, D.base, fst, v2, w);
      for (l = 1; l <= lw; l++) {
        cu_up<T>(D, l, P, O, v2, w);
        cu_gsrb<T>(D.lv[l], P + D.lv[l].off, F + D.lv[l].off, D.up, false, v2, w);
      }
    }
    __syncthreads();
  } else {
    cu_gsrb<T>(D.lv[0], P + D.lv[0].off, F + D.lv[0].off, D.base, fst, v2, g);
  }
  for (l = lw + 1; l <= q; l++) {
    cu_up<T>(D, l, P, O, v2, g);
    cu_gsrb<T>(D.lv[l], P + D.lv[l].off, F + D.lv[l].off, D.up, false, v2, g);
  }
}
// mode CU_FMG: the FMG's set-up below the top coarse level (its P and
// restricted residual are in the global arrays) and its stages on all coarse
// levels; CU_FMG_GIVEN: the stages for the mixed form's correction (F of all
// levels given, P = 0); CU_VCYCLE: the middle of a V-cycle. last: write
// every level's P and F back (else only the top level's P).
template <class T>
__global__ void __launch_bounds__(UTHR, 1) u_coarse(const __grid_constant__ UCoarse gD, T *gP, T *gF, T *gO, int mode,
                                                    int last, T v2) {
  extern __shared__ double2 u_sm[];
  __shared__ UCoarse D;
  for (int t = threadIdx.x; t < (int)(sizeof(UCoarse) / sizeof(int)); t += UTHR)
    reinterpret_cast<int *>(&D)[t] = reinterpret_cast<const int *>(&gD)[t];
  __syncthreads();
  T *P = reinterpret_cast<T *>(u_sm), *F = P + D.cells, *O = F + D.cells;
  const int top = D.n - 1;
  const Team g{(int)threadIdx.x, UTHR, false};
  for (int l = mode == CU_FMG_GIVEN ? 0 : top; l <= top; l++) {
    const ULv &L = D.lv[l];
    for (int t = threadIdx.x; t < 2 * L.half; t += UTHR) {
      const T p = mode == CU_FMG_GIVEN ? T(0) : gP[D.goff[l] + t];
      P[L.off + t] = p;
      O[L.off + t] = p;
      F[L.off + t] = gF[D.goff[l] + t];
    }
  }
  __syncthreads();
  if (mode == CU_VCYCLE) {
    cu_vcycle<T>(D, P, F, O, top, true, v2);
  } else {
    if (mode == CU_FMG) {
      for (int l = top; l >= 1; l--) cu_down<T>(D, l, P, F, O, true, v2, g);
      for (int t = threadIdx.x; t < 2 * D.lv[0].half; t += UTHR) add_lap_at<T>(D.lv[0], P + D.lv[0].off, F + D.lv[0].off, t, v2);
      __syncthreads();
    }
    for (int l = 0; l <= top; l++) {
      if (l > 0) cu_up<T>(D, l, P, O, v2, g);
      cu_vcycle<T>(D, P, F, O, l, false, v2);
    }
    if (mode == CU_FMG_GIVEN)
      for (int t = threadIdx.x; t < 2 * D.lv[top].half; t += UTHR) gO[D.goff[top] + t] = T(0);
  }
  for (int l = last ? 0 : top; l <= top; l++) {
    const ULv &L = D.lv[l];
    for (int t = threadIdx.x; t < 2 * L.half; t += UTHR) {
      gP[D.goff[l] + t] = P[L.off + t];
      if (last) gF[D.goff[l] + t] = F[L.off + t];
    }
  }
}

// ---------------------------------------------------------------------------
// Between box slots and dense levels: 64 threads per box, four boxes a block.
struct UAll {
  ULv lv[UMAXLV];
};
struct UBoxes {
  double *cc, *fx, *fy;
  long long cap;
  const int4 *org;  // per id: first cell x, y (0-based), level index, cells per edge
  const int4 *nbr;  // per id: neighbours lx hx ly hy, <= 0 physical
  const int *ids;   // all boxes, level by level
};
__device__ __forceinline__ double *uslot(const UBoxes &B, int iv, int id) { return B.cc + ((size_t)iv * B.cap + id) * USLOT; }

// compute_fld's space charge of the leaves (src/streamer_2d.f90:317-329) into
// their slots and the finest level, and their potential
__global__ void __launch_bounds__(256) u_ingest(UBoxes B, ULv L, int first, int n, double *P, double *F) {
  const int k = blockIdx.x * 4 + (threadIdx.x >> 6), t = threadIdx.x & 63;
  if (k >= n) return;
  const int id = B.ids[first + k];
  const int4 o = B.org[id];
  const int i = t & 7, j = t >> 3, c = i + 1 + 10 * (j + 1);
  const double v = UC_ELEM_CHARGE / UC_EPS0 * (uslot(B, I_ELEC, id)[c] - uslot(B, I_PION, id)[c]);
  uslot(B, I_RHS, id)[c] = v;
  const int d = didx(L, o.x + i, o.y + j);
  F[d] = v;
  P[d] = uslot(B, I_PHI, id)[c];
}

// The solved potential of every box (cells and side ghosts) and the parents'
// right-hand side into the slots; fld_from_pot (src/streamer_2d.f90:346-381)
// and the |E| side ghosts (copies of the neighbours' cells, Neumann on
// walls), pushed by the cells they copy.
__global__ void __launch_bounds__(256) u_finish(UBoxes B, const __grid_constant__ UAll D, int n, int hi, const double *gP,
                                                const double *gF, double v2) {
  const int kb = blockIdx.x * 4 + (threadIdx.x >> 6), t = threadIdx.x & 63;
  if (kb >= n) return;
  const int id = B.ids[kb];
  const int4 o = B.org[id];
  const int nc = o.w, g = nc + 2, sh = 31 - __clz(nc);
  if (t >= nc * nc) return;
  const ULv &L = D.lv[o.z];
  const double *P = gP + L.off;
  const int i = (t & (nc - 1)) + 1, j = (t >> sh) + 1, c = i + g * j, x = o.x + i - 1, y = o.y + j - 1;
  const int nx = 2 * L.nx2;
  const double p = P[didx(L, x, y)];
  const double xl = x > 0 ? P[didx(L, x - 1, y)] : p, xh = x < nx - 1 ? P[didx(L, x + 1, y)] : p;
  const double yl = y > 0 ? P[didx(L, x, y - 1)] : -p, yh = y < L.ny - 1 ? P[didx(L, x, y + 1)] : v2 - p;
  double *phi = uslot(B, I_PHI, id);
  phi[c] = p;
  if (i == 1) phi[c - 1] = xl;
  if (i == nc) phi[c + 1] = xh;
  if (j == 1) phi[c - g] = yl;
  if (j == nc) phi[c + g] = yh;
  if (o.z != hi) uslot(B, I_RHS, id)[c] = gF[L.off + didx(L, x, y)];
  // faces: inv_dr dphi, on box-edge faces 2 inv_dr dphi eps / (eps0 + eps)
  const double *eps = uslot(B, I_EPS, id);
  auto face = [&](double d, bool edge, int own, int other) {
    if (!edge) return L.inv_dr * d;
    const double eo = eps[own], es = eps[other];
    // (eps 1 on both sides: the division by 2 is exact)
    if (eo == 1.0 && es == 1.0) return (2 * L.inv_dr * d) * 0.5;
    return 2 * L.inv_dr * d * eo / (es + eo);
  };
  // low side: own = the ghost (g - s), other = the cell; high side: own = the ghost, other = the cell
  const double fx0 = face(xl - p, i == 1, c - 1, c), fx1 = face(p - xh, i == nc, c + 1, c);
  const double fy0 = face(yl - p, j == 1, c - g, c), fy1 = face(p - yh, j == nc, c + g, c);
  double *fx = B.fx + (B.cap + id) * UFSLOT, *fy = B.fy + (B.cap + id) * UFSLOT;
  fx[(i - 1) + (nc + 1) * (j - 1)] = fx0;
  fy[(i - 1) + nc * (j - 1)] = fy0;
  if (i == nc) fx[nc + (nc + 1) * (j - 1)] = fx1;
  if (j == nc) fy[(i - 1) + nc * nc] = fy1;
  const double sx = fx0 + fx1, sy = fy0 + fy1;
  const double e = sqrt(0.25 * (sx * sx) + 0.25 * (sy * sy));
  double *fld = uslot(B, I_FLD, id);
  fld[c] = e;
  const int4 nb = B.nbr[id];
  if (i == 1) (nb.x > 0 ? uslot(B, I_FLD, nb.x) + (nc + 1 + g * j) : fld + (c - 1))[0] = e;
  if (i == nc) (nb.y > 0 ? uslot(B, I_FLD, nb.y) + g * j : fld + (c + 1))[0] = e;
  if (j == 1) (nb.z > 0 ? uslot(B, I_FLD, nb.z) + (i + g * (nc + 1)) : fld + (c - g))[0] = e;
  if (j == nc) (nb.w > 0 ? uslot(B, I_FLD, nb.w) + i : fld + (c + g))[0] = e;
}

template <class T>
struct Arr {
  T *P, *F, *O, v2;
  int down, up, base;
};

}  // namespace

// ===========================================================================
struct A5Uniform {
  int lo = 0, hi = 0, top = 0;  // levels; lo..top in one block
  std::vector<int> first, count;  // per level index: boxes in the list
  UAll all{};
  UCoarse co{};
  int cells = 0;
  double *d64 = nullptr;
  float *d32 = nullptr;
  int4 *org = nullptr, *nbr = nullptr;
  int *ids = nullptr;
  int n_boxes = 0;
  cudaGraph_t graph[2] = {};
  cudaGraphExec_t exec[2] = {};
  int li(int l) const { return l - lo; }
};

namespace {
unsigned blocks_of(long long n, int per) { return (unsigned)((n + per - 1) / per); }

template <class T>
void sweeps(const A5Uniform *u, const Arr<T> &A, int l, int cycles, bool first, cudaStream_t s) {
  constexpr int VT = 16 / sizeof(T);
  ULv L = u->all.lv[u->li(l)];
  const int V = L.nx2 % VT == 0 ? VT : 1;
  L.m_nxv = magic(L.nx2 / V);
  T *P = A.P + L.off, *F = A.F + L.off;
  const T *O = A.O + L.off;
  const unsigned nb = blocks_of(L.half / V, 256);
  for (int it = 0; it < 2 * cycles; it++) {
    const int c = 1 - (it & 1);
    const bool f = first && it < 2;
    if (V == 1 && f) u_sweep<T, 1, true><<<nb, 256, 0, s>>>(L, P, F, O, c, A.v2);
    else if (V == 1) u_sweep<T, 1, false><<<nb, 256, 0, s>>>(L, P, F, O, c, A.v2);
    else if (f) u_sweep<T, VT, true><<<nb, 256, 0, s>>>(L, P, F, O, c, A.v2);
    else u_sweep<T, VT, false><<<nb, 256, 0, s>>>(L, P, F, O, c, A.v2);
  }
}
template <class T, bool SETUP>
void restrict_level(const A5Uniform *u, const Arr<T> &A, int l, cudaStream_t s) {
  const ULv &L = u->all.lv[u->li(l)], &C = u->all.lv[u->li(l - 1)];
  u_restrict<T, SETUP><<<blocks_of(2 * C.half, 128), 128, 0, s>>>(L, C, A.P + L.off, A.F + L.off, A.P + C.off, A.F + C.off,
                                                                  A.O + C.off, A.v2);
}
template <class T>
void correct_level(const A5Uniform *u, const Arr<T> &A, int l, cudaStream_t s) {
  const ULv &L = u->all.lv[u->li(l)], &C = u->all.lv[u->li(l - 1)];
  u_correct<T><<<blocks_of(L.half, 128), 128, 0, s>>>(L, C, A.P + L.off, A.P + C.off, A.O + C.off, A.v2);
}
template <class T>
void coarse(const A5Uniform *u, const Arr<T> &A, int mode, bool last, cudaStream_t s) {
  UCoarse D = u->co;
  D.down = A.down;
  D.up = A.up;
  D.base = A.base;
  u_coarse<T><<<1, UTHR, 3 * D.cells * sizeof(T), s>>>(D, A.P, A.F, A.O, mode, last ? 1 : 0, A.v2);
}
// mg2_fas_vcycle (afivo/src/m_aX_mg.f90:208-254) from level l0
template <class T>
void vcycle(const A5Uniform *u, const Arr<T> &A, int l0, cudaStream_t s) {
  const int lo = u->lo, top = u->top;
  for (int l = l0; l > std::max(top, lo); l--) {
    sweeps(u, A, l, A.down, l < l0, s);
    restrict_level<T, false>(u, A, l, s);
  }
  if (top >= lo) coarse(u, A, CU_VCYCLE, l0 == u->hi, s);
  else sweeps(u, A, lo, A.base, lo < l0, s);
  for (int l = std::max(top, lo) + 1; l <= l0; l++) {
    correct_level(u, A, l, s);
    sweeps(u, A, l, A.up, false, s);
  }
}
// the stages of mg2_fas_fmg (:186-202) above the one-block section
template <class T>
void stages(const A5Uniform *u, const Arr<T> &A, cudaStream_t s) {
  for (int l = std::max(u->lo, u->top + 1); l <= u->hi; l++) {
    if (l > u->lo) correct_level(u, A, l, s);
    vcycle(u, A, l, s);
  }
}

void enqueue(A5Uniform *u, const A5UniformArgs &a, cudaStream_t s) {
  const int lo = u->lo, hi = u->hi, top = u->top;
  const long long n = u->cells;
  const ULv &H = u->all.lv[u->li(hi)];
  const UBoxes B{a.cc, a.fx, a.fy, a.capacity, u->org, u->nbr, u->ids};
  const Arr<double> A{u->d64, u->d64 + n, u->d64 + 2 * n, 2 * a.voltage, 2, 2, a.n_cycle_base};
  u_ingest<<<blocks_of(u->count[u->li(hi)], 4), 256, 0, s>>>(B, H, u->first[u->li(hi)], u->count[u->li(hi)], A.P + H.off,
                                                             A.F + H.off);
  if (!a.mixed) {
    restrict_level<double, false>(u, A, hi, s);
    for (int l = hi - 1; l > std::max(lo, top); l--) restrict_level<double, true>(u, A, l, s);
    if (top >= lo) {
      coarse(u, A, CU_FMG, false, s);
    } else {
      const ULv &L = u->all.lv[0];
      u_add_lap<double><<<blocks_of(2 * L.half, 128), 128, 0, s>>>(L, A.P + L.off, A.F + L.off, A.v2);
    }
    stages(u, A, s);
  } else {
    const Arr<float> M{u->d32, u->d32 + n, u->d32 + 2 * n, 0.0f, a.sw_down, a.sw_up, a.sw_base};
    for (int pass = 0; pass < a.n_corr; pass++) {
      for (int l = hi; l > lo; l--) {
        const ULv &L = u->all.lv[u->li(l)], &C = u->all.lv[u->li(l - 1)];
        const unsigned nb = blocks_of(2 * C.half, 128);
        if (l == hi)
          u_mx_down<true><<<nb, 128, 0, s>>>(L, C, A.P + L.off, A.F + L.off, M.F + L.off, A.P + C.off, A.F + C.off,
                                             M.F + C.off, A.v2);
        else
          u_mx_down<false><<<nb, 128, 0, s>>>(L, C, A.P + L.off, A.F + L.off, M.F + L.off, A.P + C.off, A.F + C.off,
                                              M.F + C.off, A.v2);
      }
      cudaMemsetAsync(M.P, 0, n * sizeof(float), s);
      if (a.fmg) {
        cudaMemsetAsync(M.O, 0, H.off * sizeof(float), s);
        if (top >= lo) coarse(u, M, CU_FMG_GIVEN, false, s);
        stages(u, M, s);
      } else {
        vcycle(u, M, hi, s);
      }
      u_mx_acc<<<std::min<unsigned>(blocks_of(n, 256), 148 * 8), 256, 0, s>>>(A.P, M.P, (int)n);
    }
  }
  u_finish<<<blocks_of(u->n_boxes, 4), 256, 0, s>>>(B, u->all, u->n_boxes, u->li(hi), A.P, A.F, A.v2);
}
void drop_graphs(A5Uniform *u) {
  for (int k = 0; k < 2; k++) {
    if (u->exec[k]) cudaGraphExecDestroy(u->exec[k]);
    if (u->graph[k]) cudaGraphDestroy(u->graph[k]);
    u->exec[k] = nullptr;
    u->graph[k] = nullptr;
  }
}
}  // namespace

void a5u_destroy(A5Uniform *u) {
  if (!u) return;
  drop_graphs(u);
  for (void *p : {(void *)u->d64, (void *)u->d32, (void *)u->org, (void *)u->nbr, (void *)u->ids})
    if (p) cudaFree(p);
  delete u;
}

void a5u_changed(A5Uniform *u) {
  if (u) drop_graphs(u);
}

// Every level of the tree a complete rectangular grid of same-level
// neighbours with walls around it, leaves on the finest level only (which the
// level lists must say: a box on level lvls_max is in neither list).
A5Uniform *a5u_build(const A5Topo &t, const double *lv_dr, void *stream) {
  const cudaStream_t s = (cudaStream_t)stream;
  const int lo = t.min_lvl, hi = t.max_lvl, nlev = hi - lo + 1;
  if (nlev < 2 || nlev > UMAXLV || hi < 1 || lo > 0) return nullptr;
  auto A = new A5Uniform();
  A->lo = lo;
  A->hi = hi;
  const size_t nid = (size_t)t.max_id + 1;
  std::vector<int4> org(nid, int4{0, 0, 0, 0}), nbr(nid, int4{0, 0, 0, 0});
  std::vector<int> ids;
  long long off = 0;
  auto no = [&]() -> A5Uniform * {
    a5u_destroy(A);
    return nullptr;
  };
  for (int q = 0; q < nlev; q++) {
    const int l = lo + q;
    const std::vector<int> &v = t.ids[q];
    const size_t parents = t.parents[q].size(), leaves = t.leaves[q].size();
    if (v.empty() || (l < hi ? parents != v.size() || leaves != 0 : leaves != v.size() || parents != 0)) return no();
    const int nc = t.meta16[16 * (size_t)v[0] + 14];
    if (l >= 1 ? nc != UNC : nc != UNC >> (1 - l)) return no();
    int mx = 0, my = 0;
    for (int id : v) {
      const int *m = &t.meta16[16 * (size_t)id];
      if (m[14] != nc || m[2] < 1 || m[3] < 1) return no();
      mx = std::max(mx, m[2]);
      my = std::max(my, m[3]);
    }
    if ((long long)mx * my != (long long)v.size()) return no();
    std::vector<int> at((size_t)mx * my, 0);
    for (int id : v) {
      const int *m = &t.meta16[16 * (size_t)id];
      int &a = at[(size_t)(m[2] - 1) + (size_t)mx * (m[3] - 1)];
      if (a) return no();
      a = id;
    }
    for (int id : v) {
      const int *m = &t.meta16[16 * (size_t)id];
      const int x = m[2] - 1, y = m[3] - 1;
      const int want[4] = {x > 0 ? at[x - 1 + (size_t)mx * y] : -1, x < mx - 1 ? at[x + 1 + (size_t)mx * y] : -1,
                           y > 0 ? at[x + (size_t)mx * (y - 1)] : -1, y < my - 1 ? at[x + (size_t)mx * (y + 1)] : -1};
      for (int k = 0; k < 4; k++)
        if (want[k] > 0 ? m[10 + k] != want[k] : m[10 + k] >= 0) return no();
      // the box's cells lie under its parent's
      if (q > 0) {
        const int *pm = &t.meta16[16 * (size_t)m[5]];
        const int s = l >= 2 ? 1 : 0;
        if (m[5] <= 0 || pm[2] != (x >> s) + 1 || pm[3] != (y >> s) + 1) return no();
      }
      org[id] = int4{x * nc, y * nc, q, nc};
      nbr[id] = int4{m[10], m[11], m[12], m[13]};
    }
    A->first.push_back((int)ids.size());
    A->count.push_back((int)v.size());
    ids.insert(ids.end(), v.begin(), v.end());
    const long long nx = (long long)mx * nc, ny = (long long)my * nc;
    if (nx * ny >= 1LL << 29) return no();
    for (const long long d : {nx / 2, nx / 4, nx / 8}) {
      const long long m = magic(d);
      if (d > 1 && (double)(nx * ny) * (double)(m * d - (1LL << 32)) >= 4294967296.0) return no();
    }
    if (q > 0 && (2 * A->all.lv[q - 1].nx2 * 2 != nx || A->all.lv[q - 1].ny * 2 != ny)) return no();
    const double dr = lv_dr[q];
    A->all.lv[q] = ULv{(int)(nx / 2), (int)ny, (int)(nx * ny / 2), magic(nx / 2), 0, (int)off, dr * dr, 1 / (dr * dr), 1 / dr};
    off += nx * ny;
    if (off >= 1LL << 30) return no();
  }
  A->cells = (int)off;
  A->n_boxes = (int)ids.size();
  UCoarse &C = A->co;
  A->top = lo - 1;
  for (int l = lo; l < hi && C.n < 8 && 2 * A->all.lv[l - lo].half <= UCOARSE; l++) {
    const int q = l - lo;
    C.lv[q] = A->all.lv[q];
    C.goff[q] = A->all.lv[q].off;
    C.lv[q].off = C.cells;
    C.lv[q].m_nxv = magic(C.lv[q].nx2 / 2);
    C.cells += 2 * C.lv[q].half;
    if (C.nwarp == q && C.lv[q].half <= UWARP) C.nwarp = q + 1;
    C.n = q + 1;
    A->top = l;
  }
  // (the attribute belongs to the kernel: the most any run's section takes)
  constexpr int sm = 3 * (UCOARSE + UCOARSE / 3 + 4);
  if (3 * C.cells > sm) return no();
  if (cudaFuncSetAttribute(u_coarse<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm * (int)sizeof(double)) != cudaSuccess ||
      cudaFuncSetAttribute(u_coarse<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm * (int)sizeof(float)) != cudaSuccess) {
    cudaGetLastError();
    return no();
  }
  auto up = [&](void **d, const void *h, size_t bytes) {
    return cudaMalloc(d, bytes) == cudaSuccess && (!h || cudaMemcpyAsync(*d, h, bytes, cudaMemcpyHostToDevice, s) == cudaSuccess);
  };
  if (!up((void **)&A->org, org.data(), nid * sizeof(int4)) || !up((void **)&A->nbr, nbr.data(), nid * sizeof(int4)) ||
      !up((void **)&A->ids, ids.data(), ids.size() * sizeof(int)) || !up((void **)&A->d64, nullptr, 3 * off * sizeof(double)) ||
      cudaStreamSynchronize(s) != cudaSuccess) {
    cudaGetLastError();
    return no();
  }
  return A;
}

// Whether a solve with these settings can run: its memory is there and its
// launches are captured. The caller is not capturing the stream.
bool a5u_ready(A5Uniform *u, const A5UniformArgs &a, void *stream) {
  const cudaStream_t s = (cudaStream_t)stream;
  if (a.mixed && !u->d32 && cudaMalloc((void **)&u->d32, 3 * (size_t)u->cells * sizeof(float)) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  const int k = a.mixed ? 1 : 0;
  if (u->exec[k]) return true;
  if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return false;
  enqueue(u, a, s);
  if (cudaStreamEndCapture(s, &u->graph[k]) != cudaSuccess ||
      cudaGraphInstantiate(&u->exec[k], u->graph[k], 0) != cudaSuccess) {
    cudaGetLastError();
    drop_graphs(u);
    return false;
  }
  return true;
}
// compute_fld with a guess on the run's stream, after a5u_ready with the same
// settings.
int a5u_solve(A5Uniform *u, bool mixed, void *stream) {
  return (int)cudaGraphLaunch(u->exec[mixed ? 1 : 0], (cudaStream_t)stream);
}
