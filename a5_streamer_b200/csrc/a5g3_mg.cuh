// Dense multigrid of the 3D octree form, included by a5g3.cu inside its
// namespace: the field solve with a guess (compute_fld's FAS FMG and the
// mixed form's FP32 correction solve).
//
// On a uniform octree every level is complete, so a level is one rectangular
// grid. The solve keeps each level as a dense array split by colour: all
// cells with even x + y + z (0-based), then all with odd, each row holding
// nx / 2 values. A red-black half-sweep then reads one colour and one colour
// of the right-hand side and writes the other colour in place, all with
// unit-stride 16-byte accesses, no neighbour tables and no ghost cells:
// 12 bytes per cell and half-sweep against 24 for box slots with
// interleaved colours, whose rows of 8 of 10 doubles also straddle a third
// sector. HBM bounds the finest level's half-sweeps (level 6: 201 MB each);
// launch latency bounds the small levels', which is why the set-up of the
// coarse right-hand side is part of the sweeps of a level's first visit and
// the smallest levels run in one block (k3d_coarse).
// Measured against the box-slot phases (launch list of one step, us): FP64
// cube of level 4 (262,144 cells) 1,644 -> 926, of it the one-block section
// 880 -> 385 and the half-sweeps 249 -> 185; level 6 (16.8M cells) 11,319 ->
// 8,460, half-sweeps 2,593 -> 1,362 (a finest one 140 -> about 50); mixed
// form on 2 x 1 x 3 base boxes, level 4 (1.6M cells) 2,481 -> 1,454.
//
// Every value is formed by the reference's expression in its order, as the
// slot form does (k3_phase), so both give the same doubles. Notation of a
// level: P potential, F right-hand side, O the potential before the level's
// smoothing (the reference's tmp copy); on a level the restriction has just
// reached, F holds the restricted residual until the first sweeps add the
// level's own operator: F = lpl(O) + F (update_coarse, set_coarse_phi_rhs,
// afivo/src/m_aX_mg.f90:430-523).

// One level: nx2 cells per row and colour, ny, nz rows; magic numbers of the
// divisions by nx2, by nx2 / V (V the vector length of the sweeps) and ny.
struct DLv {
  int nx2, ny, nz, half;
  unsigned m_nx, m_nxv, m_ny;
  long long off;  // first cell in the arrays of all levels
  double dx2, inv_dx2;
};

// t / d through the high product; exact for t * d < 2^32 with m = ceil(2^32 / d)
// (t below the rows or cells of a level, checked at creation), d = 1 apart
__host__ __device__ __forceinline__ unsigned fastdiv(unsigned t, unsigned m) {
#ifdef __CUDA_ARCH__
  return m ? __umulhi(t, m) : t;
#else
  return m ? (unsigned)(((unsigned long long)t * m) >> 32) : t;
#endif
}

template <class T, int V>
struct alignas(sizeof(T) * V) Vec {
  T v[V];
};
template <class T, int V>
__device__ __forceinline__ Vec<T, V> ldv(const T *p) { return *reinterpret_cast<const Vec<T, V> *>(p); }

// The six neighbours of V consecutive cells of one colour in row (y, z),
// from the other colour's array a (own: their own values, which the walls
// mirror: Neumann on x and y, -own at low z, 2 V - own at high z,
// src/streamer_3d.f90:693-715). b: index of the first cell; q: x parity of
// the row's cells of this colour.
template <class T, int V>
struct Nbr {
  Vec<T, V> xm, xp, ym, yp, zm, zp;
};
template <class T, int V>
__device__ __forceinline__ Nbr<T, V> neighbours(const DLv &L, const T *a, const Vec<T, V> &own, int b, int xv, int y,
                                                int z, int q, T v2) {
  Nbr<T, V> n;
  const Vec<T, V> m = ldv<T, V>(a + b);
  const int pl = L.nx2 * L.ny;
  const bool wl = q == 0 && xv == 0, wh = q == 1 && xv + V == L.nx2;
  const T e = (wl || wh) ? (wl ? own.v[0] : own.v[V - 1]) : (q ? a[b + V] : a[b - 1]);
  n.ym = y > 0 ? ldv<T, V>(a + b - L.nx2) : own;
  n.yp = y < L.ny - 1 ? ldv<T, V>(a + b + L.nx2) : own;
  if (z > 0) n.zm = ldv<T, V>(a + b - pl);
  if (z < L.nz - 1) n.zp = ldv<T, V>(a + b + pl);
#pragma unroll
  for (int k = 0; k < V; k++) {
    n.xm.v[k] = q ? m.v[k] : (k == 0 ? e : m.v[k > 0 ? k - 1 : 0]);
    n.xp.v[k] = q ? (k == V - 1 ? e : m.v[k < V - 1 ? k + 1 : 0]) : m.v[k];
    if (z == 0) n.zm.v[k] = -own.v[k];
    if (z == L.nz - 1) n.zp.v[k] = v2 - own.v[k];
  }
  return n;
}

// mg3_box_lpl (:814-848) and mg3_box_gsrb_lpl (:769-811) of element k
template <class T, int V>
__device__ __forceinline__ T lpl_of(const Nbr<T, V> &n, int k, T own, T inv_dx2) {
  T s = n.xm.v[k] + n.xp.v[k];
  s = s + n.ym.v[k];
  s = s + n.yp.v[k];
  s = s + n.zm.v[k];
  s = s + n.zp.v[k];
  return inv_dx2 * (s - 6 * own);
}
template <class T, int V>
__device__ __forceinline__ T gsrb_of(const Nbr<T, V> &n, int k, T dx2f) {
  const T sixth = T(1 / 6.0);
  T s = n.xp.v[k] + n.xm.v[k];
  s = s + n.yp.v[k];
  s = s + n.ym.v[k];
  s = s + n.zp.v[k];
  s = s + n.zm.v[k];
  return sixth * (s - dx2f);
}

// V cells of one half-sweep of colour c (colour 0 on odd half-sweeps: the
// reference's cells with i + j + k + it even, 1-based). FIRST: the level's
// first visit in a cycle, F = lpl(O) + F before it is used; O holds P's
// values from before the visit, so the second colour's operator does not see
// the first colour's update.
template <class T, int V, bool FIRST>
__device__ __forceinline__ void sweep_cells(const DLv &L, T *P, T *F, const T *O, int c, int xv, int r, T v2) {
  const int z = fastdiv(r, L.m_ny), y = r - z * L.ny;
  const int q = (c + y + z) & 1, b = r * L.nx2 + xv;
  T *own = P + c * L.half;
  const T *oth = P + (1 - c) * L.half;
  const bool wall = y == 0 || y == L.ny - 1 || z == 0 || z == L.nz - 1 || xv == 0 || xv + V == L.nx2;
  Vec<T, V> o{};
  if (wall || FIRST) o = ldv<T, V>(own + b);
  Vec<T, V> f = ldv<T, V>(F + c * L.half + b);
  const Nbr<T, V> n = neighbours<T, V>(L, oth, o, b, xv, y, z, q, v2);
  if (FIRST) {
    const T inv = T(L.inv_dx2);
    if (c == 0) {
#pragma unroll
      for (int k = 0; k < V; k++) f.v[k] = lpl_of<T, V>(n, k, o.v[k], inv) + f.v[k];
    } else {
      const Nbr<T, V> n0 = neighbours<T, V>(L, O + (1 - c) * L.half, o, b, xv, y, z, q, v2);
#pragma unroll
      for (int k = 0; k < V; k++) f.v[k] = lpl_of<T, V>(n0, k, o.v[k], inv) + f.v[k];
    }
    *reinterpret_cast<Vec<T, V> *>(F + c * L.half + b) = f;
  }
  const T dx2 = T(L.dx2);
  Vec<T, V> w;
#pragma unroll
  for (int k = 0; k < V; k++) w.v[k] = gsrb_of<T, V>(n, k, dx2 * f.v[k]);
  *reinterpret_cast<Vec<T, V> *>(own + b) = w;
}

template <class T, int V, bool FIRST>
__global__ void __launch_bounds__(256) k3d_sweep(DLv L, T *P, T *F, const T *O, int c, T v2) {
  const unsigned t = blockIdx.x * 256u + threadIdx.x;
  if (t >= (unsigned)(L.half / V)) return;
  const int nv = L.nx2 / V, r = fastdiv(t, L.m_nxv);
  sweep_cells<T, V, FIRST>(L, P, F, O, c, (t - r * nv) * V, r, v2);
}

// Value of cell (x, y, z) of a level
template <class T>
__device__ __forceinline__ T dval(const DLv &L, const T *P, int x, int y, int z) {
  return P[((x + y + z) & 1) * L.half + (z * L.ny + y) * L.nx2 + (x >> 1)];
}
__device__ __forceinline__ int didx(const DLv &L, int x, int y, int z) {
  return ((x + y + z) & 1) * L.half + (z * L.ny + y) * L.nx2 + (x >> 1);
}

// Residual and restriction under one cell (X, Y, Z) of the coarser level C:
// the residuals F - lpl(P) of its eight fine cells and their P, each summed
// in column-major order, times 0.125 (mg3_box_rstr_lpl, :851-893) into C's F
// and into its P and O. ADD: the fine level's F still holds the restricted
// residual (the set-up of the FMG, set_coarse_phi_rhs): F = lpl(P) + F first.
template <class T, bool ADD>
__device__ __forceinline__ void restrict_cell(const DLv &L, const DLv &C, const T *P, T *F, T *Pc, T *Fc, T *Oc, int X,
                                              int Y, int Z, T v2) {
  const T inv = T(L.inv_dx2);
  const int x0 = 2 * X, y0 = 2 * Y, z0 = 2 * Z, nx = 2 * L.nx2, pl = L.nx2 * L.ny;
  // rows of the 4 x 4 neighbourhood in y and z share the x index; per row
  // and colour one load
  const int b = (z0 * L.ny + y0) * L.nx2 + X;
  T w[8], xl[4], xh[4], yl[4], yh[4], zl[4], zh[4], f[8];
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int dx = k & 1, dy = (k >> 1) & 1, dz = k >> 2, col = (dx + dy + dz) & 1;
    const int i = col * L.half + b + dy * L.nx2 + dz * pl;
    w[k] = P[i];
    f[k] = F[i];
  }
#pragma unroll
  for (int m = 0; m < 4; m++) {
    const int a = m & 1, d = m >> 1;
    // x sides: rows dy = a, dz = d; the neighbours' colours are the opposite
    // of the block's cells beside them
    const int row = b + a * L.nx2 + d * pl;
    xl[m] = x0 > 0 ? P[((1 + a + d) & 1) * L.half + row - 1] : w[2 * a + 4 * d];
    xh[m] = x0 + 2 < nx ? P[((a + d) & 1) * L.half + row + 1] : w[1 + 2 * a + 4 * d];
    // y sides: dx = a, dz = d
    yl[m] = Y > 0 ? P[((a + 1 + d) & 1) * L.half + b - L.nx2 + d * pl] : w[a + 4 * d];
    yh[m] = y0 + 2 < L.ny ? P[((a + d) & 1) * L.half + b + 2 * L.nx2 + d * pl] : w[a + 2 + 4 * d];
    // z sides: dx = a, dy = d
    zl[m] = Z > 0 ? P[((a + d + 1) & 1) * L.half + b + d * L.nx2 - pl] : -w[a + 2 * d];
    zh[m] = z0 + 2 < L.nz ? P[((a + d) & 1) * L.half + b + d * L.nx2 + 2 * pl] : v2 - w[a + 2 * d + 4];
  }
  T sr = 0, sp = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int dx = k & 1, dy = (k >> 1) & 1, dz = k >> 2;
    T s = (dx ? w[k - 1] : xl[dy + 2 * dz]) + (dx ? xh[dy + 2 * dz] : w[k + 1]);
    s = s + (dy ? w[k - 2] : yl[dx + 2 * dz]);
    s = s + (dy ? yh[dx + 2 * dz] : w[k + 2]);
    s = s + (dz ? w[k - 4] : zl[dx + 2 * dy]);
    s = s + (dz ? zh[dx + 2 * dy] : w[k + 4]);
    const T a = inv * (s - 6 * w[k]);
    T fk = f[k];
    if (ADD) {
      fk = a + fk;
      const int col = (dx + dy + dz) & 1;
      F[col * L.half + b + dy * L.nx2 + dz * pl] = fk;
    }
    const T r = fk - a;
    sr = k == 0 ? r : sr + r;
    sp = k == 0 ? w[k] : sp + w[k];
  }
  const int i = didx(C, X, Y, Z);
  const T pc = T(0.125) * sp;
  Fc[i] = T(0.125) * sr;
  Pc[i] = pc;
  Oc[i] = pc;
}

// F restricted (init_phi_rhs, :526-549: the mixed form's correction starts
// from 0, so the coarse right-hand side is the restricted residual itself)
template <class T>
__device__ __forceinline__ void restrict_f(const DLv &L, const DLv &C, const T *F, T *Fc, int X, int Y, int Z) {
  const int b = (2 * Z * L.ny + 2 * Y) * L.nx2 + X, pl = L.nx2 * L.ny;
  T s = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int dx = k & 1, dy = (k >> 1) & 1, dz = k >> 2, col = (dx + dy + dz) & 1;
    const T v = F[col * L.half + b + dy * L.nx2 + dz * pl];
    s = k == 0 ? v : s + v;
  }
  Fc[didx(C, X, Y, Z)] = T(0.125) * s;
}

enum { RS_RESID = 0, RS_SETUP, RS_F };
template <class T, int MODE>
__device__ __forceinline__ void restrict_at(const DLv &L, const DLv &C, const T *P, T *F, T *Pc, T *Fc, T *Oc,
                                            unsigned t, T v2) {
  const int nx = 2 * C.nx2;
  const unsigned r = fastdiv(t >> 1, C.m_nx);
  const int X = (int)(t - r * nx), Z = fastdiv(r, C.m_ny), Y = (int)r - Z * C.ny;
  if (MODE == RS_F) restrict_f<T>(L, C, F, Fc, X, Y, Z);
  else restrict_cell<T, MODE == RS_SETUP>(L, C, P, F, Pc, Fc, Oc, X, Y, Z, v2);
}
template <class T, int MODE>
__global__ void __launch_bounds__(128) k3d_restrict(DLv L, DLv C, const T *P, T *F, T *Pc, T *Fc, T *Oc, T v2) {
  const unsigned t = blockIdx.x * 128u + threadIdx.x;
  if (t < (unsigned)(2 * C.half)) restrict_at<T, MODE>(L, C, P, F, Pc, Fc, Oc, t, v2);
}

// correct_children (:374-401) from cell (X, Y, Z) of the coarser level C: its
// correction P - O and those of its six neighbours (ghost cells of both from
// the walls' rule), then phi += 0.25 (c1 + c2x + c2y + c2z)
// (mg3_box_corr_lpl, :714-766) on its eight fine cells. The half-sweep that
// follows overwrites colour 0 without reading it, except where a wall
// mirrors the cell itself, so colour 0 is corrected only beside walls.
// corr: where the correction is kept for the stored right-hand side (0: not),
// the values of the ghost layer above the high-z wall after the cells.
template <class T>
__device__ __forceinline__ void correct_cell(const DLv &L, const DLv &C, T *P, const T *Pc, const T *Oc, T *corr, int X,
                                             int Y, int Z, T v2) {
  const int nx = 2 * C.nx2;
  auto cv = [&](int x, int y, int z) {
    const int i = didx(C, x, y, z);
    return Pc[i] - Oc[i];
  };
  const int i0 = didx(C, X, Y, Z);
  const T p0 = Pc[i0], o0 = Oc[i0], c1 = p0 - o0;
  if (corr) corr[i0] = c1;
  T cx[2], cy[2], cz[2];
  cx[0] = X > 0 ? cv(X - 1, Y, Z) : c1;
  cx[1] = X < nx - 1 ? cv(X + 1, Y, Z) : c1;
  cy[0] = Y > 0 ? cv(X, Y - 1, Z) : c1;
  cy[1] = Y < C.ny - 1 ? cv(X, Y + 1, Z) : c1;
  cz[0] = Z > 0 ? cv(X, Y, Z - 1) : (-p0) - (-o0);
  cz[1] = Z < C.nz - 1 ? cv(X, Y, Z + 1) : (v2 - p0) - (v2 - o0);
  if (corr && Z == C.nz - 1) corr[2 * C.half + Y * nx + X] = cz[1];
  const int b = (2 * Z * L.ny + 2 * Y) * L.nx2 + X, pl = L.nx2 * L.ny;
  const bool wall = X == 0 || X == nx - 1 || Y == 0 || Y == C.ny - 1 || Z == 0 || Z == C.nz - 1;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int dx = k & 1, dy = (k >> 1) & 1, dz = k >> 2, col = (dx + dy + dz) & 1;
    if (col == 0 && !wall) continue;
    T s = c1 + cx[dx];
    s = s + cy[dy];
    s = s + cz[dz];
    T *p = P + col * L.half + b + dy * L.nx2 + dz * pl;
    *p = *p + T(0.25) * s;
  }
}
template <class T>
__device__ __forceinline__ void correct_at(const DLv &L, const DLv &C, T *P, const T *Pc, const T *Oc, T *corr,
                                           unsigned t, T v2) {
  const int nx = 2 * C.nx2;
  const unsigned r = fastdiv(t >> 1, C.m_nx);
  const int X = (int)(t - r * nx), Z = fastdiv(r, C.m_ny), Y = (int)r - Z * C.ny;
  correct_cell<T>(L, C, P, Pc, Oc, corr, X, Y, Z, v2);
}
template <class T>
__global__ void __launch_bounds__(128) k3d_correct(DLv L, DLv C, T *P, const T *Pc, const T *Oc, T *corr, T v2) {
  const unsigned t = blockIdx.x * 128u + threadIdx.x;
  if (t < (unsigned)(2 * C.half)) correct_at<T>(L, C, P, Pc, Oc, corr, t, v2);
}

// F = lpl(P) + F on one cell per thread (the coarsest level's right-hand
// side in the FMG's set-up)
template <class T>
__device__ __forceinline__ void add_lpl_at(const DLv &L, const T *P, T *F, unsigned t, T v2) {
  const int c = t >= (unsigned)L.half, b = (int)t - c * L.half;
  const int r = fastdiv(b, L.m_nx), xv = b - r * L.nx2, z = fastdiv(r, L.m_ny), y = r - z * L.ny;
  const Vec<T, 1> o{{P[t]}};
  const Nbr<T, 1> n = neighbours<T, 1>(L, P + (1 - c) * L.half, o, b, xv, y, z, (c + y + z) & 1, v2);
  F[t] = lpl_of<T, 1>(n, 0, o.v[0], T(L.inv_dx2)) + F[t];
}
template <class T>
__global__ void __launch_bounds__(128) k3d_add_lpl(DLv L, const T *P, T *F, T v2) {
  const unsigned t = blockIdx.x * 128u + threadIdx.x;
  if (t < (unsigned)(2 * L.half)) add_lpl_at<T>(L, P, F, t, v2);
}

// ---------------------------------------------------------------------------
// The coarsest levels (at most DCOARSE cells each) in one block, their three
// arrays in shared memory: a launch runs all their phases between two visits
// of the level above. What bounds it is the chain of some 60 dependent
// phases per V-cycle, each a shared-memory round trip and a barrier, so the
// levels of at most 64 cells per colour run in one warp behind warp barriers
// while the other warps wait once.
constexpr int DCOARSE = 4096, NTHD = 512, DWARP = 64, MAXLV3 = 16;
struct DCoarse {
  DLv lv[8];       // the levels, coarsest first; off: first cell in shared memory
  int n;           // number of levels
  int nwarp;       // the first nwarp of them run in one warp
  int cells;       // cells of all of them
  int down, up, base;
  long long goff[8];   // first cell of each level in the global arrays
  long long coff[8];   // first of its corrections in the correction store
  int ncorr[8];        // corrections kept per level
};
// Entries of one kept correction of level C (its cells and the layer above
// the high-z wall)
__host__ __device__ __forceinline__ long long corr_len(const DLv &C) {
  return 2LL * C.half + 2LL * C.nx2 * C.ny;
}
enum { CD_FMG = 0, CD_FMG_ZERO, CD_VCYCLE };

struct Team {
  int tid, n;
  bool warp;
  __device__ __forceinline__ void sync() const {
    if (warp) __syncwarp();
    else __syncthreads();
  }
};

template <class T, bool FIRST>
__device__ __forceinline__ void cd_sweep(const DLv &L, T *P, T *F, const T *O, int c, T v2, const Team &g) {
  for (int t = g.tid; t < L.half; t += g.n) {
    const int r = fastdiv(t, L.m_nx);
    sweep_cells<T, 1, FIRST>(L, P, F, O, c, t - r * L.nx2, r, v2);
  }
  g.sync();
}
template <class T>
__device__ __forceinline__ void cd_gsrb(const DLv &L, T *P, T *F, const T *O, int cycles, bool first, T v2,
                                        const Team &g) {
  int it = 0;
  if (first) {
    cd_sweep<T, true>(L, P, F, O, 0, v2, g);
    cd_sweep<T, true>(L, P, F, O, 1, v2, g);
    it = 2;
  }
#pragma unroll 1
  for (; it < 2 * cycles; it++) cd_sweep<T, false>(L, P, F, O, it & 1, v2, g);
}

// A V-cycle over levels 0..q (mg3_fas_vcycle, :208-255); first: level q has
// just been reached by the restriction. k: which of a level's kept
// corrections this cycle's are (k + q - l).
template <class T>
__device__ void cd_vcycle(const DCoarse &D, T *P, T *F, T *O, int q, bool first, T *corr, int k, T v2) {
  Team g{(int)threadIdx.x, NTHD, false};
  int l = q;
  bool fst = first;
  const bool w0 = threadIdx.x < 32;
  // down
  for (; l >= 1; l--) {
    if (l < D.nwarp) break;
    const DLv &L = D.lv[l], &C = D.lv[l - 1];
    cd_gsrb<T>(L, P + L.off, F + L.off, O + L.off, D.down, fst, v2, g);
    for (int t = g.tid; t < 2 * C.half; t += g.n)
      restrict_at<T, RS_RESID>(L, C, P + L.off, F + L.off, P + C.off, F + C.off, O + C.off, t, v2);
    g.sync();
    fst = true;
  }
  const int lw = l;  // levels 0..lw: one warp, or level 0 alone on the block
  if (D.nwarp > 0) {
    if (w0) {
      const Team w{(int)threadIdx.x, 32, true};
      for (; l >= 1; l--) {
        const DLv &L = D.lv[l], &C = D.lv[l - 1];
        cd_gsrb<T>(L, P + L.off, F + L.off, O + L.off, D.down, fst, v2, w);
        for (int t = w.tid; t < 2 * C.half; t += 32)
          restrict_at<T, RS_RESID>(L, C, P + L.off, F + L.off, P + C.off, F + C.off, O + C.off, t, v2);
        w.sync();
        fst = true;
      }
      cd_gsrb<T>(D.lv[0], P + D.lv[0].off, F + D.lv[0].off, O + D.lv[0].off, D.base, fst, v2, w);
      for (l = 1; l <= lw; l++) {
        const DLv &L = D.lv[l], &C = D.lv[l - 1];
        const int kk = k + q - l;
        T *cs = corr && kk + 1 < D.ncorr[l - 1] ? corr + D.coff[l - 1] + (kk + 1) * corr_len(C) : nullptr;
        for (int t = w.tid; t < 2 * C.half; t += 32)
          correct_at<T>(L, C, P + L.off, P + C.off, O + C.off, cs, t, v2);
        w.sync();
        cd_gsrb<T>(L, P + L.off, F + L.off, O + L.off, D.up, false, v2, w);
      }
    }
    __syncthreads();
  } else {
    cd_gsrb<T>(D.lv[0], P + D.lv[0].off, F + D.lv[0].off, O + D.lv[0].off, D.base, fst, v2, g);
  }
  // up
  for (l = lw + 1; l <= q; l++) {
    const DLv &L = D.lv[l], &C = D.lv[l - 1];
    const int kk = k + q - l;
    T *cs = corr && kk + 1 < D.ncorr[l - 1] ? corr + D.coff[l - 1] + (kk + 1) * corr_len(C) : nullptr;
    for (int t = g.tid; t < 2 * C.half; t += g.n) correct_at<T>(L, C, P + L.off, P + C.off, O + C.off, cs, t, v2);
    g.sync();
    cd_gsrb<T>(L, P + L.off, F + L.off, O + L.off, D.up, false, v2, g);
  }
}

// mode CD_FMG: the FMG's set-up below the top coarse level (whose P and
// restricted residual are in the global arrays) and its stages on all coarse
// levels; CD_FMG_ZERO: the same for the mixed form's correction (F given,
// P = 0); CD_VCYCLE: the middle of a V-cycle. last: write every level's P
// and F back (else only the top level's P, which the level above corrects
// from).
template <class T>
__global__ void __launch_bounds__(NTHD) k3d_coarse(const __grid_constant__ DCoarse D, T *gP, T *gF, T *gO, T *corr,
                                                   int mode, int k, int last, T v2) {
  extern __shared__ double2 sm_d2[];
  T *P = reinterpret_cast<T *>(sm_d2), *F = P + D.cells, *O = F + D.cells;
  const int top = D.n - 1;
  {
    const DLv &L = D.lv[top];
    for (int t = threadIdx.x; t < 2 * L.half; t += NTHD) {
      const T p = mode == CD_FMG_ZERO ? T(0) : gP[D.goff[top] + t];
      P[L.off + t] = p;
      O[L.off + t] = p;
      F[L.off + t] = gF[D.goff[top] + t];
    }
    if (mode == CD_FMG_ZERO)
      for (int t = threadIdx.x; t < (int)L.off; t += NTHD) P[t] = O[t] = T(0);
  }
  __syncthreads();
  if (mode == CD_VCYCLE) {
    cd_vcycle<T>(D, P, F, O, top, true, corr, k, v2);
  } else {
    for (int l = top; l >= 1; l--) {
      const DLv &L = D.lv[l], &C = D.lv[l - 1];
      for (int t = threadIdx.x; t < 2 * C.half; t += NTHD) {
        if (mode == CD_FMG)
          restrict_at<T, RS_SETUP>(L, C, P + L.off, F + L.off, P + C.off, F + C.off, O + C.off, t, v2);
        else
          restrict_at<T, RS_F>(L, C, P + L.off, F + L.off, P + C.off, F + C.off, O + C.off, t, v2);
      }
      __syncthreads();
    }
    if (mode == CD_FMG) {
      const DLv &L = D.lv[0];
      for (int t = threadIdx.x; t < 2 * L.half; t += NTHD) add_lpl_at<T>(L, P + L.off, F + L.off, t, v2);
      __syncthreads();
    }
    for (int l = 0; l <= top; l++) {
      if (l > 0) {
        const DLv &L = D.lv[l], &C = D.lv[l - 1];
        T *cs = corr && D.ncorr[l - 1] > 0 ? corr + D.coff[l - 1] : nullptr;
        for (int t = threadIdx.x; t < 2 * C.half; t += NTHD)
          correct_at<T>(L, C, P + L.off, P + C.off, O + C.off, cs, t, v2);
        __syncthreads();
      }
      cd_vcycle<T>(D, P, F, O, l, false, corr, 0, v2);
    }
    // the FMG's stage copy of the top level (its O), which the level above reads
    if (mode == CD_FMG_ZERO)
      for (int t = threadIdx.x; t < 2 * D.lv[top].half; t += NTHD) gO[D.goff[top] + t] = T(0);
  }
  for (int l = last ? 0 : top; l <= top; l++) {
    const DLv &L = D.lv[l];
    for (int t = threadIdx.x; t < 2 * L.half; t += NTHD) {
      gP[D.goff[l] + t] = P[L.off + t];
      if (last) gF[D.goff[l] + t] = F[L.off + t];
    }
  }
}

// ---------------------------------------------------------------------------
// Between box slots and dense levels.
struct DAll {
  DLv lv[MAXLV3];
  long long coff[MAXLV3];
  int ncorr[MAXLV3];
};

// compute_fld's space charge on whole slots of the leaves (k3_set_rhs), and
// the leaves' right-hand side and potential into the finest dense level. A
// row of 8 cells goes to two runs of 4, one per colour: 32-byte sectors.
__global__ void __launch_bounds__(NTH3) k3d_ingest(Run3 R, DLv L, const int *ids, double *P, double *F) {
  const int id = ids[blockIdx.x];
  constexpr int g = NC3 + 2;
  const double fac = UC_ELEM_CHARGE / UC_EPS0;
  const double *e = CC(R, I_ELEC, id), *p = CC(R, I_PION, id), *phi = CC(R, I_PHI, id);
  double *rhs = CC(R, I_RHS, id);
  const int4 o = R.org[id];
  for (int c = threadIdx.x; c < SLOT3; c += NTH3) {
    const double v = fac * (e[c] - p[c]);
    rhs[c] = v;
    const int i = c % g, j = (c / g) % g, k = c / (g * g);
    if (i >= 1 && i <= NC3 && j >= 1 && j <= NC3 && k >= 1 && k <= NC3) {
      const int d = didx(L, o.x + i - 1, o.y + j - 1, o.z + k - 1);
      F[d] = v;
      P[d] = phi[c];
    }
  }
}

// The right-hand side of a parent box as the reference leaves it: lpl(phi) +
// restricted residual on the cells, and on every other entry of the slot the
// running sum of what tmp held there at each of the solve's set-ups
// (a3_box_add_cc adds whole boxes, :471-485): |E| of the last field, then
// the kept corrections. Edge and corner entries of phi never change, so
// their corrections are 0. Also those entries of tmp (|E|). One block per
// box; runs before the field kernel overwrites |E|.
__global__ void __launch_bounds__(NTH3) k3d_store_rhs(Run3 R, const __grid_constant__ DAll D, const int *ids,
                                                      const double *F, const double *corr) {
  const int id = ids[blockIdx.x];
  const int4 o = R.org[id];
  const DLv &L = D.lv[o.w];
  const int nc = R.nc[id], g = nc + 2, gs = g * g * g, nx = 2 * L.nx2, nk = D.ncorr[o.w];
  double *rhs = CC(R, I_RHS, id), *fld = CC(R, I_FLD, id);
  const double *phi = CC(R, I_PHI, id), *cr = corr + D.coff[o.w];
  const long long cl = corr_len(L);
  for (int c = threadIdx.x; c < gs; c += NTH3) {
    const int i = c % g, j = (c / g) % g, k = c / (g * g);
    const bool in_x = i >= 1 && i <= nc, in_y = j >= 1 && j <= nc, in_z = k >= 1 && k <= nc;
    int x = o.x + i - 1, y = o.y + j - 1, z = o.z + k - 1;
    if (in_x && in_y && in_z) {
      rhs[c] = F[L.off + didx(L, x, y, z)];
      continue;
    }
    double v = rhs[c] + fld[c];
    if ((int)in_x + (int)in_y + (int)in_z < 2) {
      const double zero = phi[c] - phi[c];
      for (int q = 0; q < nk; q++) v = v + zero;
      fld[c] = zero;
    } else {
      // a side ghost: the facing cell, or the own cell behind a wall
      const bool low = z < 0, high = z >= L.nz;
      x = min(max(x, 0), nx - 1);
      y = min(max(y, 0), L.ny - 1);
      z = min(max(z, 0), L.nz - 1);
      const long long at = high ? 2LL * L.half + y * nx + x : didx(L, x, y, z);
      for (int q = 0; q < nk; q++) {
        const double w = cr[q * cl + at];
        v = v + (low ? -w : w);
      }
    }
    rhs[c] = v;
  }
}

// The potential of every box (cells and side ghosts, sides_bc_pot on the
// walls) from the dense levels into its slot, then fld_from_pot
// (src/streamer_3d.f90:348-393) from the staged values, as fld_box, with
// the |E| side ghosts pushed. Leaves: the edge and corner entries of tmp as
// the FMG's copy leaves them (phi's).
template <int NCT>
__device__ __forceinline__ void field_box(const Run3 &R, const DLv &L, const int4 o, int id, bool leaf, const double *P,
                                          double *sp, double *sfc) {
  const int nc = NCT ? NCT : R.nc[id], g = nc + 2, gs = g * g * g, F = (nc + 1) * nc * nc, nx = 2 * L.nx2;
  const double inv_dr = 1 / R.geo[4 * id + 3], v2 = 2 * R.voltage;
  const double *eps = CC(R, I_EPS, id);
  double *phi = CC(R, I_PHI, id), *fld = CC(R, I_FLD, id);
  for (int c = threadIdx.x; c < gs; c += NTH3) {
    const int i = c % g, j = (c / g) % g, k = c / (g * g);
    const int in = (i >= 1 && i <= nc) + (j >= 1 && j <= nc) + (k >= 1 && k <= nc);
    if (in < 2) {
      if (leaf) fld[c] = phi[c];
      continue;
    }
    const int x = o.x + i - 1, y = o.y + j - 1, z = o.z + k - 1;
    const double p = dval(L, P + L.off, min(max(x, 0), nx - 1), min(max(y, 0), L.ny - 1), min(max(z, 0), L.nz - 1));
    const double v = z < 0 ? -p : (z >= L.nz ? v2 - p : p);
    sp[c] = v;
    phi[c] = v;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < 3 * F; q += NTH3) {
    const int d = q / F, r = q - d * F;
    int i, j, k, a;
    if (d == 0) {
      i = r % (nc + 1) + 1;
      j = (r / (nc + 1)) % nc + 1;
      k = r / ((nc + 1) * nc) + 1;
      a = i;
    } else if (d == 1) {
      i = r % nc + 1;
      j = (r / nc) % (nc + 1) + 1;
      k = r / (nc * (nc + 1)) + 1;
      a = j;
    } else {
      i = r % nc + 1;
      j = (r / nc) % nc + 1;
      k = r / (nc * nc) + 1;
      a = k;
    }
    const int st = d == 0 ? 1 : d == 1 ? g : g * g;
    const int c0 = ix3(g, i, j, k), cm = c0 - st;
    double v;
    if (a == 1) {
      v = 2 * inv_dr * (sp[cm] - sp[c0]) * eps[cm] / (eps[c0] + eps[cm]);
    } else if (a == nc + 1) {
      v = 2 * inv_dr * (sp[cm] - sp[c0]) * eps[c0] / (eps[c0] + eps[cm]);
    } else {
      v = inv_dr * (sp[cm] - sp[c0]);
    }
    sfc[d * FSLOT3 + r] = v;
    FC(R, d, F_FLD, id)[r] = v;
  }
  __syncthreads();
  const int n = nc * nc * nc;
  for (int t = threadIdx.x; t < n; t += NTH3) {
    const int i = t % nc + 1, j = (t / nc) % nc + 1, k = t / (nc * nc) + 1;
    const int xl = (i - 1) + (nc + 1) * ((j - 1) + nc * (k - 1));
    const int yl = (i - 1) + nc * ((j - 1) + (nc + 1) * (k - 1));
    const int zl = (i - 1) + nc * ((j - 1) + nc * (k - 1));
    const double sx = sfc[xl] + sfc[xl + 1];
    const double sy = sfc[FSLOT3 + yl] + sfc[FSLOT3 + yl + nc];
    const double sz = sfc[2 * FSLOT3 + zl] + sfc[2 * FSLOT3 + zl + nc * nc];
    const double v = 0.5 * sqrt(sx * sx + sy * sy + sz * sz);
    fld[ix3(g, i, j, k)] = v;
    push_side_ghosts(R, I_FLD, id, nc, i, j, k, v);
  }
}
__global__ void __launch_bounds__(NTH3) k3d_field(Run3 R, const __grid_constant__ DAll D, const int *ids, int hi,
                                                  const double *P) {
  __shared__ double sp[SLOT3], sfc[3 * FSLOT3];
  const int id = ids[blockIdx.x];
  const int4 o = R.org[id];
  const DLv &L = D.lv[o.w];
  if (R.nc[id] == NC3) field_box<NC3>(R, L, o, id, o.w == hi, P, sp, sfc);
  else field_box<0>(R, L, o, id, o.w == hi, P, sp, sfc);
}

// The mixed form: the FP64 residual of the leaves rhs - lpl(phi), ghost
// neighbours from their sources with the applied voltage, into the FP32
// correction's finest level; and phi += c on the cells of every box with the
// FP64 ghost fill of phi pushed in the same pass.
__global__ void __launch_bounds__(NTH3) k3d_mx_resid(Run3 R, DLv L, const int *ids, float *F) {
  const int id = ids[blockIdx.x];
  constexpr int nc = NC3, g = nc + 2;
  const MG3<double> M{VAR(R, I_PHI), VAR(R, I_RHS), VAR(R, I_FLD), R.voltage};
  const double dr = R.geo[4 * id + 3], inv_dr_sq = 1 / (dr * dr);
  const double *phi = SL(M.phi, id), *rhs = SL(M.rhs, id);
  const int4 o = R.org[id];
  for (int t = threadIdx.x; t < nc * nc * nc; t += NTH3) {
    const int i = t % nc + 1, j = (t / nc) % nc + 1, k = t / (nc * nc) + 1, c = ix3(g, i, j, k);
    F[didx(L, o.x + i - 1, o.y + j - 1, o.z + k - 1)] =
        (float)(rhs[c] - lpl3_src(R, M, id, nc, phi, c, i, j, k, inv_dr_sq));
  }
}
__global__ void __launch_bounds__(NTH3) k3d_mx_acc(Run3 R, const __grid_constant__ DAll D, const int *ids,
                                                   const float *P) {
  const int id = ids[blockIdx.x];
  const int nc = R.nc[id], g = nc + 2, n = nc * nc * nc;
  const int4 o = R.org[id];
  const DLv &L = D.lv[o.w];
  double *phi = CC(R, I_PHI, id);
  for (int t = threadIdx.x; t < n; t += NTH3) {
    const int i = t % nc + 1, j = (t / nc) % nc + 1, k = t / (nc * nc) + 1;
    const int c = ix3(g, i, j, k);
    const double v = phi[c] + (double)dval(L, P + L.off, o.x + i - 1, o.y + j - 1, o.z + k - 1);
    phi[c] = v;
    push_side_ghosts(R, I_PHI, id, nc, i, j, k, v, 1);
  }
}
