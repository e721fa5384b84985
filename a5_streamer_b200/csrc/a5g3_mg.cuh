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
// Measured against the box-slot phases (launch list of one FP64 step, us; the
// step's transport apart, which was fused later): cube of level 4 (262,144
// cells) one-block section 880 -> 246, half-sweeps 249 -> 182; level 6 (16.8M
// cells) half-sweeps 2,593 -> 1,226, a finest one 140 -> 35 (5.8 TB/s).
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

// t / d through the high product; exact for t (m d - 2^32) < 2^32 with m =
// ceil(2^32 / d), which setup_dense checks for every t of a level; m 0 for d = 1
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

// V consecutive cells of one colour: index of the first within the colour,
// parity of the row's y + z, and which of the group's sides are walls.
struct Group {
  int b;
  unsigned fl;
};
enum { GF_ODD = 1, GF_XL = 2, GF_XH = 4, GF_YL = 8, GF_YH = 16, GF_ZL = 32, GF_ZH = 64 };
template <int V>
__device__ __forceinline__ Group group_of(const DLv &L, int xv, int r) {
  const int z = fastdiv(r, L.m_ny), y = r - z * L.ny;
  return Group{r * L.nx2 + xv, (unsigned)((y + z) & 1) | (xv == 0 ? GF_XL : 0) | (xv + V == L.nx2 ? GF_XH : 0) |
                                   (y == 0 ? GF_YL : 0) | (y == L.ny - 1 ? GF_YH : 0) | (z == 0 ? GF_ZL : 0) |
                                   (z == L.nz - 1 ? GF_ZH : 0)};
}

// The six neighbours of group g of colour c from the arrays P (both
// colours). Beyond a wall the group's own values are mirrored (Neumann on x
// and y, -own at low z, 2 V - own at high z, src/streamer_3d.f90:693-715):
// the address is selected, not the branch, so the loads go out together.
template <class T, int V>
struct Nbr {
  Vec<T, V> xm, xp, ym, yp, zm, zp;
};
template <class T, int V>
__device__ __forceinline__ Nbr<T, V> neighbours(const DLv &L, const T *P, int c, const Group &g, T v2) {
  Nbr<T, V> n;
  const T *own = P + c * L.half + g.b, *a = P + (1 - c) * L.half + g.b;
  const int pl = L.nx2 * L.ny;
  const bool q = ((g.fl ^ c) & GF_ODD) != 0;  // x parity of the group's cells
  const Vec<T, V> m = ldv<T, V>(a);
  const T e = *(q ? ((g.fl & GF_XH) ? own + V - 1 : a + V) : ((g.fl & GF_XL) ? own : a - 1));
  n.ym = ldv<T, V>((g.fl & GF_YL) ? own : a - L.nx2);
  n.yp = ldv<T, V>((g.fl & GF_YH) ? own : a + L.nx2);
  n.zm = ldv<T, V>((g.fl & GF_ZL) ? own : a - pl);
  n.zp = ldv<T, V>((g.fl & GF_ZH) ? own : a + pl);
#pragma unroll
  for (int k = 0; k < V; k++) {
    n.xm.v[k] = q ? m.v[k] : (k == 0 ? e : m.v[k > 0 ? k - 1 : 0]);
    n.xp.v[k] = q ? (k == V - 1 ? e : m.v[k < V - 1 ? k + 1 : 0]) : m.v[k];
    if (g.fl & GF_ZL) n.zm.v[k] = -n.zm.v[k];
    if (g.fl & GF_ZH) n.zp.v[k] = v2 - n.zp.v[k];
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

// One group of a half-sweep of colour c (colour 0 on odd half-sweeps: the
// reference's cells with i + j + k + it even, 1-based). FIRST: the level's
// first visit in a cycle, F = lpl(O) + F before it is used; O holds P's
// values from before the visit, so the second colour's operator does not see
// the first colour's update.
template <class T, int V, bool FIRST>
__device__ __forceinline__ void sweep_group(const DLv &L, T *P, T *F, const T *O, int c, const Group &g, T v2) {
  T *own = P + c * L.half + g.b, *fp = F + c * L.half + g.b;
  Vec<T, V> f = ldv<T, V>(fp);
  const Nbr<T, V> n = neighbours<T, V>(L, P, c, g, v2);
  if (FIRST) {
    const T inv = T(L.inv_dx2);
    const Vec<T, V> o = ldv<T, V>(own);
    if (c == 0) {
#pragma unroll
      for (int k = 0; k < V; k++) f.v[k] = lpl_of<T, V>(n, k, o.v[k], inv) + f.v[k];
    } else {
      const Nbr<T, V> n0 = neighbours<T, V>(L, O, c, g, v2);
#pragma unroll
      for (int k = 0; k < V; k++) f.v[k] = lpl_of<T, V>(n0, k, o.v[k], inv) + f.v[k];
    }
    *reinterpret_cast<Vec<T, V> *>(fp) = f;
  }
  const T dx2 = T(L.dx2);
  Vec<T, V> w;
#pragma unroll
  for (int k = 0; k < V; k++) w.v[k] = gsrb_of<T, V>(n, k, dx2 * f.v[k]);
  *reinterpret_cast<Vec<T, V> *>(own) = w;
}

template <class T, int V, bool FIRST>
__global__ void __launch_bounds__(256) k3d_sweep(DLv L, T *P, T *F, const T *O, int c, T v2) {
  const unsigned t = blockIdx.x * 256u + threadIdx.x;
  if (t >= (unsigned)(L.half / V)) return;
  const int nv = L.nx2 / V, r = fastdiv(t, L.m_nxv);
  sweep_group<T, V, FIRST>(L, P, F, O, c, group_of<V>(L, (t - r * nv) * V, r), v2);
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
// The same for one fine cell (x, y, z), where there are more threads than
// coarse cells to spread them over; the first cell of each block of eight
// keeps the correction.
template <class T>
__device__ __forceinline__ void correct_fine(const DLv &L, const DLv &C, T *P, const T *Pc, const T *Oc, T *corr,
                                             unsigned t, T v2) {
  const int c = t >= (unsigned)L.half, b = (int)t - c * L.half, r = fastdiv(b, L.m_nx), z = fastdiv(r, L.m_ny),
            y = r - z * L.ny, x = 2 * (b - r * L.nx2) + ((c + y + z) & 1);
  const int X = x >> 1, Y = y >> 1, Z = z >> 1, nx = 2 * C.nx2;
  const int X2 = X + (x & 1 ? 1 : -1), Y2 = Y + (y & 1 ? 1 : -1), Z2 = Z + (z & 1 ? 1 : -1);
  const int i0 = didx(C, X, Y, Z);
  const T p0 = Pc[i0], o0 = Oc[i0], c1 = p0 - o0;
  const bool wx = X2 < 0 || X2 >= nx, wy = Y2 < 0 || Y2 >= C.ny, zl = Z2 < 0, zh = Z2 >= C.nz;
  const int ix = wx ? i0 : didx(C, X2, Y, Z), iy = wy ? i0 : didx(C, X, Y2, Z), iz = (zl || zh) ? i0 : didx(C, X, Y, Z2);
  T pz = Pc[iz], oz = Oc[iz];
  if (zl) pz = -pz, oz = -oz;
  if (zh) pz = v2 - pz, oz = v2 - oz;
  const T cz = pz - oz;
  T s = c1 + (Pc[ix] - Oc[ix]);
  s = s + (Pc[iy] - Oc[iy]);
  s = s + cz;
  P[t] = P[t] + T(0.25) * s;
  if (corr && !(x & 1) && !(y & 1) && !(z & 1)) corr[i0] = c1;
  if (corr && zh && !(x & 1) && !(y & 1)) corr[2 * C.half + Y * nx + X] = cz;
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
  const int c = t >= (unsigned)L.half, b = (int)t - c * L.half, r = fastdiv(b, L.m_nx);
  const Nbr<T, 1> n = neighbours<T, 1>(L, P, c, group_of<1>(L, b - r * L.nx2, r), v2);
  F[t] = lpl_of<T, 1>(n, 0, P[t], T(L.inv_dx2)) + F[t];
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
// while the other warps wait once, a level visit keeps its addresses in
// registers, and the phases are out of line: inlined copies overran the
// instruction cache. Per launch on the level-4 cube 64 us with inlined
// phases and addresses formed in every sweep, 41 so (FP64); 38 -> 22 in the
// mixed form on 2 x 1 x 3 base boxes.
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

// The half-sweeps of a level visit. A thread's groups (at most K of each
// colour, V cells each) keep their neighbours' places, their wall flags and
// dx^2 F in registers through the visit: with one block the phases are bound
// by instruction issue and latency, not by shared memory.
struct Places {
  int own, m, e, ym, yp, zm, zp;  // as neighbours(), from the start of the level
  unsigned fl;
};
template <int V>
__device__ __forceinline__ Places places_of(const DLv &L, int c, const Group &g) {
  const int own = c * L.half + g.b, a = (1 - c) * L.half + g.b, pl = L.nx2 * L.ny;
  const bool q = ((g.fl ^ c) & GF_ODD) != 0;
  Places w;
  w.own = own;
  w.m = a;
  w.e = q ? ((g.fl & GF_XH) ? own + V - 1 : a + V) : ((g.fl & GF_XL) ? own : a - 1);
  w.ym = (g.fl & GF_YL) ? own : a - L.nx2;
  w.yp = (g.fl & GF_YH) ? own : a + L.nx2;
  w.zm = (g.fl & GF_ZL) ? own : a - pl;
  w.zp = (g.fl & GF_ZH) ? own : a + pl;
  w.fl = (g.fl & ~(unsigned)GF_ODD) | (q ? GF_ODD : 0);
  return w;
}
template <class T, int V>
__device__ __forceinline__ Nbr<T, V> neighbours_at(const T *P, const Places &w, T v2) {
  Nbr<T, V> n;
  const Vec<T, V> m = ldv<T, V>(P + w.m);
  const T e = P[w.e];
  n.ym = ldv<T, V>(P + w.ym);
  n.yp = ldv<T, V>(P + w.yp);
  n.zm = ldv<T, V>(P + w.zm);
  n.zp = ldv<T, V>(P + w.zp);
  const bool q = w.fl & GF_ODD;
#pragma unroll
  for (int k = 0; k < V; k++) {
    n.xm.v[k] = q ? m.v[k] : (k == 0 ? e : m.v[k > 0 ? k - 1 : 0]);
    n.xp.v[k] = q ? (k == V - 1 ? e : m.v[k < V - 1 ? k + 1 : 0]) : m.v[k];
    if (w.fl & GF_ZL) n.zm.v[k] = -n.zm.v[k];
    if (w.fl & GF_ZH) n.zp.v[k] = v2 - n.zp.v[k];
  }
  return n;
}
template <class T, int V, int K>
__device__ __forceinline__ void cd_visit(const DLv &L, T *P, T *F, int cycles, bool first, T v2, const Team &g) {
  const int n = L.half / V, nv = L.nx2 / V;
  const T dx2 = T(L.dx2), inv = T(L.inv_dx2);
  Places w[2][K];
  Vec<T, V> df[2][K];
#pragma unroll
  for (int k = 0; k < K; k++) {
    const int t = g.tid + k * g.n;
    if (t < n) {
      const int r = fastdiv(t, V == 1 ? L.m_nx : L.m_nxv);
      const Group gr = group_of<V>(L, (t - r * nv) * V, r);
#pragma unroll
      for (int c = 0; c < 2; c++) {
        w[c][k] = places_of<V>(L, c, gr);
        Vec<T, V> f = ldv<T, V>(F + w[c][k].own);
        if (first) {  // F = lpl(P) + F, before any cell of P changes
          const Nbr<T, V> nb = neighbours_at<T, V>(P, w[c][k], v2);
          const Vec<T, V> o = ldv<T, V>(P + w[c][k].own);
#pragma unroll
          for (int v = 0; v < V; v++) f.v[v] = lpl_of<T, V>(nb, v, o.v[v], inv) + f.v[v];
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
    for (int c = 0; c < 2; c++) {
#pragma unroll
      for (int k = 0; k < K; k++) {
        if (g.tid + k * g.n < n) {
          const Nbr<T, V> nb = neighbours_at<T, V>(P, w[c][k], v2);
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
// V = 2 where rows allow it. The block form takes at most DCOARSE / 2 cells
// per colour, the warp form DWARP.
// Out of line: its copies would not fit the instruction cache together.
template <class T>
__device__ __noinline__ void cd_gsrb(const DLv &L, T *P, T *F, int cycles, bool first, T v2, const Team &g) {
  if (g.warp) {
    if (L.half <= 32) cd_visit<T, 1, 1>(L, P, F, cycles, first, v2, g);
    else cd_visit<T, 1, DWARP / 32>(L, P, F, cycles, first, v2, g);
  } else if (L.nx2 & 1) {
    // (rows of odd length: coarse levels of odd base grids only)
    if (first) {
      for (int t = g.tid; t < 2 * L.half; t += g.n) add_lpl_at<T>(L, P, F, t, v2);
      g.sync();
    }
    for (int it = 0; it < 2 * cycles; it++) {
      for (int t = g.tid; t < L.half; t += g.n) {
        const int r = fastdiv(t, L.m_nx);
        sweep_group<T, 1, false>(L, P, F, P, it & 1, group_of<1>(L, t - r * L.nx2, r), v2);
      }
      g.sync();
    }
  } else {
    cd_visit<T, 2, DCOARSE / 4 / NTHD>(L, P, F, cycles, first, v2, g);
  }
}

template <class T>
__device__ __noinline__ void cd_correct(const DLv &L, const DLv &C, T *P, const T *Pc, const T *Oc, T *cs, T v2) {
  if (2 * L.half <= 2 * NTHD) {
    for (int t = threadIdx.x; t < 2 * L.half; t += NTHD) correct_fine<T>(L, C, P, Pc, Oc, cs, t, v2);
  } else {
    for (int t = threadIdx.x; t < 2 * C.half; t += NTHD) correct_at<T>(L, C, P, Pc, Oc, cs, t, v2);
  }
}

// A V-cycle over levels 0..q (mg3_fas_vcycle, :208-255); first: level q has
// just been reached by the restriction. k: which of a level's kept
// corrections this cycle's are (k + q - l).
template <class T>
__device__ __noinline__ void cd_vcycle(const DCoarse &D, T *P, T *F, T *O, int q, bool first, T *corr, int k, T v2) {
  Team g{(int)threadIdx.x, NTHD, false};
  int l = q;
  bool fst = first;
  const bool w0 = threadIdx.x < 32;
  // down
  for (; l >= 1; l--) {
    if (l < D.nwarp) break;
    const DLv &L = D.lv[l], &C = D.lv[l - 1];
    cd_gsrb<T>(L, P + L.off, F + L.off, D.down, fst, v2, g);
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
        cd_gsrb<T>(L, P + L.off, F + L.off, D.down, fst, v2, w);
        for (int t = w.tid; t < 2 * C.half; t += 32)
          restrict_at<T, RS_RESID>(L, C, P + L.off, F + L.off, P + C.off, F + C.off, O + C.off, t, v2);
        w.sync();
        fst = true;
      }
      cd_gsrb<T>(D.lv[0], P + D.lv[0].off, F + D.lv[0].off, D.base, fst, v2, w);
      for (l = 1; l <= lw; l++) {
        const DLv &L = D.lv[l], &C = D.lv[l - 1];
        const int kk = k + q - l;
        T *cs = corr && kk + 1 < D.ncorr[l - 1] ? corr + D.coff[l - 1] + (kk + 1) * corr_len(C) : nullptr;
        for (int t = w.tid; t < 2 * L.half; t += 32)
          correct_fine<T>(L, C, P + L.off, P + C.off, O + C.off, cs, t, v2);
        w.sync();
        cd_gsrb<T>(L, P + L.off, F + L.off, D.up, false, v2, w);
      }
    }
    __syncthreads();
  } else {
    cd_gsrb<T>(D.lv[0], P + D.lv[0].off, F + D.lv[0].off, D.base, fst, v2, g);
  }
  // up
  for (l = lw + 1; l <= q; l++) {
    const DLv &L = D.lv[l], &C = D.lv[l - 1];
    const int kk = k + q - l;
    T *cs = corr && kk + 1 < D.ncorr[l - 1] ? corr + D.coff[l - 1] + (kk + 1) * corr_len(C) : nullptr;
    cd_correct<T>(L, C, P + L.off, P + C.off, O + C.off, cs, v2);
    g.sync();
    cd_gsrb<T>(L, P + L.off, F + L.off, D.up, false, v2, g);
  }
}

// mode CD_FMG: the FMG's set-up below the top coarse level (whose P and
// restricted residual are in the global arrays) and its stages on all coarse
// levels; CD_FMG_ZERO: the same for the mixed form's correction (F given,
// P = 0); CD_VCYCLE: the middle of a V-cycle. last: write every level's P
// and F back (else only the top level's P, which the level above corrects
// from).
template <class T>
__global__ void __launch_bounds__(NTHD, 1) k3d_coarse(const __grid_constant__ DCoarse gD, T *gP, T *gF, T *gO, T *corr,
                                                      int mode, int k, int last, T v2) {
  extern __shared__ double2 sm_d2[];
  // the levels are indexed at run time: their description in shared memory
  __shared__ DCoarse D;
  for (int t = threadIdx.x; t < (int)(sizeof(DCoarse) / sizeof(int)); t += NTHD)
    reinterpret_cast<int *>(&D)[t] = reinterpret_cast<const int *>(&gD)[t];
  __syncthreads();
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
        cd_correct<T>(L, C, P + L.off, P + C.off, O + C.off, cs, v2);
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
__device__ __forceinline__ double space_charge(double e, double p) { return UC_ELEM_CHARGE / UC_EPS0 * (e - p); }

// compute_fld's space charge on whole slots of the leaves (k3_set_rhs), into
// the slots and the finest dense level. A row of 8 cells goes to two runs of
// 4, one per colour: 32-byte sectors.
__global__ void __launch_bounds__(NTH3) k3d_ingest_rhs(Run3 R, DLv L, const int *ids, double *F) {
  const int id = ids[blockIdx.x];
  constexpr int g = NC3 + 2;
  const double *e = CC(R, I_ELEC, id), *p = CC(R, I_PION, id);
  double *rhs = CC(R, I_RHS, id);
  const int4 o = R.org[id];
  for (int c = threadIdx.x; c < SLOT3; c += NTH3) {
    const double v = space_charge(e[c], p[c]);
    rhs[c] = v;
    const int i = c % g, j = (c / g) % g, k = c / (g * g);
    if (i >= 1 && i <= NC3 && j >= 1 && j <= NC3 && k >= 1 && k <= NC3)
      F[didx(L, o.x + i - 1, o.y + j - 1, o.z + k - 1)] = v;
  }
}
// the potential of the boxes in ids into their dense levels
__global__ void __launch_bounds__(NTH3) k3d_ingest_phi(Run3 R, const __grid_constant__ DAll D, const int *ids,
                                                       double *P) {
  const int id = ids[blockIdx.x];
  const int4 o = R.org[id];
  const DLv &L = D.lv[o.w];
  const int nc = R.nc[id], g = nc + 2;
  const double *phi = CC(R, I_PHI, id);
  for (int t = threadIdx.x; t < nc * nc * nc; t += NTH3) {
    const int i = t % nc, j = (t / nc) % nc, k = t / (nc * nc);
    P[L.off + didx(L, o.x + i, o.y + j, o.z + k)] = phi[ix3(g, i + 1, j + 1, k + 1)];
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
      const double *w = cr + (high ? 2LL * L.half + y * nx + x : didx(L, x, y, z));
      for (int q = 0; q < nk; q += 4) {  // four loads in flight, added in order
        double a[4];
#pragma unroll
        for (int m = 0; m < 4; m++) a[m] = q + m < nk ? w[(q + m) * cl] : 0.0;
#pragma unroll
        for (int m = 0; m < 4; m++)
          if (q + m < nk) v = v + (low ? -a[m] : a[m]);
      }
    }
    rhs[c] = v;
  }
}

// Potential at (x, y, z) of a dense level or one cell beyond a wall
// (sides_bc_pot, src/streamer_3d.f90:693-715)
__device__ __forceinline__ double phi_at(const DLv &L, const double *P, int x, int y, int z, double v2) {
  const double p = dval(L, P, min(max(x, 0), 2 * L.nx2 - 1), min(max(y, 0), L.ny - 1), min(max(z, 0), L.nz - 1));
  return z < 0 ? -p : (z >= L.nz ? v2 - p : p);
}
// Field of a face from the potentials beside it (fld_from_pot,
// src/streamer_3d.f90:348-393): on box-edge faces 2 inv_dr dphi eps / (eps0 +
// eps), whose division by 2 is exact where both eps are 1.
__device__ __forceinline__ double face_of(double dphi, double inv_dr, bool edge, double e_own, double e_sum) {
  if (!edge) return inv_dr * dphi;
  if (e_own == 1.0 && e_sum == 2.0) return (2 * inv_dr * dphi) * 0.5;
  return 2 * inv_dr * dphi * e_own / e_sum;
}

// The potential of every box (cells and side ghosts) from the dense levels
// into its slot, then fld_from_pot from the staged values: each thread forms
// the six faces of its cells, so no face passes through shared memory, and
// pushes the |E| side ghosts (level 6: 568 us with staged faces and eps read
// on every face, 468 so). EPS: read eps on the box-edge faces (else it
// is 1 everywhere). tail: the edge and corner entries of the leaves' tmp as
// the FP64 FMG's copy leaves them (phi's).
template <int NCT, bool EPS>
__device__ __forceinline__ void field_box(const Run3 &R, const DLv &L, const int4 o, int id, bool tail, const double *P,
                                          double *sp) {
  const int nc = NCT ? NCT : R.nc[id], g = nc + 2, gs = g * g * g;
  const double inv_dr = 1 / R.geo[4 * id + 3], v2 = 2 * R.voltage;
  const double *eps = CC(R, I_EPS, id);
  double *phi = CC(R, I_PHI, id), *fld = CC(R, I_FLD, id);
  for (int c = threadIdx.x; c < gs; c += NTH3) {
    const int i = c % g, j = (c / g) % g, k = c / (g * g);
    const int in = (i >= 1 && i <= nc) + (j >= 1 && j <= nc) + (k >= 1 && k <= nc);
    if (in < 2) {
      if (tail) fld[c] = phi[c];
      continue;
    }
    const double v = phi_at(L, P + L.off, o.x + i - 1, o.y + j - 1, o.z + k - 1, v2);
    sp[c] = v;
    phi[c] = v;
  }
  __syncthreads();
  const int n = nc * nc * nc;
  double *fx = FC(R, 0, F_FLD, id), *fy = FC(R, 1, F_FLD, id), *fz = FC(R, 2, F_FLD, id);
  for (int t = threadIdx.x; t < n; t += NTH3) {
    const int i = t % nc + 1, j = (t / nc) % nc + 1, k = t / (nc * nc) + 1, c = ix3(g, i, j, k);
    const int pos[3] = {i, j, k}, st[3] = {1, g, g * g};
    double f[3][2];
#pragma unroll
    for (int d = 0; d < 3; d++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        // face h of direction d: between cells cm and c0
        const int c0 = c + h * st[d], cm = c0 - st[d], a = pos[d] + h;
        const bool edge = a == 1 || a == nc + 1;
        double eo = 1.0, es = 2.0;
        if (EPS && edge) {
          eo = eps[a == 1 ? cm : c0];
          es = eps[c0] + eps[cm];
        }
        f[d][h] = face_of(sp[cm] - sp[c0], inv_dr, edge, eo, es);
      }
    const int xl = (i - 1) + (nc + 1) * ((j - 1) + nc * (k - 1));
    const int yl = (i - 1) + nc * ((j - 1) + (nc + 1) * (k - 1));
    const int zl = (i - 1) + nc * ((j - 1) + nc * (k - 1));
    fx[xl] = f[0][0];
    fy[yl] = f[1][0];
    fz[zl] = f[2][0];
    if (i == nc) fx[xl + 1] = f[0][1];
    if (j == nc) fy[yl + nc] = f[1][1];
    if (k == nc) fz[zl + nc * nc] = f[2][1];
    const double sx = f[0][0] + f[0][1], sy = f[1][0] + f[1][1], sz = f[2][0] + f[2][1];
    const double v = 0.5 * sqrt(sx * sx + sy * sy + sz * sz);
    fld[c] = v;
    push_side_ghosts(R, I_FLD, id, nc, i, j, k, v);
  }
}
template <bool EPS>
__global__ void __launch_bounds__(NTH3) k3d_field(Run3 R, const __grid_constant__ DAll D, const int *ids, int hi,
                                                  const double *P) {
  __shared__ double sp[SLOT3];
  const int id = ids[blockIdx.x];
  const int4 o = R.org[id];
  const DLv &L = D.lv[o.w];
  if (R.nc[id] == NC3) field_box<NC3, EPS>(R, L, o, id, o.w == hi, P, sp);
  else field_box<0, EPS>(R, L, o, id, o.w == hi, P, sp);
}

// The mixed form: the FP64 residual F - lpl(P) of the finest level into the
// FP32 correction's right-hand side, and P += c on every cell of every level.
__global__ void __launch_bounds__(256) k3d_mx_resid(DLv L, const double *P, const double *F, float *F32, double v2) {
  const unsigned t = blockIdx.x * 256u + threadIdx.x;
  constexpr int V = 2;
  if (t >= (unsigned)(2 * L.half / V)) return;
  const int c = t >= (unsigned)(L.half / V), u = t - c * (L.half / V);
  const int nv = L.nx2 / V, r = fastdiv(u, L.m_nxv), xv = (u - r * nv) * V;
  const Group g = group_of<V>(L, xv, r);
  const int b = g.b;
  const Vec<double, V> o = ldv<double, V>(P + c * L.half + b), f = ldv<double, V>(F + c * L.half + b);
  const Nbr<double, V> n = neighbours<double, V>(L, P, c, g, v2);
  Vec<float, V> w;
#pragma unroll
  for (int k = 0; k < V; k++) w.v[k] = (float)(f.v[k] - lpl_of<double, V>(n, k, o.v[k], L.inv_dx2));
  *reinterpret_cast<Vec<float, V> *>(F32 + c * L.half + b) = w;
}
__global__ void __launch_bounds__(256) k3d_mx_acc(double *P, const float *c, long long n) {
  for (long long k = blockIdx.x * 256LL + threadIdx.x; k < n; k += gridDim.x * 256LL) P[k] = P[k] + (double)c[k];
}

// ---------------------------------------------------------------------------
// The transport of a time step on the leaves (eps 1 everywhere), one block
// per box. Two kernels replace the old-density copy, the two flux and update
// passes, the average and the space charge of the slot form; what is read
// again only inside the step stays in dense arrays (x fastest): stage 1
// writes n_e, n_i and the right-hand side of the first solve, stage 2 takes
// |E| and the face fields from the dense potential, so that the first solve
// needs no field pass. The parents' densities after stage 1 are never read,
// so only stage 2's are restricted. At level 6 (16.8M cells, launch list):
// copies, fluxes, updates, average and space charge 3,450 us in the slot
// form; here stage 1 640, stage 2 903, k3d_final 311.
struct Stage3 {
  double *e1, *p1, *e2;  // dense densities of the finest level (p: updated in place)
  double *P, *F;         // finest dense level: potential, right-hand side
  DLv L;
};
constexpr int G12 = NC3 + 4, S12 = G12 * G12 * G12;
__device__ __forceinline__ int ix12(int i, int j, int k) { return (i + 1) + G12 * ((j + 1) + G12 * (k + 1)); }
__device__ __forceinline__ size_t nat(const DLv &L, int x, int y, int z) {
  return ((size_t)z * L.ny + y) * (2 * L.nx2) + x;
}
// bytes of shared memory: n_e with two ghost layers, |E|, the fluxes, and in
// stage 2 the potential
template <class T, int STAGE>
constexpr size_t stage_smem() {
  return (STAGE == 2 ? sizeof(double) * S12 : 0) + sizeof(T) * (S12 + SLOT3 + 3 * FSLOT3);
}

// Electron flux through one face (src/streamer_3d.f90:396-554, as
// k3_fluxes): em2, em1 | e0, ep1 the scaled densities along the normal, fm,
// f0 the |E| beside it, fld the face field.
template <class T>
__device__ __forceinline__ double koren_flux(const Run3 &R, T em2, T em1, T e0, T ep1, T fm, T f0, T fld, T fac,
                                             T inv_dr) {
  const LocT<T> loc = lt_locT<T>(R, T(0.5) * (f0 + fm));
  T mobility, diff_coeff;
  lt_pairT<T>(R, C_MOB, loc, mobility, diff_coeff);
  const T v_drift = -mobility * fld;
  const T gradc = e0 - em1;
  const bool neg = v_drift < T(0);
  const T grad2 = neg ? ep1 - e0 : em1 - em2;
  const T lim = koren_mlimT<T>(gradc, grad2), ff = fac * fld;
  T out;
  if (neg) {
    out = v_drift * (e0 - lim);
    if (out < ff) out = ff;
  } else {
    out = v_drift * (em1 + lim);
    if (out > ff) out = ff;
  }
  return (double)(out - diff_coeff * gradc * inv_dr) / (double)dscale<T>();
}

// A thread owns the cells (i, j, k) and (i, j, k + 1) of the box: their low
// faces (and, on 192 threads, one high face of the box) with the direction
// known at compile time, six independent chains per thread. What bounds the
// kernel is instruction issue and the latency of its FP64 chains, not HBM:
// with faces dealt out flat (index divisions, one chain per thread) stage 1
// took 1,621 us and stage 2 1,088 us at level 6.
template <class T, int STAGE>
__global__ void __launch_bounds__(NTH3, 3) k3d_stage(Run3 R, const __grid_constant__ Stage3 S, const int *ids) {
  extern __shared__ double2 sm_d2[];
  constexpr int nc = NC3, g = nc + 2, F = (nc + 1) * nc * nc;
  double *sphi = reinterpret_cast<double *>(sm_d2);
  T *se = reinterpret_cast<T *>(sphi + (STAGE == 2 ? S12 : 0)), *sf = se + S12, *sfx = sf + SLOT3;
  const int id = ids[blockIdx.x];
  const int4 o = R.org[id];
  const DLv &L = S.L;
  const int nx = 2 * L.nx2, tid = threadIdx.x;
  const int i = tid & 7, j = (tid >> 3) & 7, k0 = (tid >> 6) * 2;
  const T ds = dscale<T>();
  const double inv64 = 1 / R.geo[4 * id + 3];
  const T inv_dr = T(inv64);
  const double dt = R.scal[S_DT];
  const double *e = CC(R, I_ELEC, id), *p = CC(R, I_PION, id);
  const int xf0 = i + (nc + 1) * (j + nc * k0), yf0 = i + nc * (j + (nc + 1) * k0), zf0 = i + nc * (j + nc * k0);
  // the box's high face of this thread (tid < 192): direction bd, at (i, j)
  const int bd = tid >> 6;
  const int bq = bd == 0 ? nc + (nc + 1) * (i + nc * j) : bd == 1 ? i + nc * (nc + (nc + 1) * j) : i + nc * (j + nc * nc);
  double fl[2][3], fb = 0;  // face fields
  if (STAGE == 1) {
    // densities saved whole; n_e, |E| and the second ghost layer staged
    double *eo = CC(R, I_ELEC_OLD, id), *po = CC(R, I_PION_OLD, id);
    const double *f = CC(R, I_FLD, id), *phi = CC(R, I_PHI, id);
    double ve[4], vp[4], vf[4], vh[4], vn[2];
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int c = tid + m * NTH3;
      if (c < SLOT3) {
        ve[m] = e[c];
        vf[m] = f[c];
        vp[m] = p[c];
        vh[m] = phi[c];
      }
    }
    const int *nb = R.nbr + 6 * id;
    int dst[2];
#pragma unroll
    for (int m = 0; m < 2; m++) {
      const int t = tid + m * NTH3;
      if (t < 6 * nc * nc) {
        const int s = t >> 6, a = (t & 7) + 1, b = ((t >> 3) & 7) + 1, d = s >> 1;
        const bool hi = s & 1;
        const int n = nb[s];
        // a3_gc2_box: the neighbour's second cell from the shared side, or the own one
        const int q = n > 0 ? (hi ? 2 : nc - 1) : (hi ? nc - 1 : 2), w = hi ? nc + 2 : -1;
        const double *x = n > 0 ? CC(R, I_ELEC, n) : e;
        vn[m] = x[d == 0 ? ix3(g, q, a, b) : d == 1 ? ix3(g, a, q, b) : ix3(g, a, b, q)];
        dst[m] = d == 0 ? ix12(w, a, b) : d == 1 ? ix12(a, w, b) : ix12(a, b, w);
      }
    }
    const double *fx = FC(R, 0, F_FLD, id), *fy = FC(R, 1, F_FLD, id), *fz = FC(R, 2, F_FLD, id);
#pragma unroll
    for (int u = 0; u < 2; u++) {
      fl[u][0] = fx[xf0 + u * (nc + 1) * nc];
      fl[u][1] = fy[yf0 + u * (nc + 1) * nc];
      fl[u][2] = fz[zf0 + u * nc * nc];
    }
    if (tid < 192) fb = (bd == 0 ? fx : bd == 1 ? fy : fz)[bq];
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int c = tid + m * NTH3;
      if (c < SLOT3) {
        eo[c] = ve[m];
        po[c] = vp[m];
        const int ci = c % g, cj = (c / g) % g, ck = c / (g * g);
        se[ix12(ci, cj, ck)] = T(ve[m]) * ds;
        sf[c] = T(vf[m]);
        if (ci >= 1 && ci <= nc && cj >= 1 && cj <= nc && ck >= 1 && ck <= nc)
          S.P[didx(L, o.x + ci - 1, o.y + cj - 1, o.z + ck - 1)] = vh[m];
      }
    }
#pragma unroll
    for (int m = 0; m < 2; m++)
      if (tid + m * NTH3 < 6 * nc * nc) se[dst[m]] = T(vn[m]) * ds;
  } else {
    // n_e with two layers and the potential around the box from the dense
    // arrays; beyond a wall n_e mirrors (a3_gc_neumann, a3_gc2_neumann)
    const double v2 = 2 * R.voltage;
#pragma unroll
    for (int m = 0; m < 7; m++) {
      const int c = tid + m * NTH3;
      if (c >= S12) continue;
      const int ci = c % G12 - 1, cj = (c / G12) % G12 - 1, ck = c / (G12 * G12) - 1;
      const int out = (ci < 1 || ci > nc) + (cj < 1 || cj > nc) + (ck < 1 || ck > nc);
      if (out > 2) continue;
      const int x = o.x + ci - 1, y = o.y + cj - 1, z = o.z + ck - 1;
      if (out <= 1) {
        const int mx = x < 0 ? -1 - x : (x >= nx ? 2 * nx - 1 - x : x);
        const int my = y < 0 ? -1 - y : (y >= L.ny ? 2 * L.ny - 1 - y : y);
        const int mz = z < 0 ? -1 - z : (z >= L.nz ? 2 * L.nz - 1 - z : z);
        se[c] = T(S.e1[nat(L, mx, my, mz)]) * ds;
      }
      sphi[c] = phi_at(L, S.P, x, y, z, v2);
    }
    __syncthreads();
    // |E| of the cells and of the facing cells of the neighbours (a wall's
    // ghost mirrors the cell); faces at multiples of nc are box-edge faces
    auto fields = [&](int ci, int cj, int ck, double lo[3]) {
      const int c = ix12(ci, cj, ck);
      const int pos[3] = {ci, cj, ck}, st[3] = {1, G12, G12 * G12};
      const double v = sphi[c];
      double s3[3];
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const int m = pos[d] & (nc - 1);  // 1: low face, 0: high face on the box edge
        lo[d] = face_of(sphi[c - st[d]] - v, inv64, m == 1, 1.0, 2.0);
        s3[d] = lo[d] + face_of(v - sphi[c + st[d]], inv64, m == 0, 1.0, 2.0);
      }
      return T(0.5 * sqrt(s3[0] * s3[0] + s3[1] * s3[1] + s3[2] * s3[2]));
    };
#pragma unroll
    for (int u = 0; u < 2; u++) sf[ix3(g, i + 1, j + 1, k0 + u + 1)] = fields(i + 1, j + 1, k0 + u + 1, fl[u]);
#pragma unroll
    for (int m = 0; m < 2; m++) {
      const int t = tid + m * NTH3;
      if (t >= 6 * nc * nc) continue;
      const int s = t >> 6, a = (t & 7) + 1, b = ((t >> 3) & 7) + 1, d = s >> 1;
      const bool hi = s & 1;
      const int org = d == 0 ? o.x : d == 1 ? o.y : o.z, end = d == 0 ? nx : d == 1 ? L.ny : L.nz;
      const bool wall = hi ? org + nc >= end : org == 0;
      const int q = hi ? nc + 1 : 0, w = wall ? (hi ? nc : 1) : q;
      double lo[3];
      const T v = d == 0 ? fields(w, a, b, lo) : d == 1 ? fields(a, w, b, lo) : fields(a, b, w, lo);
      sf[d == 0 ? ix3(g, q, a, b) : d == 1 ? ix3(g, a, q, b) : ix3(g, a, b, q)] = v;
    }
    if (tid < 192) {
      const int c = bd == 0 ? ix12(nc + 1, i + 1, j + 1) : bd == 1 ? ix12(i + 1, nc + 1, j + 1) : ix12(i + 1, j + 1, nc + 1);
      fb = face_of(sphi[c - (bd == 0 ? 1 : bd == 1 ? G12 : G12 * G12)] - sphi[c], inv64, true, 1.0, 2.0);
    }
  }
  __syncthreads();
  const T fac = T(-0.8 * UC_EPS0 / (UC_ELEM_CHARGE * dt)) * ds;
  double *ex = FC(R, 0, F_ELEC, id), *ey = FC(R, 1, F_ELEC, id), *ez = FC(R, 2, F_ELEC, id);
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const int c = ix12(i + 1, j + 1, k0 + u + 1), f = ix3(g, i + 1, j + 1, k0 + u + 1);
    const T e0 = se[c], f0 = sf[f];
    const int q[3] = {xf0 + u * (nc + 1) * nc, yf0 + u * (nc + 1) * nc, zf0 + u * nc * nc};
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const int st = d == 0 ? 1 : d == 1 ? G12 : G12 * G12, gt = d == 0 ? 1 : d == 1 ? g : g * g;
      const double v = koren_flux<T>(R, se[c - 2 * st], se[c - st], e0, se[c + st], sf[f - gt], f0, T(fl[u][d]), fac, inv_dr);
      if (STAGE == 2) (d == 0 ? ex : d == 1 ? ey : ez)[q[d]] = v;
      sfx[d * F + q[d]] = T(v);
    }
  }
  if (tid < 192) {
    const int c = bd == 0 ? ix12(nc + 1, i + 1, j + 1) : bd == 1 ? ix12(i + 1, nc + 1, j + 1) : ix12(i + 1, j + 1, nc + 1);
    const int f = bd == 0 ? ix3(g, nc + 1, i + 1, j + 1) : bd == 1 ? ix3(g, i + 1, nc + 1, j + 1) : ix3(g, i + 1, j + 1, nc + 1);
    const int st = bd == 0 ? 1 : bd == 1 ? G12 : G12 * G12, gt = bd == 0 ? 1 : bd == 1 ? g : g * g;
    const double v = koren_flux<T>(R, se[c - 2 * st], se[c - st], se[c], se[c + st], sf[f - gt], sf[f], T(fb), fac, inv_dr);
    if (STAGE == 2) (bd == 0 ? ex : bd == 1 ? ey : ez)[bq] = v;
    sfx[bd * F + bq] = T(v);
  }
  __syncthreads();
  // update_solution (src/streamer_3d.f90:566-615), as k3_update
  const T tdt = T(dt);
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const int x = o.x + i, y = o.y + j, z = o.z + k0 + u, c = ix3(g, i + 1, j + 1, k0 + u + 1);
    const size_t n = nat(L, x, y, z);
    const double e_in = STAGE == 1 ? e[c] : S.e1[n], p_in = STAGE == 1 ? p[c] : S.p1[n];
    const LocT<T> loc = lt_locT<T>(R, sf[c]);
    T alpha, eta;
    lt_pairT<T>(R, C_ALPHA, loc, alpha, eta);
    const T *xf = sfx + xf0 + u * (nc + 1) * nc, *yf = sfx + F + yf0 + u * (nc + 1) * nc, *zf = sfx + 2 * F + zf0 + u * nc * nc;
    const T x0 = xf[0], x1 = xf[1], y0 = yf[0], y1 = yf[nc], z0 = zf[0], z1 = zf[nc * nc];
    T dflux[3];
    dflux[0] = x0 + x1;
    dflux[1] = y0 + y1;
    dflux[2] = z0 + z1;
    const T src = T(0.5) * norm2_3T<T>(dflux) * (alpha - eta);
    T sflux = x0 - x1;
    sflux = sflux + y0;
    sflux = sflux - y1;
    sflux = sflux + z0;
    sflux = sflux - z1;
    sflux = sflux * inv_dr;
    const double ev = e_in + (double)((src + sflux) * tdt);
    const double pv = p_in + (double)(src * tdt);
    if (STAGE == 1) {
      S.e1[n] = ev;
      S.F[didx(L, x, y, z)] = space_charge(ev, pv);
    } else {
      S.e2[n] = ev;
    }
    S.p1[n] = pv;
  }
}

// The end of the transport on the leaves: average_dens
// (src/streamer_3d.f90:557-563) on whole slots, the ghost cells of the
// updated densities from their sources (a3_gc_tree with Neumann sides), and
// the space charge of the second solve. Edge and corner entries are never
// updated: their average is the saved value.
__global__ void __launch_bounds__(NTH3) k3d_final(Run3 R, const __grid_constant__ Stage3 S, const int *ids) {
  const int id = ids[blockIdx.x];
  constexpr int nc = NC3, g = nc + 2;
  const int4 o = R.org[id];
  const DLv &L = S.L;
  double *e = CC(R, I_ELEC, id), *p = CC(R, I_PION, id), *rhs = CC(R, I_RHS, id);
  const double *eo = CC(R, I_ELEC_OLD, id), *po = CC(R, I_PION_OLD, id);
  for (int c = threadIdx.x; c < SLOT3; c += NTH3) {
    const int i = c % g, j = (c / g) % g, k = c / (g * g);
    const int in = (i >= 1 && i <= nc) + (j >= 1 && j <= nc) + (k >= 1 && k <= nc);
    const int x = o.x + i - 1, y = o.y + j - 1, z = o.z + k - 1;
    const double a = eo[c], b = po[c];
    double ev = a, pv = b;
    if (in >= 2) {
      const size_t n = nat(L, min(max(x, 0), 2 * L.nx2 - 1), min(max(y, 0), L.ny - 1), min(max(z, 0), L.nz - 1));
      ev = S.e2[n];
      pv = S.p1[n];
    }
    ev = 0.5 * (ev + a);
    pv = 0.5 * (pv + b);
    const double v = space_charge(ev, pv);
    e[c] = ev;
    p[c] = pv;
    rhs[c] = v;
    if (in == 3) S.F[didx(L, x, y, z)] = v;
  }
}

// a3_restrict_box (afivo/src/m_aX_restrict.f90:67-142) of the dense leaf
// densities into the parents' slots, one block per parent
__global__ void __launch_bounds__(NTH3) k3d_restrict_dens(Run3 R, const __grid_constant__ Stage3 S, const int *ids) {
  const int id = ids[blockIdx.x];
  constexpr int nc = NC3;
  const int4 o = R.org[id];
  const DLv &L = S.L;
  const size_t nx = 2 * L.nx2, pl = nx * L.ny;
  for (int t = threadIdx.x; t < 2 * nc * nc * nc; t += NTH3) {
    const int w = t / (nc * nc * nc), u = t % (nc * nc * nc), i = u % nc, j = (u / nc) % nc, k = u / (nc * nc);
    const double *c = (w ? S.p1 : S.e2) + nat(L, 2 * (o.x + i), 2 * (o.y + j), 2 * (o.z + k));
    double s = c[0];
    s = s + c[1];
    s = s + c[nx];
    s = s + c[nx + 1];
    s = s + c[pl];
    s = s + c[pl + 1];
    s = s + c[pl + nx];
    s = s + c[pl + nx + 1];
    CC(R, w ? I_PION : I_ELEC, id)[ix3(nc + 2, i + 1, j + 1, k + 1)] = 0.125 * s;
  }
}
// The restriction of both densities from level top down to the coarsest,
// all levels' few boxes in one block.
__global__ void __launch_bounds__(1024) k3_restrict_low(Run3 R, int top) {
  for (int l = top; l > R.lo; l--) {
    const Lv v = lv_of(R, l);
    const int hnc = v.nc >> 1, nh = hnc * hnc * hnc;
    for (int t = threadIdx.x; t < 2 * nh * v.n; t += 1024) {
      const int id = v.first + t / (2 * nh), u = t % (2 * nh);
      restrict_item(R, id, v.nc, u % nh, u < nh ? I_ELEC : I_PION);
    }
    __syncthreads();
  }
}
