// vibe-model_gb300/csrc/helmholtz_mg.cu
//
// Right-preconditioned BiCGSTAB (van der Vorst 1992) with a geometric
// multigrid V-cycle as preconditioner, for the reference's Helmholtz
// operator y = -div(a grad x) + b x (src/time/helmholtz.cpp:173-201),
// templated on the working precision (FP32 for the mixed solver, FP64).
//
// Operator in coupling form. For a cell, with W/E/S/N/B/T neighbours,
//   (A x) = cD x + cE (x - xE) + cW (x - xW) + cN (x - xN) + cS (x - xS)
//           + cT (x - xT) + cB (x - xB),
// cE = (a + aE)/2 / dx^2 (0 on the east boundary: the reference's clamp
// makes that flux vanish), cW(i) = cE(i-1), likewise N/S; cT = (a + aT)/2 /
// dz^2 and cB = (a + aB)/2 / dz^2 with the cell's own dz (so A is not
// symmetric on a stretched grid), cD = b.
//
// Multigrid. The vertical couplings dominate (dz << dx), so the smoother is
// a vertical-line Gauss-Seidel: every column solves its tridiagonal system
// exactly with the horizontal neighbours fixed, columns in red-black order
// ((i + j) parity), 32 columns per 256 threads with the column recurrences
// run as scans over 8 level segments (k_smooth_scan); the column LU factors
// are computed once per coefficient set. Coarse grids halve nx and ny and
// keep nz (semi-coarsening); coarse couplings are the 2x2 aggregates: cT,
// cB, cD averaged, the horizontal face couplings summed over the two fine
// faces of the coarse face and divided by 8 (= the rediscretised
// a/(2h)^2). An odd nx or ny leaves a last aggregate of half the width, whose
// equation is kept in the volume-weighted form (sums over the cells there
// are), which keeps the couplings of its faces symmetric. Residuals are restricted by the 2x2 mean (computed and
// restricted in one pass) and corrections prolonged piecewise constant.
// V(1,1) cycle, the coarsest grid smoothed 4 or 8 times in one cluster
// launch. The half sweep before a restriction leaves the residual zero on its
// colour, so only the other colour's is computed and restricted; the one after
// a prolongation overwrites its colour, so the correction is added where it
// reads the other colour and never stored. The
// BiCGSTAB loop runs on the device as a conditional CUDA graph.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "helmholtz.cuh"

namespace vgb {

constexpr int kMgMaxLevels = 8;
constexpr int kMT = 256;
// blocks of the Krylov kernels that reduce (6 x 152 SMs: the occupancy of
// their 256-thread blocks, so the grid-stride loops keep enough loads in flight)
constexpr int kMgRedBlocks = 912;
static_assert(kMgRedBlocks >= kRedBlocks, "dot64 shares the partials");

template <typename T>
struct MgLevel {
  int nx, ny, nz;
  size_t n;
  T *cE, *cN, *cT, *cB, *cD;  // couplings and mass term
  T *lc, *li;                 // column LU: c'_k, 1/denom_k
  T *x, *r;                   // correction, right-hand side
};

template <typename T>
struct MgSolver {
  HGeo g;
  int L = 0;
  MgLevel<T> lv[kMgMaxLevels];
  T *x, *r, *r0, *p, *v, *s, *t, *ph, *sh;  // Krylov vectors (fine level)
  double* part = nullptr;                   // 2 x kMgRedBlocks partial sums
  double* sc = nullptr;                     // device scalars
  unsigned* done = nullptr;                 // blocks of a reducing kernel that are through
  double* hsc = nullptr;                    // pinned host copy
  std::vector<void*> allocs;
  // the iteration loop as a CUDA graph: a WHILE node around one iteration,
  // whose condition the last kernel of the iteration clears (0 = not built
  // yet, 1 = built, -1 = not available: the host loop runs instead)
  int graph_state = 0;
  int coarse_ctas = 0;  // CTAs of the one-cluster coarsest smoothing (0: one launch per half sweep)
  int coarse_sweeps = 8;
  bool coarse_resident = false;  // ... whose CTAs keep their one tile per colour in shared memory
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t gexec = nullptr;
};

namespace {

enum Sc {
  RHO_OLD = 0, ALPHA = 1, OMEGA = 2, RHO_NEW = 3, RV = 4, TS = 5, TT = 6, RR = 7, BREAK = 8,
  ITERS = 9, RTOL2 = 10, MAXIT = 11,  // iterations done; stop test (squared tolerance, iteration limit)
  BETA = 12,                           // the next iteration's (rho_new / rho_old) (alpha / omega)
  NSC = 16
};

__device__ __forceinline__ void cell_of(size_t c, int nx, int ny, int& i, int& j, int& k) {
  if (c <= 0xffffffffull) {  // 32-bit divisions (64-bit ones are long integer sequences)
    const unsigned cu = (unsigned)c, row = cu / (unsigned)nx, plane = row / (unsigned)ny;
    i = (int)(cu - row * (unsigned)nx);
    j = (int)(row - plane * (unsigned)ny);
    k = (int)plane;
    return;
  }
  i = (int)(c % nx);
  const size_t cj = c / nx;
  j = (int)(cj % ny);
  k = (int)(cj / ny);
}

// A x at cell c of level l (coupling form)
template <typename T>
__device__ __forceinline__ T apply_at(const MgLevel<T>& l, const T* __restrict__ x, size_t c, int i, int j, int k) {
  const size_t pl = (size_t)l.nx * l.ny;
  const T xc = x[c];
  T y = l.cD[c] * xc;
  const T ce = l.cE[c], cn = l.cN[c], ct = l.cT[c], cb = l.cB[c];
  if (i + 1 < l.nx) y += ce * (xc - x[c + 1]);
  if (i > 0) y += l.cE[c - 1] * (xc - x[c - 1]);
  if (j + 1 < l.ny) y += cn * (xc - x[c + l.nx]);
  if (j > 0) y += l.cN[c - l.nx] * (xc - x[c - l.nx]);
  if (k + 1 < l.nz) y += ct * (xc - x[c + pl]);
  if (k > 0) y += cb * (xc - x[c - pl]);
  return y;
}

// ---- the FP64 residual of the refinement loop ----
// Tiles of 31 x 8 columns marching up the levels: a warp's 32 lanes hold the
// west-face fluxes of 31 cells and the next one's (by shuffle), nine rows the
// south-face fluxes of eight (through shared memory), and a thread carries its
// lower face: each flux a (x - x) once, the spacings as reciprocals. About 20
// FP64 operations a cell, the bound (one thread per cell with six faces and
// three divisions, in the reference's order, took 539 us at 256 x 256 x 64).
constexpr int kResRows = 8, kResCols = 31;
__global__ void __launch_bounds__(32 * (kResRows + 1)) k_residual64(HGeo g, const double* __restrict__ a,
                                                                    const double* __restrict__ b,
                                                                    const double* __restrict__ f,
                                                                    const double* __restrict__ x,
                                                                    double* __restrict__ r, int xtiles, int kz) {
  __shared__ double sy[2][kResRows + 1][32];
  const int lane = threadIdx.x, row = threadIdx.y;
  const int i0 = (int)(blockIdx.x % (unsigned)xtiles) * kResCols, j0 = (int)(blockIdx.x / (unsigned)xtiles) * kResRows;
  const int k0 = blockIdx.y * kz, k1 = imin(k0 + kz, g.nz);
  const int i = i0 + lane, j = j0 + row;
  const bool in = i < g.nx && j < g.ny;  // (outside: the clamped cell's values, whose fluxes are not used)
  const bool cells = row < kResRows;
  const size_t pl = (size_t)g.nx * g.ny;
  const size_t c = (size_t)imin(j, g.ny - 1) * g.nx + imin(i, g.nx - 1);
  const double hx = 0.5 / (g.dx * g.dx), hy = 0.5 / (g.dy * g.dy), is = g.inv_scale[c];
  size_t o = (size_t)k0 * pl + c;
  double ac = a[o], xc = x[o], fb = 0.0;
  if (cells && k0 > 0) fb = (a[o - pl] + ac) * (xc - x[o - pl]);
  for (int k = k0; k < k1; ++k, o += pl) {
    // boundary faces carry no flux: the south face of row 0, and the faces beyond the grid
    const double fs = (j > 0 && j < g.ny) ? (a[o - g.nx] + ac) * (xc - x[o - g.nx]) : 0.0;
    sy[k & 1][row][lane] = fs;
    double at = 0.0, xt = 0.0, ft = 0.0, fw = 0.0, fe = 0.0;
    if (k + 1 < g.nz) {
      at = a[o + pl];
      xt = x[o + pl];
    }
    if (cells) {
      if (k + 1 < g.nz) ft = (ac + at) * (xt - xc);
      double aw = __shfl_up_sync(0xffffffffu, ac, 1), xw = __shfl_up_sync(0xffffffffu, xc, 1);
      if (lane == 0 && i > 0) {
        aw = a[o - 1];
        xw = x[o - 1];
      }
      if (i > 0 && i < g.nx) fw = (aw + ac) * (xc - xw);
      fe = __shfl_down_sync(0xffffffffu, fw, 1);
    }
    __syncthreads();  // (the buffer of two levels ago was read before the barrier in between)
    if (cells && in && lane < kResCols) {
      const double iz = g.inv_dzeta[k] * is;
      const double hz = (unsigned)__double2hiint(iz) < 0x3ff00000u ? 0.5 * iz * iz : 0.5;  // 1/2 / max(dz, 1)^2
      const double fn = sy[k & 1][row + 1][lane];
      r[o] = f[o] + ((fe - fw) * hx + (fn - fs) * hy + (ft - fb) * hz - b[o] * xc);
    }
    ac = at;
    xc = xt;
    fb = ft;
  }
}

// ---- coefficient set-up ----
template <typename T>
__global__ void k_fine_coefs(HGeo g, const double* __restrict__ a, const double* __restrict__ b, MgLevel<T> l) {
  const size_t n = g.n(), pl = (size_t)g.nx * g.ny;
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    cell_of(c, g.nx, g.ny, i, j, k);
    const double dz = dmax(g.dzeta[k] * g.scale[(size_t)j * g.nx + i], 1.0);
    const double ac = a[c], idx2 = 1.0 / (g.dx * g.dx), idy2 = 1.0 / (g.dy * g.dy), idz2 = 1.0 / (dz * dz);
    l.cE[c] = (T)(i + 1 < g.nx ? 0.5 * (ac + a[c + 1]) * idx2 : 0.0);
    l.cN[c] = (T)(j + 1 < g.ny ? 0.5 * (ac + a[c + g.nx]) * idy2 : 0.0);
    l.cT[c] = (T)(k + 1 < g.nz ? 0.5 * (ac + a[c + pl]) * idz2 : 0.0);
    l.cB[c] = (T)(k > 0 ? 0.5 * (ac + a[c - pl]) * idz2 : 0.0);
    l.cD[c] = (T)b[c];
  }
}

template <typename T>
__global__ void k_coarse_coefs(MgLevel<T> f, MgLevel<T> cl) {
  const size_t pf = (size_t)f.nx * f.ny;
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < cl.n; c += (size_t)gridDim.x * blockDim.x) {
    int I, J, k;
    cell_of(c, cl.nx, cl.ny, I, J, k);
    const size_t f00 = (size_t)k * pf + (size_t)(2 * J) * f.nx + 2 * I;
    const size_t f10 = f00 + 1, f01 = f00 + f.nx, f11 = f01 + 1;
    if (2 * I + 1 < f.nx && 2 * J + 1 < f.ny) {
      // (a face beside a last cell of half the width: centres 1.5 h apart instead of 2 h)
      const T wE = (T)(2 * I + 3 == f.nx ? 1.0 / 6.0 : 0.125), wN = (T)(2 * J + 3 == f.ny ? 1.0 / 6.0 : 0.125);
      cl.cE[c] = (f.cE[f10] + f.cE[f11]) * wE;
      cl.cN[c] = (f.cN[f01] + f.cN[f11]) * wN;
      cl.cT[c] = (f.cT[f00] + f.cT[f10] + f.cT[f01] + f.cT[f11]) * (T)0.25;
      cl.cB[c] = (f.cB[f00] + f.cB[f10] + f.cB[f01] + f.cB[f11]) * (T)0.25;
      cl.cD[c] = (f.cD[f00] + f.cD[f10] + f.cD[f01] + f.cD[f11]) * (T)0.25;
      continue;
    }
    // the last column or row of an odd grid: the same sums over the cells there
    // are, so the equation carries the cell's share of a full one's volume
    const bool x2 = 2 * I + 1 < f.nx, y2 = 2 * J + 1 < f.ny;
    T t = f.cT[f00], bb = f.cB[f00], dd = f.cD[f00], ce = 0, cn = 0;
    if (x2) {
      t += f.cT[f10];
      bb += f.cB[f10];
      dd += f.cD[f10];
      ce = f.cE[f10];  // (no second row: the face of the one there is)
      cn = 0;
    }
    if (y2) {
      t += f.cT[f01];
      bb += f.cB[f01];
      dd += f.cD[f01];
      cn = f.cN[f01];
    }
    cl.cE[c] = ce * (T)(2 * I + 3 == f.nx ? 1.0 / 6.0 : 0.125);
    cl.cN[c] = cn * (T)(2 * J + 3 == f.ny ? 1.0 / 6.0 : 0.125);
    cl.cT[c] = t * (T)0.25;
    cl.cB[c] = bb * (T)0.25;
    cl.cD[c] = dd * (T)0.25;
  }
}

template <typename T>
__device__ __forceinline__ T diag_at(const MgLevel<T>& l, size_t c, int i, int j) {
  T m = l.cD[c] + l.cE[c] + l.cN[c] + l.cT[c] + l.cB[c];
  if (i > 0) m += l.cE[c - 1];
  if (j > 0) m += l.cN[c - l.nx];
  return m;
}

// column LU of (diag, -cB, -cT): denom_k = m_k + cB_k c'_{k-1}, c'_k = -cT_k / denom_k
template <typename T>
__global__ void k_column_lu(MgLevel<T> l) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= l.nx * l.ny) return;
  const int i = col % l.nx, j = col / l.nx;
  const size_t pl = (size_t)l.nx * l.ny;
  T cprev = 0;
  for (int k = 0; k < l.nz; ++k) {
    const size_t c = (size_t)k * pl + col;
    const T den = diag_at(l, c, i, j) + (k > 0 ? l.cB[c] * cprev : (T)0);
    const T inv = (T)1 / den;
    cprev = -l.cT[c] * inv;
    l.li[c] = inv;
    l.lc[c] = cprev;
  }
}

// ---- multigrid kernels ----
// one red-black half sweep of vertical-line Gauss-Seidel on columns with
// (i + j) % 2 == color; zero_nb: the horizontal neighbours are taken as 0
// (first half sweep from a zero initial guess), one thread per column, the
// levels in order (the recurrence carries dp from level to level). Used for
// columns too tall for the tiled form below.
template <typename T>
__global__ void k_smooth(MgLevel<T> l, const T* __restrict__ rhs, T* __restrict__ x, int color, int zero_nb) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= l.nx * l.ny) return;
  const int i = col % l.nx, j = col / l.nx;
  if (((i + j) & 1) != color) return;
  const size_t pl = (size_t)l.nx * l.ny;
  T dp = 0;
  for (int k = 0; k < l.nz; ++k) {
    const size_t c = (size_t)k * pl + col;
    T d = rhs[c];
    if (!zero_nb) {
      if (i + 1 < l.nx) d += l.cE[c] * x[c + 1];
      if (i > 0) d += l.cE[c - 1] * x[c - 1];
      if (j + 1 < l.ny) d += l.cN[c] * x[c + l.nx];
      if (j > 0) d += l.cN[c - l.nx] * x[c - l.nx];
    }
    dp = (d + (k > 0 ? l.cB[c] * dp : (T)0)) * l.li[c];
    x[c] = dp;
  }
  T xn = dp;
  for (int k = l.nz - 1; k-- > 0;) {
    const size_t c = (size_t)k * pl + col;
    xn = x[c] - l.lc[c] * xn;
    x[c] = xn;
  }
}
// The same half sweep, tiled: 256 threads take a tile of 32 columns of the
// colour (the colour's columns numbered row by row, q = j per_row + m, column
// i = 2m + (j + colour) % 2; 32 consecutive q, which at 64 columns per row
// and more lie in one row) and all nz levels.
//   1. loads, coalesced along the row: per level and column the right-hand
//      side d (with the other colour's current neighbours unless zero_nb) and
//      the recurrences' coefficients, A = cB li, B = d li, C = -lc, into
//      shared memory (rows padded to 33 against bank conflicts). The loads
//      of a batch of levels are all issued before any of them is used: their
//      addresses are clamped into the grid and the values masked afterwards,
//      so no branch separates them (one memory round trip per batch);
//   2. the forward recurrence dp_k = A_k dp_(k-1) + B_k and then the back
//      substitution x_k = C_k x_(k+1) + dp_k, each as a scan: a column's
//      levels are cut into 8 segments held by 8 consecutive lanes; every lane
//      composes its segment into one affine map, the maps are scanned across
//      the 8 lanes with shuffles (3 steps), and each lane re-runs its segment
//      from its incoming value;
//   3. coalesced stores.
// A column then costs one memory round trip instead of 2 nz dependent ones.
// The result equals the sequential sweep up to rounding (the scan
// reassociates the recurrence; 2e-7 relative in FP32).
constexpr int kScanRS = 33;  // shared-memory row stride of a tile (32 columns + 1)

template <typename T>
struct ScanTile {
  T *A, *B, *C;
  __device__ ScanTile(T* base, int nz) : A(base), B(base + (size_t)nz * kScanRS), C(base + 2 * (size_t)nz * kScanRS) {}
};

// lane's column of tile t of the colour; false outside the grid
template <typename T>
__device__ __forceinline__ bool tile_column(const MgLevel<T>& l, int t, int color, int lane, int& i, int& j) {
  const int per_row = (l.nx + 1) / 2;
  const int q = t * 32 + lane;
  j = q / per_row;
  i = 2 * (q - j * per_row) + ((j + color) & 1);
  const bool ok = j < l.ny && i < l.nx;
  if (!ok) i = j = 0;
  return ok;
}

// kB: levels per batch and thread (12 kB values in registers, 16 kB with kAdd)
// kAdd: the neighbours' x plus the coarse grid's correction xc (cnx x cny
// columns, piecewise constant over the aggregates)
template <typename T, bool kZeroNb, int kB, bool kAdd = false>
__device__ __forceinline__ void scan_tile_load(const MgLevel<T>& l, const T* __restrict__ rhs,
                                               const T* __restrict__ x, int t, int color, ScanTile<T> st,
                                               int tid, const T* __restrict__ xc = nullptr, int cnx = 0,
                                               size_t cpl = 0) {
  const int nz = l.nz;
  const int lane = tid & 31, w = tid >> 5;
  int i, j;
  const bool ok = tile_column(l, t, color, lane, i, j);
  const size_t pl = (size_t)l.nx * l.ny;
  const int col = j * l.nx + i;
  const bool e = ok && i + 1 < l.nx, wv = ok && i > 0, n = ok && j + 1 < l.ny, so = ok && j > 0;
  const int de = e ? 1 : 0, dw = wv ? 1 : 0, dn = n ? l.nx : 0, ds = so ? l.nx : 0;
  const int ge = (j >> 1) * cnx + ((i + de) >> 1), gw = (j >> 1) * cnx + ((i - dw) >> 1);
  const int gn = ((j + (n ? 1 : 0)) >> 1) * cnx + (i >> 1), gs = ((j - (so ? 1 : 0)) >> 1) * cnx + (i >> 1);
  for (int kb = w; kb < nz; kb += 8 * kB) {
    T rv[kB], ce[kB], xe[kB], cw[kB], xw[kB], cn[kB], xn[kB], cs[kB], xs[kB], li[kB], cb[kB], lc[kB];
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int k = kb + 8 * u;
      const size_t c = (size_t)(k < nz ? k : nz - 1) * pl + col;
      rv[u] = rhs[c];
      if (!kZeroNb) {
        ce[u] = l.cE[c];
        xe[u] = x[c + de];
        cw[u] = l.cE[c - dw];
        xw[u] = x[c - dw];
        cn[u] = l.cN[c];
        xn[u] = x[c + dn];
        cs[u] = l.cN[c - ds];
        xs[u] = x[c - ds];
        if (kAdd) {
          const T* g = xc + (size_t)(k < nz ? k : nz - 1) * cpl;
          xe[u] += g[ge];
          xw[u] += g[gw];
          xn[u] += g[gn];
          xs[u] += g[gs];
        }
      }
      li[u] = l.li[c];
      cb[u] = l.cB[c];
      lc[u] = l.lc[c];
    }
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int k = kb + 8 * u;
      if (k < nz) {
        T d = rv[u];
        if (!kZeroNb) {
          if (e) d += ce[u] * xe[u];
          if (wv) d += cw[u] * xw[u];
          if (n) d += cn[u] * xn[u];
          if (so) d += cs[u] * xs[u];
        }
        st.A[k * kScanRS + lane] = (ok && k > 0) ? cb[u] * li[u] : (T)0;
        st.B[k * kScanRS + lane] = ok ? d * li[u] : (T)0;
        st.C[k * kScanRS + lane] = (ok && k + 1 < nz) ? -lc[u] : (T)0;
      }
    }
  }
}

template <typename T>
__device__ __forceinline__ void scan_tile_solve(int nz, ScanTile<T> st, int tid) {
  const int cl = tid >> 3, sg = tid & 7;  // column, segment: a column's segments in consecutive lanes
  const int S = (nz + 7) / 8, k0 = sg * S, k1 = (k0 + S < nz) ? k0 + S : nz;
  T a = 1, b = 0;
  for (int kq = k0; kq < k1; kq += 8) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = kq + u;
      if (k < k1) {
        const T Ak = st.A[k * kScanRS + cl];
        a = Ak * a;
        b = Ak * b + st.B[k * kScanRS + cl];
      }
    }
  }
#pragma unroll
  for (int off = 1; off < 8; off <<= 1) {
    const T ap = __shfl_up_sync(0xffffffffu, a, off, 8);
    const T bp = __shfl_up_sync(0xffffffffu, b, off, 8);
    if (sg >= off) {
      b = a * bp + b;
      a = a * ap;
    }
  }
  T dp = __shfl_up_sync(0xffffffffu, b, 1, 8);  // dp at the top of the segment below
  if (sg == 0) dp = 0;
  for (int kq = k0; kq < k1; kq += 8) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = kq + u;
      if (k < k1) {
        dp = st.A[k * kScanRS + cl] * dp + st.B[k * kScanRS + cl];
        st.B[k * kScanRS + cl] = dp;
      }
    }
  }
  a = 1;
  b = 0;
  for (int kq = k1 - 1; kq >= k0; kq -= 8) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = kq - u;
      if (k >= k0) {
        const T Ck = st.C[k * kScanRS + cl];
        a = Ck * a;
        b = Ck * b + st.B[k * kScanRS + cl];
      }
    }
  }
#pragma unroll
  for (int off = 1; off < 8; off <<= 1) {
    const T an = __shfl_down_sync(0xffffffffu, a, off, 8);
    const T bn = __shfl_down_sync(0xffffffffu, b, off, 8);
    if (sg + off < 8) {
      b = a * bn + b;
      a = a * an;
    }
  }
  T xv = __shfl_down_sync(0xffffffffu, b, 1, 8);  // x at the bottom of the segment above
  if (sg == 7) xv = 0;
  for (int kq = k1 - 1; kq >= k0; kq -= 8) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = kq - u;
      if (k >= k0) {
        xv = st.C[k * kScanRS + cl] * xv + st.B[k * kScanRS + cl];
        st.B[k * kScanRS + cl] = xv;
      }
    }
  }
}

template <typename T>
__device__ __forceinline__ void scan_tile_store(const MgLevel<T>& l, T* __restrict__ x, int t, int color,
                                                ScanTile<T> st, int tid) {
  const int lane = tid & 31, w = tid >> 5;
  int i, j;
  if (!tile_column(l, t, color, lane, i, j)) return;
  const size_t pl = (size_t)l.nx * l.ny;
  const int col = j * l.nx + i;
#pragma unroll 8
  for (int k = w; k < l.nz; k += 8) x[(size_t)k * pl + col] = st.B[k * kScanRS + lane];
}

template <typename T, bool kZeroNb>
__global__ void __launch_bounds__(256) k_smooth_scan(MgLevel<T> l, const T* __restrict__ rhs, T* __restrict__ x,
                                                     int color) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const ScanTile<T> st(reinterpret_cast<T*>(smem_raw), l.nz);
  scan_tile_load<T, kZeroNb, sizeof(T) == 4 ? 8 : 4>(l, rhs, x, blockIdx.x, color, st, threadIdx.x);
  __syncthreads();
  scan_tile_solve<T>(l.nz, st, threadIdx.x);
  __syncthreads();
  scan_tile_store<T>(l, x, blockIdx.x, color, st, threadIdx.x);
}

// the half sweep after the coarse grid's correction
template <typename T>
__global__ void __launch_bounds__(256) k_smooth_add(MgLevel<T> l, const T* __restrict__ rhs, T* __restrict__ x,
                                                    int color, const T* __restrict__ xc, int cnx, size_t cpl) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const ScanTile<T> st(reinterpret_cast<T*>(smem_raw), l.nz);
  scan_tile_load<T, false, sizeof(T) == 4 ? 4 : 2, true>(l, rhs, x, blockIdx.x, color, st, threadIdx.x, xc, cnx, cpl);
  __syncthreads();
  scan_tile_solve<T>(l.nz, st, threadIdx.x);
  __syncthreads();
  scan_tile_store<T>(l, x, blockIdx.x, color, st, threadIdx.x);
}

// The coarsest grid's smoothing, `sweeps` red-black sweeps (the first
// half sweep from a zero guess), in one launch of one thread-block cluster:
// CTA b takes tiles b, b + gridDim.x, ... of each half sweep, and the
// cluster barrier (release/acquire at cluster scope, so x's global stores
// are seen by the cluster's loads after it) separates the half sweeps; a
// half sweep reads only the other colour, so its tiles are independent.
// Replaces 2 sweeps launches of a few tiles each (16 x 16 x 64: 4 tiles per half
// sweep).
// Four sweeps leave the residuals that eight do where the coarsest grid is short
// (a sweep carries a correction two columns on) and coarse enough that its
// columns couple weakly: 256 x 256 x 64, coarsest 16 x 16 of the fifth level, 2.4e-14
// either way after 7 iterations, 0.25 ms less a solve. Else they do not: 12 x 2000
// x 16, coarsest 6 x 1000, 2.9e-11 and 8.6e-12 after 5; 40 x 30 x 20, coarsest 20 x 15 of
// the second level, 3.3e-10 and 2.0e-11 after 5.
constexpr int kCoarseExtent = 32, kCoarseLevels = 3;
constexpr int kCoarseMaxCtas = 8;  // portable cluster size

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <typename T>
__global__ void __launch_bounds__(256) k_coarse_smooth(MgLevel<T> l, const T* __restrict__ rhs, T* __restrict__ x,
                                                       int sweeps) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const ScanTile<T> st(reinterpret_cast<T*>(smem_raw), l.nz);
  const int ntiles = ((l.nx + 1) / 2 * l.ny + 31) / 32;
  constexpr int kB = sizeof(T) == 4 ? 8 : 4;
  for (int sw = 0; sw < 2 * sweeps; ++sw) {
    const int color = sw & 1;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
      if (sw == 0)
        scan_tile_load<T, true, kB>(l, rhs, x, t, color, st, threadIdx.x);
      else
        scan_tile_load<T, false, kB>(l, rhs, x, t, color, st, threadIdx.x);
      __syncthreads();
      scan_tile_solve<T>(l.nz, st, threadIdx.x);
      __syncthreads();
      scan_tile_store<T>(l, x, t, color, st, threadIdx.x);
      __syncthreads();  // the next tile overwrites the shared memory
    }
    cluster_sync();  // the half sweep's stores before the next half sweep's loads
  }
}

// The same when every CTA has one tile of each colour: the two tiles' right-hand
// side, couplings, factors and x stay in shared memory for all the sweeps, and
// a half sweep reads the other colour's x from the CTA that holds it (its own
// for the east and west neighbours and most of the others) through distributed
// shared memory, so no sweep goes through L2. Same arithmetic. 14 calls of a
// 256 x 256 x 64 solve at 16 x 16 x 64: 30 us each, and 61 us with twice the
// sweeps and x and the couplings read from global memory.
template <typename T>
size_t coarse_resident_smem(int nz) {
  return (size_t)nz * (6 * kScanRS + 12 * 32) * sizeof(T);
}
// x of column (i, j), whose colour is (i + j) % 2, at level offset: the shared
// address in the CTA that holds its tile
template <typename T>
__device__ __forceinline__ unsigned remote_column(const MgLevel<T>& l, unsigned xbase, unsigned colour_stride, int i, int j) {
  const int q = j * ((l.nx + 1) / 2) + (i >> 1);  // (tile_column: i = 2m + (j + colour) % 2)
  const unsigned local = xbase + ((i + j) & 1) * colour_stride + (unsigned)(q & 31) * (unsigned)sizeof(T);
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(q >> 5));
  return r;
}
__device__ __forceinline__ float ld_cluster(unsigned a, float) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ double ld_cluster(unsigned a, double) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
template <typename T>
__global__ void __launch_bounds__(256) k_coarse_resident(MgLevel<T> l, const T* __restrict__ rhs, T* __restrict__ x,
                                                         int sweeps) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* base = reinterpret_cast<T*>(smem_raw);
  const int nz = l.nz, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const size_t sc = (size_t)nz * kScanRS, rc = (size_t)nz * 32;
  T* X = base;            // per colour: the half sweep's right-hand side, then x (scan layout)
  T* AC = base + 2 * sc;  // per colour: A, C (scan layout)
  T* Q = base + 6 * sc;   // per colour: rhs, cE, cW, cN, cS, li
  const size_t pl = (size_t)l.nx * l.ny;
  const unsigned xa = (unsigned)__cvta_generic_to_shared(X), xs = (unsigned)(sc * sizeof(T));
  bool ee[2], ww[2], nn[2], ss[2];
  unsigned ae[2], aw[2], an[2], as[2];  // the neighbours' x, level 0
#pragma unroll
  for (int color = 0; color < 2; ++color) {
    int i, j;
    const bool ok = tile_column(l, blockIdx.x, color, lane, i, j);
    const int col = j * l.nx + i;
    const bool e = ee[color] = ok && i + 1 < l.nx, wv = ww[color] = ok && i > 0;
    const bool n = nn[color] = ok && j + 1 < l.ny, so = ss[color] = ok && j > 0;
    ae[color] = remote_column(l, xa, xs, e ? i + 1 : i, j);
    aw[color] = remote_column(l, xa, xs, wv ? i - 1 : i, j);
    an[color] = remote_column(l, xa, xs, i, n ? j + 1 : j);
    as[color] = remote_column(l, xa, xs, i, so ? j - 1 : j);
    T* A = AC + color * 2 * sc;
    T* q = Q + color * 6 * rc;
    constexpr int kL = 4;  // levels whose loads are all in flight (addresses clamped, values masked)
    const int dw = wv ? 1 : 0, ds = so ? l.nx : 0;
    for (int kb = w; kb < nz; kb += 8 * kL) {
      T v[kL][8];
#pragma unroll
      for (int u = 0; u < kL; ++u) {
        const int k = kb + 8 * u;
        const size_t c = (size_t)(k < nz ? k : nz - 1) * pl + col;
        v[u][0] = rhs[c];
        v[u][1] = l.cE[c];
        v[u][2] = l.cE[c - dw];
        v[u][3] = l.cN[c];
        v[u][4] = l.cN[c - ds];
        v[u][5] = l.li[c];
        v[u][6] = l.cB[c];
        v[u][7] = l.lc[c];
      }
#pragma unroll
      for (int u = 0; u < kL; ++u) {
        const int k = kb + 8 * u, m = k * 32 + lane;
        if (k >= nz) break;
        q[m] = ok ? v[u][0] : (T)0;
        q[rc + m] = e ? v[u][1] : (T)0;
        q[2 * rc + m] = wv ? v[u][2] : (T)0;
        q[3 * rc + m] = n ? v[u][3] : (T)0;
        q[4 * rc + m] = so ? v[u][4] : (T)0;
        q[5 * rc + m] = ok ? v[u][5] : (T)0;
        A[k * kScanRS + lane] = (ok && k > 0) ? v[u][6] * v[u][5] : (T)0;
        A[sc + k * kScanRS + lane] = (ok && k + 1 < nz) ? -v[u][7] : (T)0;
      }
    }
  }
  __syncthreads();
  for (int sw = 0; sw < 2 * sweeps; ++sw) {
    const int color = sw & 1;
    const T* q = Q + color * 6 * rc;
    ScanTile<T> st(X, nz);
    st.B = X + color * sc;
    st.A = AC + color * 2 * sc;
    st.C = st.A + sc;
    constexpr int kB = 8;
    for (int kb = w; kb < nz; kb += 8 * kB) {
      T xe[kB], xw[kB], xn[kB], xv[kB];
      if (sw > 0) {
#pragma unroll
        for (int u = 0; u < kB; ++u) {
          const int k = kb + 8 * u;
          const unsigned o = (unsigned)((k < nz ? k : nz - 1) * kScanRS * (int)sizeof(T));
          xe[u] = ld_cluster(ae[color] + o, (T)0);
          xw[u] = ld_cluster(aw[color] + o, (T)0);
          xn[u] = ld_cluster(an[color] + o, (T)0);
          xv[u] = ld_cluster(as[color] + o, (T)0);
        }
      }
#pragma unroll
      for (int u = 0; u < kB; ++u) {
        const int k = kb + 8 * u;
        if (k < nz) {
          const int m = k * 32 + lane;
          T d = q[m];
          if (sw > 0) {
            if (ee[color]) d += q[rc + m] * xe[u];
            if (ww[color]) d += q[2 * rc + m] * xw[u];
            if (nn[color]) d += q[3 * rc + m] * xn[u];
            if (ss[color]) d += q[4 * rc + m] * xv[u];
          }
          st.B[k * kScanRS + lane] = d * q[5 * rc + m];
        }
      }
    }
    __syncthreads();
    scan_tile_solve<T>(nz, st, tid);
    cluster_sync();  // the half sweep's x before the next half sweep's loads
  }
#pragma unroll
  for (int color = 0; color < 2; ++color) {
    ScanTile<T> st(X, nz);
    st.B = X + color * sc;
    scan_tile_store<T>(l, x, blockIdx.x, color, st, tid);
  }
  // (the last cluster_sync came after every read of a neighbour's shared memory)
}

constexpr size_t kScanSmemMax = 200 * 1024;   // one tile's shared memory, at most
constexpr int kOddTiles = 200;                  // tiles up to which an odd grid is its own coarsest (mg_create)
constexpr int kCoarseMaxTiles = 64;             // tiles per half sweep up to which one cluster smooths the coarsest grid
template <typename T>
size_t scan_smem(int nz) {
  return 3 * (size_t)nz * kScanRS * sizeof(T);
}

// the residual rhs - A x on the fine cells of each coarse cell that the half
// sweep just done (colour 1) did not solve: the two with (i + j) even; the
// mean over the four is the coarse right-hand side
template <typename T>
__global__ void k_resid_restrict(MgLevel<T> f, const T* __restrict__ rhs, const T* __restrict__ x, MgLevel<T> cl) {
  const size_t pf = (size_t)f.nx * f.ny;
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < cl.n; c += (size_t)gridDim.x * blockDim.x) {
    int I, J, k;
    cell_of(c, cl.nx, cl.ny, I, J, k);
    const int i = 2 * I, j = 2 * J;
    const size_t f00 = (size_t)k * pf + (size_t)j * f.nx + i, f11 = f00 + f.nx + 1;
    T t = rhs[f00] - apply_at(f, x, f00, i, j, k);
    // (the last column or row of an odd grid has no such partner)
    if (i + 1 < f.nx && j + 1 < f.ny) t += rhs[f11] - apply_at(f, x, f11, i + 1, j + 1, k);
    cl.r[c] = t * (T)0.25;
  }
}

template <typename T>
__global__ void k_prolong_add(MgLevel<T> f, T* __restrict__ x, MgLevel<T> cl) {
  const size_t pc = (size_t)cl.nx * cl.ny;
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < f.n; c += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    cell_of(c, f.nx, f.ny, i, j, k);
    x[c] += cl.x[(size_t)k * pc + (size_t)(j >> 1) * cl.nx + (i >> 1)];
  }
}

// ---- Krylov kernels ----
// Dot products: an FP32 solver's threads accumulate their partial in FP32
// carrying the products' rounding errors (fmaf) and the sums' (Neumaier), so
// a partial is as accurate as an FP64 sum of the exact products while the
// FP64 pipe (a small fraction of the FP32 rate on this GPU) sees one
// conversion per thread; the partials are then summed in FP64. An FP64
// solver accumulates in FP64.
template <typename T>
struct DotAcc;
template <>
struct DotAcc<float> {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float v) {
    const float t = s + v;
    c += (fabsf(s) >= fabsf(v)) ? (s - t) + v : (v - t) + s;
    s = t;
  }
  __device__ __forceinline__ void prod(float a, float b) {
    const float p = a * b;
    add(p);
    c += fmaf(a, b, -p);
  }
  __device__ __forceinline__ double value() const { return (double)s + (double)c; }
};
template <>
struct DotAcc<double> {
  double s = 0.0;
  __device__ __forceinline__ void prod(double a, double b) { s = fma(a, b, s); }
  __device__ __forceinline__ double value() const { return s; }
};

// the block's sum, in thread 0 (the tree halves the FP64 additions down to one
// warp, which finishes by shuffles)
__device__ __forceinline__ double block_sum(double v, double* sh) {
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int w = kMT / 2; w >= 32; w >>= 1) {
    if ((int)threadIdx.x < w) v = sh[threadIdx.x] = v + sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x < 32)
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  return v;
}

enum Op { OP_INIT = 0, OP_ALPHA = 1, OP_OMEGA = 2, OP_XR = 3 };

// What a reducing kernel needs to finish by itself: the block that ends last
// sums the partials (in block order, whichever it is) and updates the scalars,
// instead of a launch of its own. done: a counter the last block resets.
// use_cond: the iteration runs as the body of a graph WHILE node whose
// condition OP_XR sets (1 = go on, 0 = stop: converged, broken down, or at
// the iteration limit)
struct Finish {
  double *part, *sc;
  unsigned* done;
  cudaGraphConditionalHandle cond;
  int use_cond;
};
__device__ __forceinline__ void finish(const Finish& F, int op, double* sh) {
  __shared__ int last;
  if (threadIdx.x == 0) {
    __threadfence();  // this block's partials before its count
    last = atomicAdd(F.done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double a1 = 0.0, a2 = 0.0;
  for (int q = threadIdx.x; q < (int)gridDim.x; q += kMT) {
    a1 += __ldcg(F.part + q);
    a2 += __ldcg(F.part + kMgRedBlocks + q);
  }
  const double s1 = block_sum(a1, sh);
  __syncthreads();  // sh is used again
  const double s2 = block_sum(a2, sh);
  if (threadIdx.x != 0) return;
  *F.done = 0u;
  double* sc = F.sc;
  if (op == OP_INIT) {
    sc[RR] = s1;
    sc[RHO_NEW] = s1;
    sc[RHO_OLD] = 1.0;
    sc[ALPHA] = 1.0;
    sc[OMEGA] = 1.0;
    sc[BETA] = 0.0;  // (p = v = 0: the first p is r whatever beta is)
    sc[BREAK] = 0.0;
  } else if (op == OP_ALPHA) {
    sc[RV] = s1;
    if (s1 == 0.0 || !isfinite(s1)) {
      sc[BREAK] = 1.0;
      sc[ALPHA] = 0.0;
    } else {
      sc[ALPHA] = sc[RHO_NEW] / s1;
    }
  } else if (op == OP_OMEGA) {
    sc[TS] = s1;
    sc[TT] = s2;
    if (!(s2 > 0.0) || !isfinite(s2)) {
      sc[BREAK] = 1.0;
      sc[OMEGA] = 0.0;
    } else {
      sc[OMEGA] = s1 / s2;
      if (sc[OMEGA] == 0.0) sc[BREAK] = 1.0;
    }
  } else {  // OP_XR
    sc[RR] = s1;
    sc[RHO_OLD] = sc[RHO_NEW];
    sc[RHO_NEW] = s2;
    if (s2 == 0.0 || !isfinite(s1)) sc[BREAK] = 1.0;
    const double ro = sc[RHO_OLD], om = sc[OMEGA];
    sc[BETA] = (ro != 0.0 && om != 0.0) ? (s2 / ro) * (sc[ALPHA] / om) : 0.0;
    sc[ITERS] += 1.0;
    if (F.use_cond) {
      const bool stop = sc[BREAK] != 0.0 || !(s1 > sc[RTOL2]) || sc[ITERS] >= sc[MAXIT];
      cudaGraphSetConditional(F.cond, stop ? 0u : 1u);
    }
  }
}
template <typename T>
__global__ void k_init(const double* __restrict__ r64, double inv, size_t n, T* r, T* r0, T* x, T* p, T* v, Finish F) {
  __shared__ double sh[kMT];
  DotAcc<T> acc;
  for (size_t q = blockIdx.x * (size_t)kMT + threadIdx.x; q < n; q += (size_t)gridDim.x * kMT) {
    const T rv = (T)(r64[q] * inv);
    r[q] = rv;
    r0[q] = rv;
    x[q] = 0;
    p[q] = 0;
    v[q] = 0;
    acc.prod(rv, rv);
  }
  const double s = block_sum(acc.value(), sh);
  if (threadIdx.x == 0) {
    F.part[blockIdx.x] = s;
    F.part[kMgRedBlocks + blockIdx.x] = 0.0;
  }
  __syncthreads();
  finish(F, OP_INIT, sh);
}

// p = r + beta (p - omega v), beta from the previous iteration's scalars
template <typename T>
__global__ void k_upd_p(const T* __restrict__ r, T* __restrict__ p, const T* __restrict__ v, size_t n,
                        const double* __restrict__ sc) {
  const T b = (T)sc[BETA], om = (T)sc[OMEGA];
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x)
    p[q] = r[q] + b * (p[q] - om * v[q]);
}

// y = A xin, partials of (w1, y) [and (y, y) when two]
template <typename T, bool kTwo>
__global__ void k_apply_dot(MgLevel<T> l, const T* __restrict__ xin, T* __restrict__ y, const T* __restrict__ w1,
                            Finish F) {
  __shared__ double sh[kMT];
  DotAcc<T> a1, a2;
  for (size_t c = blockIdx.x * (size_t)kMT + threadIdx.x; c < l.n; c += (size_t)gridDim.x * kMT) {
    int i, j, k;
    cell_of(c, l.nx, l.ny, i, j, k);
    const T yv = apply_at(l, xin, c, i, j, k);
    y[c] = yv;
    a1.prod(w1[c], yv);
    if (kTwo) a2.prod(yv, yv);
  }
  const double s1 = block_sum(a1.value(), sh);
  if (threadIdx.x == 0) F.part[blockIdx.x] = s1;
  __syncthreads();
  double s2 = 0.0;
  if (kTwo) s2 = block_sum(a2.value(), sh);
  if (threadIdx.x == 0) F.part[kMgRedBlocks + blockIdx.x] = s2;
  __syncthreads();
  finish(F, kTwo ? OP_OMEGA : OP_ALPHA, sh);
}

// s = r - alpha v
template <typename T>
__global__ void k_upd_s(const T* __restrict__ r, const T* __restrict__ v, T* __restrict__ s, size_t n,
                        const double* __restrict__ sc) {
  const T al = (T)sc[ALPHA];
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x)
    s[q] = r[q] - al * v[q];
}

// x += alpha ph + omega sh; r = s - omega t; partials (r, r), (r0, r)
template <typename T>
__global__ void k_upd_xr(T* __restrict__ x, const T* __restrict__ ph, const T* __restrict__ shv,
                         const T* __restrict__ s, const T* __restrict__ t, T* __restrict__ r,
                         const T* __restrict__ r0, size_t n, Finish F) {
  __shared__ double sh[kMT];
  const T al = (T)F.sc[ALPHA], om = (T)F.sc[OMEGA];
  DotAcc<T> a1, a2;
  for (size_t q = blockIdx.x * (size_t)kMT + threadIdx.x; q < n; q += (size_t)gridDim.x * kMT) {
    x[q] += al * ph[q] + om * shv[q];
    const T rv = s[q] - om * t[q];
    r[q] = rv;
    a1.prod(rv, rv);
    a2.prod(r0[q], rv);
  }
  const double s1 = block_sum(a1.value(), sh);
  if (threadIdx.x == 0) F.part[blockIdx.x] = s1;
  __syncthreads();
  const double s2 = block_sum(a2.value(), sh);
  if (threadIdx.x == 0) F.part[kMgRedBlocks + blockIdx.x] = s2;
  __syncthreads();
  finish(F, OP_XR, sh);
}

__global__ void k_stop_test(double* sc, double rtol2, int max_iter) {
  sc[RTOL2] = rtol2;
  sc[MAXIT] = (double)max_iter;
  sc[ITERS] = 0.0;
}

template <typename T>
__global__ void k_out(const T* __restrict__ x, double scale, double* __restrict__ d, size_t n) {
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x)
    d[q] = (double)x[q] * scale;
}

int cells_grid(size_t n) {
  const size_t b = (n + kMT - 1) / kMT;
  return (int)(b < 4096 ? (b > 0 ? b : 1) : 4096);
}
int red_grid(size_t n) {
  const size_t b = (n + kMT - 1) / kMT;
  return (int)(b < (size_t)kMgRedBlocks ? (b > 0 ? b : 1) : kMgRedBlocks);
}
int cols_grid(const int cols) { return (cols + 127) / 128; }

// the launch of k_coarse_smooth: one cluster of ctas CTAs
void coarse_config(int ctas, size_t smem, cudaStream_t s, cudaLaunchConfig_t& cfg, cudaLaunchAttribute& at) {
  at = cudaLaunchAttribute{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = ctas;
  at.val.clusterDim.y = 1;
  at.val.clusterDim.z = 1;
  cfg = cudaLaunchConfig_t{};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
}

template <typename T>
void smooth(const MgLevel<T>& l, const T* rhs, T* x, int color, int zero_nb, cudaStream_t s) {
  const size_t sm = scan_smem<T>(l.nz);
  if (sm <= kScanSmemMax) {  // (the shared-memory limit is raised in mg_create)
    const int g = ((l.nx + 1) / 2 * l.ny + 31) / 32;
    if (zero_nb)
      k_smooth_scan<T, true><<<g, 256, sm, s>>>(l, rhs, x, color);
    else
      k_smooth_scan<T, false><<<g, 256, sm, s>>>(l, rhs, x, color);
  } else {
    k_smooth<T><<<cols_grid(l.nx * l.ny), 128, 0, s>>>(l, rhs, x, color, zero_nb);
  }
}

// x = V(rhs) on level li (zero initial guess)
template <typename T>
void vcycle(MgSolver<T>* m, int li, const T* rhs, T* x, cudaStream_t s) {
  MgLevel<T>& l = m->lv[li];
  if (li == m->L - 1) {
    if (m->coarse_ctas > 0) {
      cudaLaunchConfig_t cfg;
      cudaLaunchAttribute at;
      coarse_config(m->coarse_ctas, m->coarse_resident ? coarse_resident_smem<T>(l.nz) : scan_smem<T>(l.nz), s, cfg,
                    at);
      const int sweeps = m->coarse_sweeps;
      if (m->coarse_resident) cudaLaunchKernelEx(&cfg, k_coarse_resident<T>, l, rhs, x, sweeps);
      else cudaLaunchKernelEx(&cfg, k_coarse_smooth<T>, l, rhs, x, sweeps);
      return;
    }
    smooth(l, rhs, x, 0, 1, s);
    smooth(l, rhs, x, 1, 0, s);
    for (int it = 1; it < m->coarse_sweeps; ++it) {
      smooth(l, rhs, x, 0, 0, s);
      smooth(l, rhs, x, 1, 0, s);
    }
    return;
  }
  MgLevel<T>& cl = m->lv[li + 1];
  smooth(l, rhs, x, 0, 1, s);
  smooth(l, rhs, x, 1, 0, s);
  k_resid_restrict<T><<<cells_grid(cl.n), kMT, 0, s>>>(l, rhs, x, cl);
  vcycle(m, li + 1, cl.r, cl.x, s);
  const size_t sm = scan_smem<T>(l.nz);
  if (sm <= kScanSmemMax) {
    k_smooth_add<T><<<((l.nx + 1) / 2 * l.ny + 31) / 32, 256, sm, s>>>(l, rhs, x, 1, cl.x, cl.nx,
                                                                      (size_t)cl.nx * cl.ny);
  } else {
    k_prolong_add<T><<<cells_grid(l.n), kMT, 0, s>>>(l, x, cl);
    smooth(l, rhs, x, 1, 0, s);
  }
  smooth(l, rhs, x, 0, 0, s);
}

template <typename T>
T* dev_alloc(MgSolver<T>* m, size_t n) {
  void* p = nullptr;
  if (cudaMalloc(&p, n * sizeof(T)) != cudaSuccess) return nullptr;
  m->allocs.push_back(p);
  return (T*)p;
}

// the arrays of one size in one allocation, each on a 256-byte boundary
template <typename T, size_t N>
bool dev_alloc_all(MgSolver<T>* m, T** (&arrs)[N], size_t n) {
  const size_t na = (n + 63) / 64 * 64;
  T* const base = dev_alloc(m, N * na);
  for (size_t q = 0; q < N; ++q) *arrs[q] = base ? base + q * na : nullptr;
  return base != nullptr;
}

}  // namespace

void hz_residual(const HGeo& g, const double* a, const double* b, const double* f, const double* x, double* r,
                 cudaStream_t s) {
  const int xt = (g.nx + kResCols - 1) / kResCols;
  const size_t tiles = (size_t)xt * ((g.ny + kResRows - 1) / kResRows);
  // about 24 blocks an SM (the last wave), chunks of at least 4 levels (a chunk computes its first lower face again)
  const int want = tiles >= 3648 ? 1 : (int)(3648 / tiles);
  int kz = imax((g.nz + want - 1) / want, 4);
  kz = imax(kz, (g.nz + 65534) / 65535);
  k_residual64<<<dim3((unsigned)tiles, (g.nz + kz - 1) / kz), dim3(32, kResRows + 1), 0, s>>>(g, a, b, f, x, r, xt, kz);
}

template <typename T>
MgSolver<T>* mg_create(const HGeo& g, int max_levels) {
  auto* m = new MgSolver<T>();
  m->g = g;
  int nx = g.nx, ny = g.ny;
  const int cap = max_levels < 1 ? 1 : (max_levels > kMgMaxLevels ? kMgMaxLevels : max_levels);
  bool ok = true, odd = false;
  for (int l = 0; l < cap; ++l) {
    MgLevel<T>& L = m->lv[l];
    L.nx = nx;
    L.ny = ny;
    L.nz = g.nz;
    L.n = (size_t)nx * ny * g.nz;
    T** arrs[] = {&L.cE, &L.cN, &L.cT, &L.cB, &L.cD, &L.lc, &L.li, &L.x, &L.r};
    ok = dev_alloc_all(m, arrs, L.n) && ok;
    m->L = l + 1;
    if (nx / 2 < 4 || ny / 2 < 4) break;
    if (nx % 2 || ny % 2) {
      // A first odd grid of this many tiles a half sweep would save iterations with
      // coarser levels, but their launches cost more: 97 x 64 x 40 (98 tiles), FP32
      // 3060 us with five levels, 2590 with one; FP64 4390 and 3820. In FP32 up to
      // kCoarseMaxTiles the one level would be smoothed by a single cluster (63 x
      // 63 x 24: 2770 us with five levels, 7800 with one), unless it is of a tile a
      // CTA, which is fast (40 x 30 x 20, second level 20 x 15). Larger grids are bound
      // by their work (193 x 193 x 60, FP64: 7950 and 13700).
      const int tiles = ((nx + 1) / 2 * ny + 31) / 32;
      const bool few = sizeof(T) == 4 && l > 0 && tiles <= kCoarseMaxCtas;
      if (!odd && (few || (tiles > (sizeof(T) == 4 ? kCoarseMaxTiles : 16) && tiles <= kOddTiles))) break;
      odd = true;
    }
    nx = (nx + 1) / 2;
    ny = (ny + 1) / 2;
  }
  const MgLevel<T>& last = m->lv[m->L - 1];
  m->coarse_sweeps = m->L >= kCoarseLevels && imax(last.nx, last.ny) <= kCoarseExtent ? 4 : 8;
  const size_t n = g.n();
  T** kv[] = {&m->x, &m->r, &m->r0, &m->p, &m->v, &m->s, &m->t, &m->ph, &m->sh};
  ok = dev_alloc_all(m, kv, n) && ok;
  void* p = nullptr;
  ok = ok && cudaMalloc(&p, 2 * kMgRedBlocks * sizeof(double)) == cudaSuccess;
  if (p) m->allocs.push_back(p), m->part = (double*)p;
  p = nullptr;
  ok = ok && cudaMalloc(&p, NSC * sizeof(double)) == cudaSuccess;
  if (p) m->allocs.push_back(p), m->sc = (double*)p;
  p = nullptr;
  ok = ok && cudaMalloc(&p, sizeof(unsigned)) == cudaSuccess && cudaMemset(p, 0, sizeof(unsigned)) == cudaSuccess;
  if (p) m->allocs.push_back(p), m->done = (unsigned*)p;
  ok = ok && cudaMallocHost(&m->hsc, NSC * sizeof(double)) == cudaSuccess;
  // the tiled smoother's FP64 tiles need more than the default 48 KB
  if (scan_smem<T>(g.nz) <= kScanSmemMax) {
    ok = ok && cudaFuncSetAttribute(k_smooth_scan<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kScanSmemMax) == cudaSuccess;
    ok = ok && cudaFuncSetAttribute(k_smooth_scan<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kScanSmemMax) == cudaSuccess;
    ok = ok && cudaFuncSetAttribute(k_smooth_add<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kScanSmemMax) == cudaSuccess;
    // the coarsest grid in one cluster launch when it is a few tiles: one
    // CTA per tile, up to a portable cluster (FP32 only: the FP64 rate of a
    // few SMs is far too low for the whole coarse solve)
    const MgLevel<T>& c = m->lv[m->L - 1];
    const int ntiles = ((c.nx + 1) / 2 * c.ny + 31) / 32;
    const int ctas = ntiles < kCoarseMaxCtas ? ntiles : kCoarseMaxCtas;
    if (sizeof(T) == 4 && ok && ntiles <= kCoarseMaxTiles) {
      ok = ok && cudaFuncSetAttribute(k_coarse_smooth<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kScanSmemMax) == cudaSuccess;
      cudaLaunchConfig_t cfg;
      cudaLaunchAttribute at;
      coarse_config(ctas, scan_smem<T>(g.nz), nullptr, cfg, at);
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, k_coarse_smooth<T>, &cfg) == cudaSuccess && clusters > 0)
        m->coarse_ctas = ctas;
      if (m->coarse_ctas == ntiles && coarse_resident_smem<T>(g.nz) <= kScanSmemMax) {
        ok = ok && cudaFuncSetAttribute(k_coarse_resident<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)kScanSmemMax) == cudaSuccess;
        coarse_config(ctas, coarse_resident_smem<T>(g.nz), nullptr, cfg, at);
        clusters = 0;
        m->coarse_resident =
            cudaOccupancyMaxActiveClusters(&clusters, k_coarse_resident<T>, &cfg) == cudaSuccess && clusters > 0;
      }
      cudaGetLastError();  // (a cluster launch that cannot run leaves the launches per half sweep)
    }
  }
  if (!ok) {
    mg_destroy(m);
    return nullptr;
  }
  return m;
}

template <typename T>
void mg_destroy(MgSolver<T>* m) {
  if (!m) return;
  if (m->gexec) cudaGraphExecDestroy(m->gexec);
  if (m->graph) cudaGraphDestroy(m->graph);
  for (void* p : m->allocs) cudaFree(p);
  if (m->hsc) cudaFreeHost(m->hsc);
  delete m;
}

template <typename T>
bool mg_odd(const MgSolver<T>* m) {
  return m->L > 1 && (m->lv[0].nx % 2 || m->lv[0].ny % 2);
}

template <typename T>
int mg_levels(const MgSolver<T>* m) {
  return m->L;
}

template <typename T>
int mg_set_coefficients(MgSolver<T>* m, const double* a, const double* b, cudaStream_t s) {
  k_fine_coefs<T><<<cells_grid(m->g.n()), kMT, 0, s>>>(m->g, a, b, m->lv[0]);
  for (int l = 1; l < m->L; ++l)
    k_coarse_coefs<T><<<cells_grid(m->lv[l].n), kMT, 0, s>>>(m->lv[l - 1], m->lv[l]);
  for (int l = 0; l < m->L; ++l)
    k_column_lu<T><<<cols_grid(m->lv[l].nx * m->lv[l].ny), 128, 0, s>>>(m->lv[l]);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// one BiCGSTAB iteration (right-preconditioned by a V-cycle)
template <typename T>
void enqueue_iteration(MgSolver<T>* m, cudaStream_t s, cudaGraphConditionalHandle cond, int use_cond) {
  const size_t n = m->g.n();
  const int nb = red_grid(n), cg = cells_grid(n);
  MgLevel<T>& f = m->lv[0];
  k_upd_p<T><<<cg, kMT, 0, s>>>(m->r, m->p, m->v, n, m->sc);
  vcycle(m, 0, m->p, m->ph, s);
  const Finish F{m->part, m->sc, m->done, cond, use_cond};
  k_apply_dot<T, false><<<nb, kMT, 0, s>>>(f, m->ph, m->v, m->r0, F);
  k_upd_s<T><<<cg, kMT, 0, s>>>(m->r, m->v, m->s, n, m->sc);
  vcycle(m, 0, m->s, m->sh, s);
  k_apply_dot<T, true><<<nb, kMT, 0, s>>>(f, m->sh, m->t, m->s, F);
  k_upd_xr<T><<<nb, kMT, 0, s>>>(m->x, m->ph, m->sh, m->s, m->t, m->r, m->r0, n, F);
}

// The iteration loop as one graph: a WHILE conditional node (default 1 at
// every launch) whose body is one iteration captured from the stream.
template <typename T>
bool build_loop_graph(MgSolver<T>* m, cudaStream_t s) {
  cudaGraph_t g = nullptr;
  if (cudaGraphCreate(&g, 0) != cudaSuccess) return false;
  cudaGraphConditionalHandle cond;
  cudaGraphNodeParams p = {};
  cudaGraphNode_t node;
  cudaGraph_t captured = nullptr;
  bool ok = cudaGraphConditionalHandleCreate(&cond, g, 1, cudaGraphCondAssignDefault) == cudaSuccess;
  if (ok) {
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = cond;
    p.conditional.type = cudaGraphCondTypeWhile;
    p.conditional.size = 1;
    ok = cudaGraphAddNode(&node, g, nullptr, nullptr, 0, &p) == cudaSuccess;
  }
  if (ok) {
    cudaGraph_t body = p.conditional.phGraph_out[0];
    ok = cudaStreamBeginCaptureToGraph(s, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal) ==
         cudaSuccess;
    if (ok) {
      enqueue_iteration(m, s, cond, 1);
      ok = cudaStreamEndCapture(s, &captured) == cudaSuccess && captured == body;
    }
  }
  if (ok) ok = cudaGraphInstantiate(&m->gexec, g, 0) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();  // the host loop takes over
    if (m->gexec) cudaGraphExecDestroy(m->gexec);
    m->gexec = nullptr;
    cudaGraphDestroy(g);
    return false;
  }
  m->graph = g;
  return true;
}

template <typename T>
int mg_solve(MgSolver<T>* m, const double* r64, double* d64, double rtol, int max_iter, cudaStream_t s,
             double r_norm2) {
  const size_t n = m->g.n();
  const int nb = red_grid(n), cg = cells_grid(n);
  // scale the right-hand side to unit norm (FP32 range), FP64 dot
  if (r_norm2 < 0.0) {
    dot64(r64, r64, n, m->part, m->sc + NSC - 1, s);
    if (cudaMemcpyAsync(m->hsc, m->sc + NSC - 1, sizeof(double), cudaMemcpyDeviceToHost, s) != cudaSuccess)
      return -1;
    if (cudaStreamSynchronize(s) != cudaSuccess) return -1;
    r_norm2 = m->hsc[0];
  }
  const double rn = std::sqrt(r_norm2);
  if (!(rn > 0.0) || !std::isfinite(rn)) {
    cudaMemsetAsync(d64, 0, n * sizeof(double), s);
    return 0;
  }
  k_init<T><<<nb, kMT, 0, s>>>(r64, 1.0 / rn, n, m->r, m->r0, m->x, m->p, m->v,
                               Finish{m->part, m->sc, m->done, cudaGraphConditionalHandle{}, 0});
  k_stop_test<<<1, 1, 0, s>>>(m->sc, rtol * rtol, max_iter);
  if (m->graph_state == 0) {
    // VIBE_GB300_HELMHOLTZ_GRAPH=0 keeps the host loop (one scalar read per iteration)
    const char* e = std::getenv("VIBE_GB300_HELMHOLTZ_GRAPH");
    m->graph_state = (e && std::atoi(e) == 0) ? -1 : (build_loop_graph(m, s) ? 1 : -1);
  }
  int it = 0;
  bool broke = false;
  if (m->graph_state == 1 && max_iter > 0) {
    // the whole loop on the device: one launch, one read of the scalars
    if (cudaGraphLaunch(m->gexec, s) != cudaSuccess) return -1;
    if (cudaMemcpyAsync(m->hsc, m->sc, NSC * sizeof(double), cudaMemcpyDeviceToHost, s) != cudaSuccess) return -1;
    if (cudaStreamSynchronize(s) != cudaSuccess) return -1;
    it = (int)m->hsc[ITERS];
    broke = m->hsc[BREAK] != 0.0;
  } else {
    for (; it < max_iter; ++it) {
      enqueue_iteration(m, s, cudaGraphConditionalHandle{}, 0);
      if (cudaMemcpyAsync(m->hsc, m->sc, NSC * sizeof(double), cudaMemcpyDeviceToHost, s) != cudaSuccess) return -1;
      if (cudaStreamSynchronize(s) != cudaSuccess) return -1;
      if (m->hsc[BREAK] != 0.0) {
        broke = true;
        ++it;
        break;
      }
      if (std::sqrt(m->hsc[RR]) <= rtol) {
        ++it;
        break;
      }
    }
  }
  k_out<T><<<cg, kMT, 0, s>>>(m->x, rn, d64, n);
  if (cudaGetLastError() != cudaSuccess) return -1;
  return broke ? -it : it;
}

template MgSolver<float>* mg_create<float>(const HGeo&, int);
template MgSolver<double>* mg_create<double>(const HGeo&, int);
template void mg_destroy<float>(MgSolver<float>*);
template void mg_destroy<double>(MgSolver<double>*);
template bool mg_odd<float>(const MgSolver<float>*);
template int mg_levels<float>(const MgSolver<float>*);
template int mg_levels<double>(const MgSolver<double>*);
template int mg_set_coefficients<float>(MgSolver<float>*, const double*, const double*, cudaStream_t);
template int mg_set_coefficients<double>(MgSolver<double>*, const double*, const double*, cudaStream_t);
template int mg_solve<float>(MgSolver<float>*, const double*, double*, double, int, cudaStream_t, double);
template int mg_solve<double>(MgSolver<double>*, const double*, double*, double, int, cudaStream_t, double);

}  // namespace vgb
