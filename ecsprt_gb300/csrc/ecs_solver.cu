// Potential solve of the ECSPRT hot path on sm_103a: the matrix-free
// 11-point operator of src/lhs.c:337-505 and the KSP solve of
// src/potential.c:6-15.
//
// FGMRES(m) preconditioned by one geometric-multigrid V(1,1) cycle (full
// coarsening, full-weighting restriction, trilinear prolongation, coarse
// operators rediscretised from the full-weighted density, damped z-line
// Jacobi smoothing: the z couplings carry (1+kappa^2) and dominate).
//   ECS_PREC_FP64:  FGMRES and multigrid in FP64 to the requested rtol.
//   ECS_PREC_MIXED: FP64 iterative refinement; each correction is an FP32
//     FGMRES/multigrid solve; residuals, their norms, the update of phi and
//     the mean projection are FP64.
//
// One FGMRES cycle runs entirely on the device: the Gram-Schmidt
// coefficients, the Hessenberg matrix, the Givens rotations and the
// convergence test live in a device control block (KrylovDev), and the
// kernels that need the Arnoldi index read it from there.  The cycle is a
// CUDA graph whose Arnoldi step is the body of a conditional WHILE node; the
// step's last small kernel clears the condition once the residual estimate
// meets the tolerance, so the host waits once per cycle.  Without graphs the
// host launches the same kernels step by step and reads the stop flag after
// each step.
//
// All reductions use fixed block partials summed in a fixed order, so every
// result is reproducible run to run.
#include <math.h>
#include <string.h>

#include <cooperative_groups.h>

#include <algorithm>
#include <vector>

#include "ecs_stencil.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int kKrylovMax = 30;            // restart length m (upper bound)
constexpr int kSlots = kKrylovMax + 2;    // dot-product slots per pass
constexpr int kDotBlocks = 1024;          // block partials per dot pass
constexpr int kB = 256;

// Device control block of one FGMRES cycle.
struct KrylovDev {
  // set by the host before a cycle
  double tol_rel;  // stop when the estimate <= tol_rel * beta
  int maxit;       // Arnoldi steps allowed in this cycle (<= kKrylovMax)
  int pad0;
  // cycle state
  int j;           // current Arnoldi index
  int jprev;       // index of the step that just finished
  int done;        // 1: converged, broke down or out of steps
  int nits;        // Arnoldi steps taken
  double beta, res, inv_scale, mean, hn;
  double h1[kSlots], h2[kSlots];
  double H[(kKrylovMax + 1) * kKrylovMax];
  double cs[kKrylovMax], sn[kKrylovMax], g[kKrylovMax + 1], y[kKrylovMax];
  // completion tickets of the grid-wide reductions (0 between launches)
  unsigned int ticket[8];
};

// ---- operator ------------------------------------------------------------------
// A row's 11 coefficients: in FP64 from the arrays of k_coef64 (coef[e * n +
// c]), where there are any, since forming them takes 39 of the row's 50 FP64
// operations and FP64 is the scarce resource here (64^3 operator: 25 -> 10 us);
// in FP32 always from the density, which is 7 words instead of 11.
template <typename T>
__device__ __forceinline__ void row_coef(const OpK &o, const T *__restrict__ n, const T *__restrict__ coef,
                                         const Nbr &q, T v[11]) {
  if (sizeof(T) == 8 && coef) {
#pragma unroll
    for (int e = 0; e < 11; e++) v[e] = __ldg(&coef[(size_t)e * o.g.n + q.c]);
  } else {
    row11_n(n, o, q, v);
  }
}

// y = A x   (mode 0)     or     y = b - A x   (mode 1)
template <typename T>
__global__ void k_apply(OpK o, const T *__restrict__ n, const T *__restrict__ coef, const T *__restrict__ x,
                        const T *__restrict__ b, T *__restrict__ y, int mode) {
  ECS_PDL_ENTRY_FOR(T);
  int i, j, k;
  if (!at3(o.g.nx, o.g.ny, i, j, k)) return;
  const Nbr q = nbr_of(o.g, i, j, k);
  T v[11], xe[11];
  row_coef(o, n, coef, q, v);
  row_x(x, q, xe);
  T s = T(0);
#pragma unroll
  for (int e = 0; e < 11; e++) s += v[e] * xe[e];
  y[q.c] = mode ? b[q.c] - s : s;
}

// ---- FP32 rows four cells a thread ----------------------------------------------
// Four consecutive x cells of one row: their 18 operands a cell overlap, so a
// thread loads 10 float4 and 8 words for all four instead of 72 words.  The
// one-cell kernels are bound by those loads on the large levels (128^3:
// residual 16.8 -> 8.8 us, z-line right-hand side 12.8 -> 6.8, Arnoldi operator
// 18.6 -> 10.0, prolongation 12.3 -> 4.8, restriction 6.0 -> 4.2); the same
// operands give the same bits.  For rows that are a multiple of 4 long (16-byte
// alignment) and levels of at least kRow4Cells cells: below, a quarter of the
// threads hides latency worse than the loads cost (32^3 solve 0.675 against
// 0.666 ms; 48^3 0.930 against 0.943 ms).  x and y are periodic on every grid
// the solver takes; z may have ghosts.
constexpr size_t kRow4Cells = 1 << 16;
struct Row4 {
  float m, p;  // the cells before and after
  float4 c;
  // value d cells (-1, 0, 1) from cell e of the four
  __device__ __forceinline__ float at(int e) const {
    return e < 0 ? m : (e == 0 ? c.x : (e == 1 ? c.y : (e == 2 ? c.z : (e == 3 ? c.w : p))));
  }
};
struct Cell4 {
  unsigned c;          // linear index of the first cell
  int xm, xp;          // offsets of the cells before the first and after the last
  int ym, yp, zm, zp;  // row and plane offsets
  bool vzm, vzp;
};
__device__ __forceinline__ float4 ld4(const float *__restrict__ f, unsigned c) {
  return *reinterpret_cast<const float4 *>(f + c);
}
__device__ __forceinline__ Row4 row4(const float *__restrict__ f, const Cell4 &q, int off) {
  const unsigned c = (unsigned)((int)q.c + off);
  return {f[(unsigned)((int)c + q.xm)], f[(unsigned)((int)c + q.xp)], ld4(f, c)};
}
__device__ __forceinline__ float4 plane4(const float *__restrict__ f, const Cell4 &q, int off, bool valid) {
  return valid ? ld4(f, (unsigned)((int)q.c + off)) : make_float4(0.f, 0.f, 0.f, 0.f);
}
// Block of row quarters: blockDim.x packs along x, blockDim.y rows.
__device__ __forceinline__ bool at4(const GridG &g, Cell4 &q) {
  const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x) * 4, j = (int)(blockIdx.y * blockDim.y + threadIdx.y),
            k = (int)blockIdx.z;
  if (i >= g.nx || j >= g.ny) return false;
  const Nbr n = nbr_of(g, i, j, k);
  q.c = n.c;
  q.xm = n.xm;
  q.xp = i + 4 < g.nx ? 4 : 4 - g.nx;
  q.ym = n.ym; q.yp = n.yp; q.zm = n.zm; q.zp = n.zp;
  q.vzm = n.vzm; q.vzp = n.vzp;
  return true;
}
static inline dim3 threads4(int nx) {
  const int w = std::min(nx / 4, 32);
  return dim3((unsigned)w, (unsigned)(256 / w));
}
static inline dim3 blocks4(const GridG &g) {
  const dim3 t = threads4(g.nx);
  return dim3((unsigned)((g.nx / 4 + (int)t.x - 1) / (int)t.x), (unsigned)((g.ny + (int)t.y - 1) / (int)t.y), (unsigned)g.nz);
}
static inline bool use_row4(const GridG &g) { return g.nx % 4 == 0 && g.n >= kRow4Cells; }
// The row sums of the four cells: start[e] + sign * sum of v[e'] x[e'] over the
// row's entries in the order of off_i (in-plane ones only without Z), x less m.
template <bool Z, bool SUB>
__device__ __forceinline__ void rows4(const OpK &o, const float *__restrict__ n, const float *__restrict__ x,
                                      const Cell4 &q, float m, float s[4]) {
  const Row4 nc = row4(n, q, 0);
  const float4 nym = ld4(n, (unsigned)((int)q.c + q.ym)), nyp = ld4(n, (unsigned)((int)q.c + q.yp));
  float4 nzm = make_float4(0.f, 0.f, 0.f, 0.f), nzp = nzm, xzm = nzm, xzp = nzm;
  const Row4 xc = row4(x, q, 0), xym = row4(x, q, q.ym), xyp = row4(x, q, q.yp);
  if (Z) {
    nzm = plane4(n, q, q.zm, q.vzm);
    nzp = plane4(n, q, q.zp, q.vzp);
    xzm = plane4(x, q, q.zm, q.vzm);
    xzp = plane4(x, q, q.zp, q.vzp);
  }
  auto f4 = [](const float4 &f, int e) { return e == 0 ? f.x : (e == 1 ? f.y : (e == 2 ? f.z : f.w)); };
#pragma unroll
  for (int e = 0; e < 4; e++) {
    float v[11];
    row11_vals(o, nc.at(e), nc.at(e - 1), nc.at(e + 1), f4(nym, e), f4(nyp, e), f4(nzm, e), f4(nzp, e), v);
    const float xe[11] = {xc.at(e + 1),  xc.at(e - 1),  xyp.at(e),     xym.at(e),     f4(xzp, e), f4(xzm, e),
                          xyp.at(e + 1), xym.at(e + 1), xyp.at(e - 1), xym.at(e - 1), xc.at(e)};
#pragma unroll
    for (int r = 0; r < 11; r++) {
      if (!Z && (r == 4 || r == 5 || r == 10)) continue;
      if (SUB) s[e] -= v[r] * xe[r];
      else s[e] += v[r] * (xe[r] - m);
    }
  }
}
// y = b - A x (k_apply, mode 1)
__global__ void __launch_bounds__(256) k_apply4(OpK o, const float *__restrict__ n, const float *__restrict__ x,
                                                const float *__restrict__ b, float *__restrict__ y) {
  ECS_PDL_ENTRY();
  Cell4 q;
  if (!at4(o.g, q)) return;
  const float4 bv = ld4(b, q.c);
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  rows4<true, false>(o, n, x, q, 0.f, s);
  *reinterpret_cast<float4 *>(y + q.c) = make_float4(bv.x - s[0], bv.y - s[1], bv.z - s[2], bv.w - s[3]);
}
// r = b - A_xy x (k_zline_rhs)
__global__ void __launch_bounds__(256) k_zline_rhs4(OpK o, const float *__restrict__ n, const float *__restrict__ b,
                                                    const float *__restrict__ x, float *__restrict__ r) {
  ECS_PDL_ENTRY();
  Cell4 q;
  if (!at4(o.g, q)) return;
  const float4 bv = ld4(b, q.c);
  float s[4] = {bv.x, bv.y, bv.z, bv.w};
  rows4<false, true>(o, n, x, q, 0.f, s);
  *reinterpret_cast<float4 *>(r + q.c) = make_float4(s[0], s[1], s[2], s[3]);
}
// Z_j = x - mean, V_{j+1} = A Z_j (k_apply_dyn)
__global__ void __launch_bounds__(256) k_apply_dyn4(OpK o, const float *__restrict__ n, const float *__restrict__ x,
                                                    const double *__restrict__ mean, float *__restrict__ Z,
                                                    float *__restrict__ V, const KrylovDev *__restrict__ kd) {
  ECS_PDL_ENTRY();
  Cell4 q;
  if (!at4(o.g, q)) return;
  const int jj = kd->j;
  const float m = mean ? (float)mean[0] : 0.f;
  const float4 xc = ld4(x, q.c);
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  rows4<true, false>(o, n, x, q, m, s);
  *reinterpret_cast<float4 *>(Z + (size_t)jj * o.g.n + q.c) = make_float4(xc.x - m, xc.y - m, xc.z - m, xc.w - m);
  *reinterpret_cast<float4 *>(V + (size_t)(jj + 1) * o.g.n + q.c) = make_float4(s[0], s[1], s[2], s[3]);
}

// ---- z-line smoother --------------------------------------------------------------
// Column (i,j) carries the z-tridiagonal part of the rows: lo = z- entry,
// diag = centre, up = z+ entry.  A periodic z closes the cycle, solved with
// Sherman-Morrison around the Thomas factorisation of the modified matrix;
// reflecting z drops the out-of-range couplings (Dirichlet-0 ghosts).
// The solve runs in segments of S cells along z, one thread per segment; the
// forward recurrence d_k = (r_k - a_k d_{k-1}) / m_k and the backward one
// y_k = d_k - cp_k y_{k+1} are affine in the value carried in, so each
// segment solves from zero and the carried values are stitched afterwards
// with the in-segment products fb_k = prod(-a_i/m_i) and bb_k = prod(-cp_i).
// FP32 with segments of 8 stores 1/m and the Sherman-Morrison vector q only:
// a, cp, fb and bb follow from the density and 1/m with the set-up's own
// operations (the same bits), which is cheaper than reading four more words a
// cell.  On this GPU FP64 arithmetic is the scarcer resource, so FP64 reads
// them all; so do segments of 16 and more, whose recomputed factors would not
// fit the registers.
template <typename T>
__host__ __device__ constexpr bool zl_stored(int S) { return sizeof(T) == 8 || S > 8; }
template <typename T>
struct ZlP {
  T *a, *cp, *minv, *q, *fb, *bb;  // per cell (a, cp, fb, bb: zl_stored only, else nullptr)
  T *a0g, *qden;                   // per column
};
// At most 16 segments a column (block of 32 x 16 threads); segments of 8,
// 16, 32 or 64 cells, the shortest that fits.
constexpr int kMaxSeg = 16;
template <typename T>
static inline int seg_len(int N) {
  for (int S = 8; S < 64; S *= 2)
    if (N <= S * kMaxSeg) return S;
  return 64;
}

// The z couplings of the rows: lower entry of plane k from the densities of
// planes k and k - 1, upper entry from those of planes k and k + 1 (the same
// operations as row11_vals); unit: density 1 everywhere.
template <typename T>
struct ZCoup {
  T szz;
  int unit;
  __device__ __forceinline__ T operator()(T here, T other) const {
    return unit ? szz * (T(1) + T(1)) : szz * (other + here);
  }
};
template <typename T>
static inline ZCoup<T> z_coupling(const OpK &o) {
  return {sizeof(T) == 8 ? (T)o.szz : (T)o.fzz, o.unit};
}

// The diagonal of every row, one thread per cell: the parallel half of the
// z-line set-up.
template <typename T>
__global__ void k_zline_rows(OpK o, const T *__restrict__ n, T *__restrict__ dg) {
  ECS_PDL_ENTRY_FOR(T);
  int i, j, k;
  if (!at3(o.g.nx, o.g.ny, i, j, k)) return;
  const Nbr q = nbr_of(o.g, i, j, k);
  T v[11];
  row11_n(n, o, q, v);
  dg[q.c] = v[10];
}

// Factorisation of every column's z tridiagonal (one thread a column) from
// the density and the diagonal of k_zline_rows.
template <typename T>
__global__ void k_zline_setup(GridG g, ZCoup<T> zc, const T *__restrict__ n, const T *__restrict__ dg, ZlP<T> z,
                              int S) {
  ECS_PDL_ENTRY_FOR(T);
  const int ncol = g.nx * g.ny;
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= ncol) return;
  const size_t plane = (size_t)g.nx * g.ny;
  // a one-cell column (2-D) has no z coupling: the plain solve, no periodic closure
  const bool cyc = g.bc[2] == 0 && g.nz > 1;
  const int N = g.nz;
  const bool stored = z.a != nullptr;
  const T n0 = __ldg(&n[col]), nN = __ldg(&n[(size_t)(N - 1) * plane + col]);
  const T lo0 = cyc ? zc(n0, nN) : T(0), d0 = __ldg(&dg[col]);
  const T gamma = -d0;
  T cp_prev = T(0), dq_prev = T(0), fprod = T(1);
  // forward: factor T' and forward-substitute u = (gamma, 0, .., up_{N-1});
  // the operands are read kBatch at a time, all loads first, so the
  // recurrence waits on one memory latency a batch rather than one a cell
  constexpr int kBatch = 8;
  T nprev = nN, nhere = n0;
  for (int k0 = 0; k0 < N; k0 += kBatch) {
    T nv[kBatch], dv[kBatch];
#pragma unroll
    for (int e = 0; e < kBatch; e++) {
      const int k = min(k0 + e, N - 1), kn = k + 1 < N ? k + 1 : 0;  // the plane above, wrapped
      nv[e] = __ldg(&n[(size_t)kn * plane + col]);
      dv[e] = __ldg(&dg[(size_t)k * plane + col]);
    }
#pragma unroll
    for (int e = 0; e < kBatch; e++) {
      const int k = k0 + e;
      if (k >= N) break;
      const size_t c = (size_t)k * plane + col;
      const T lk = zc(nhere, nprev), uk = zc(nhere, nv[e]), dk = dv[e];
      T a = (k == 0) ? T(0) : lk;
      T upk = (k == N - 1) ? T(0) : uk;
      T bb = dk;
      if (cyc && k == 0) bb = d0 - gamma;
      if (cyc && k == N - 1) bb = dk - uk * lo0 / gamma;
      T m = bb - a * cp_prev;
      T minv = T(1) / m;
      T cp = upk * minv;
      T u = cyc ? ((k == 0) ? gamma : ((k == N - 1) ? uk : T(0))) : T(0);
      T dq = (u - a * dq_prev) * minv;
      z.minv[c] = minv;
      z.q[c] = dq;
      if (stored) {
        z.a[c] = a;
        z.cp[c] = cp;
        if (k % S == 0) fprod = T(1);
        fprod *= -(a * minv);
        z.fb[c] = fprod;
      }
      cp_prev = cp;
      dq_prev = dq;
      nprev = nhere;
      nhere = nv[e];
    }
  }
  // backward substitution for q (this thread's own values from above, read
  // back a batch at a time) and, where they are stored, the in-segment
  // products of -cp
  T qn = z.q[(size_t)(N - 1) * plane + col];
  T bprod = T(1);
  if (stored) {
    bprod = -z.cp[(size_t)(N - 1) * plane + col];
    z.bb[(size_t)(N - 1) * plane + col] = bprod;
  }
  T nup = nN;  // density of the plane above the current one
  for (int k0 = N - 2; k0 >= 0; k0 -= kBatch) {
    T qv[kBatch], cv[kBatch], nv[kBatch];
#pragma unroll
    for (int e = 0; e < kBatch; e++) {
      const size_t c = (size_t)max(k0 - e, 0) * plane + col;
      qv[e] = z.q[c];
      cv[e] = z.minv[c];
      nv[e] = __ldg(&n[c]);
    }
#pragma unroll
    for (int e = 0; e < kBatch; e++) {
      const int k = k0 - e;
      if (k < 0) break;
      const size_t c = (size_t)k * plane + col;
      const T cp = zc(nv[e], nup) * cv[e];
      nup = nv[e];
      qn = qv[e] - cp * qn;
      z.q[c] = qn;
      if (stored) {
        if ((k + 1) % S == 0) bprod = T(1);
        bprod *= -cp;
        z.bb[c] = bprod;
      }
    }
  }
  if (cyc) {
    T a0g = lo0 / gamma;
    T q0 = z.q[col], qN = z.q[(size_t)(N - 1) * plane + col];
    z.a0g[col] = a0g;
    z.qden[col] = T(1) / (T(1) + q0 + a0g * qN);
  } else {
    z.a0g[col] = T(0);
    z.qden[col] = T(0);
  }
}

// Right-hand side of the z-line systems: r = b - A_xy xo.
template <typename T>
__global__ void k_zline_rhs(OpK o, const T *__restrict__ n, const T *__restrict__ coef, const T *__restrict__ b,
                            const T *__restrict__ xo, T *__restrict__ r) {
  ECS_PDL_ENTRY_FOR(T);
  int i, j, k;
  if (!at3(o.g.nx, o.g.ny, i, j, k)) return;
  const Nbr q = nbr_of(o.g, i, j, k);
  T v[11], xe[11];
  row_coef(o, n, coef, q, v);
  row_x(xo, q, xe);
  T s = b[q.c];
#pragma unroll
  for (int e = 0; e < 10; e++) {
    if (e == 4 || e == 5) continue;
    s -= v[e] * xe[e];
  }
  r[q.c] = s;
}

// Damped z-line Jacobi update: T' y = r by segments, Sherman-Morrison
// closure of the periodic cycle, xn = xo + omega (y - s q - xo) (xo nullptr:
// zero).  Block = 32 columns (consecutive x at one y) x P segments of S
// cells.  Bound by memory latency on the small levels and by L2 traffic on the
// large ones.  FP32 with segments of 8 reads 5 words a cell instead of 9, and
// its last operands are requested before the first barrier, so that two
// memory latencies cover the solve.  Every thread runs the carried-value scan
// over the segments itself (two barriers instead of four): 9.1 -> 4.7 us at
// 32^3, 21.4 -> 13.2 us at 128^3 (launch list).  Each phase keeps only the arrays that it
// needs, so that two blocks of 512 threads fit an SM (with everything held
// from the start, one block an SM, it took 1.1 us more at 96^3).
template <typename T, int S>
__global__ void __launch_bounds__(32 * kMaxSeg, zl_stored<T>(S) ? 1 : 2)
    k_zline_seg(GridG g, ZCoup<T> zc, const T *__restrict__ n, ZlP<T> z, const T *__restrict__ r,
                const T *__restrict__ xo, T *__restrict__ xn, T omega) {
  ECS_PDL_ENTRY_FOR(T);
  constexpr bool kStored = zl_stored<T>(S);
  __shared__ T sA[kMaxSeg][33], sB[kMaxSeg][33], sC[kMaxSeg][33], sD[kMaxSeg][33];
  __shared__ T sLast[32];
  const int tx = threadIdx.x, p = threadIdx.y, P = blockDim.y;
  const int i = blockIdx.x * 32 + tx, j = blockIdx.y;
  const bool act = i < g.nx;
  const size_t plane = (size_t)g.nx * g.ny;
  const int col = j * g.nx + i;
  const int N = g.nz, k0 = p * S, k1 = min(N, k0 + S);
  const size_t c0 = (size_t)k0 * plane + col;
  auto in = [&](int q) { return act && k0 + q < k1; };
  T rv[S];          // r, then d, then y
  T cv[S], fv[S];   // cp, fb
  T qv[S], ov[kStored ? 1 : S];
  T a0g = T(0), qden = T(0);
  // forward, from zero at the segment start
  if constexpr (kStored) {
#pragma unroll
    for (int q = 0; q < S; q++) {
      const size_t c = c0 + (size_t)q * plane;
      rv[q] = in(q) ? r[c] : T(0);
      cv[q] = in(q) ? z.a[c] : T(0);
      fv[q] = in(q) ? z.minv[c] : T(0);
    }
    T d = T(0);
#pragma unroll
    for (int q = 0; q < S; q++)
      if (in(q)) {
        d = (rv[q] - cv[q] * d) * fv[q];
        rv[q] = d;
      }
    sA[p][tx] = d;
    sB[p][tx] = act && k0 < k1 ? z.fb[(size_t)(k1 - 1) * plane + col] : T(0);
  } else {
    T nv[S + 2];  // densities of planes k0 - 1 .. k0 + S
    nv[0] = act && k0 > 0 && k0 < N ? n[c0 - plane] : T(0);
    nv[S + 1] = act && k0 + S < N ? n[c0 + (size_t)S * plane] : T(0);
#pragma unroll
    for (int q = 0; q < S; q++) {
      const size_t c = c0 + (size_t)q * plane;
      rv[q] = in(q) ? r[c] : T(0);
      nv[q + 1] = in(q) ? n[c] : T(0);
      cv[q] = in(q) ? z.minv[c] : T(0);
    }
    T d = T(0), fprod = T(1);
#pragma unroll
    for (int q = 0; q < S; q++)
      if (in(q)) {
        const T a = k0 + q == 0 ? T(0) : zc(nv[q + 1], nv[q]);
        const T up = k0 + q == N - 1 ? T(0) : zc(nv[q + 1], nv[q + 2]);
        d = (rv[q] - a * d) * cv[q];
        rv[q] = d;
        fprod *= -(a * cv[q]);
        fv[q] = fprod;
        cv[q] = up * cv[q];
      }
    sA[p][tx] = d;
    sB[p][tx] = k0 < k1 ? fprod : T(0);
#pragma unroll
    for (int q = 0; q < S; q++) {
      const size_t c = c0 + (size_t)q * plane;
      qv[q] = in(q) ? z.q[c] : T(0);
      ov[q] = (in(q) && xo) ? xo[c] : T(0);
    }
  }
  if (act) {
    a0g = z.a0g[col];
    qden = z.qden[col];
  }
  __syncthreads();
  // the value carried in, then backward from zero at the segment end
  {
    T din = T(0);
    for (int pp = 0; pp < p; pp++) din = sA[pp][tx] + sB[pp][tx] * din;
    if constexpr (kStored) {
#pragma unroll
      for (int q = 0; q < S; q++) {
        const size_t c = c0 + (size_t)q * plane;
        fv[q] = in(q) ? z.fb[c] : T(0);
        cv[q] = in(q) ? z.cp[c] : T(0);
      }
    }
    T y = T(0), bprod = T(1);
#pragma unroll
    for (int q = S - 1; q >= 0; q--) {
      if (in(q)) {
        y = (rv[q] + fv[q] * din) - cv[q] * y;
        rv[q] = y;
        if constexpr (!kStored) bprod *= -cv[q];
        if (k0 + q == N - 1) sLast[tx] = y;  // y_{N-1}: nothing is carried into the last segment
      }
    }
    if constexpr (kStored) bprod = in(0) ? z.bb[c0] : T(0);
    sC[p][tx] = y;
    sD[p][tx] = in(0) ? bprod : T(0);
  }
  __syncthreads();
  {
    T yin = T(0), run = T(0);
    for (int pp = P - 1; pp >= 0; pp--) {
      if (pp == p) yin = run;
      run = sC[pp][tx] + sD[pp][tx] * run;
    }
    const T s = act ? (run + a0g * sLast[tx]) * qden : T(0);  // run = y_0
    if constexpr (kStored) {
#pragma unroll
      for (int q = 0; q < S; q++) {
        const size_t c = c0 + (size_t)q * plane;
        fv[q] = in(q) ? z.bb[c] : T(0);
        qv[q] = in(q) ? z.q[c] : T(0);
      }
    }
    T bprod = T(1);
#pragma unroll
    for (int q = S - 1; q >= 0; q--) {
      if (in(q)) {
        const size_t c = c0 + (size_t)q * plane;
        T o, bb;
        if constexpr (kStored) {
          o = xo ? xo[c] : T(0);
          bb = fv[q];
        } else {
          o = ov[q];
          bprod *= -cv[q];
          bb = bprod;
        }
        const T yk = rv[q] + bb * yin;
        xn[c] = o + omega * ((yk - s * qv[q]) - o);
      }
    }
  }
}

// ---- inter-grid transfer ---------------------------------------------------------
// A level of more than one plane whose coarser level has as many planes is
// coarsened in x and y only (reflecting z, see mg_alloc): its transfers act
// within each plane.
__host__ __device__ __forceinline__ bool semi_z(const GridG &gf, const GridG &gc) { return gf.nz == gc.nz && gf.nz > 1; }

// The transfers between small levels are bound by the latency of one thread's
// loads: all of them are asked for before the first sum (predicated, not
// branched around), and SEMI (semi_z) is a parameter of the kernel.  Solves:
// 32^3 0.610 -> 0.585 ms, 128^3 1.568 -> 1.532, 256^2 in 2-D 0.781 -> 0.747, FP64
// 64^3 1.728 -> 1.694.

// Full weighting (1/4,1/2,1/4 per coarsened axis) from fine (2I+a) to coarse
// I: the 27 (9 when z is not coarsened) fine cells through the neighbour
// offsets of the fine cell (2I, 2J, 2K) (or (2I, 2J, K)).
template <typename T, bool SEMI>
__global__ void k_restrict(GridG gf, GridG gc, const T *__restrict__ f, T *__restrict__ c) {
  ECS_PDL_ENTRY_FOR(T);
  int I, J, K;
  if (!at3(gc.nx, gc.ny, I, J, K)) return;
  const Nbr q = nbr_of(gf, 2 * I, 2 * J, SEMI ? K : 2 * K);
  const int oz[3] = {q.zm, 0, q.zp}, oy[3] = {q.ym, 0, q.yp}, ox[3] = {q.xm, 0, q.xp};
  const bool vz[3] = {q.vzm, true, q.vzp}, vy[3] = {q.vym, true, q.vyp}, vx[3] = {q.vxm, true, q.vxp};
  constexpr int k0 = SEMI ? 1 : 0, k1 = SEMI ? 2 : 3;
  T v[27];
#pragma unroll
  for (int dk = k0; dk < k1; dk++)
#pragma unroll
    for (int dj = 0; dj < 3; dj++)
#pragma unroll
      for (int di = 0; di < 3; di++)
        v[dk * 9 + dj * 3 + di] = nval(f, q, oz[dk] + oy[dj] + ox[di], vz[dk] && vy[dj] && vx[di]);
  T s = T(0);
#pragma unroll
  for (int dk = k0; dk < k1; dk++) {
    const T wk = SEMI ? T(1) : (dk == 1 ? T(0.5) : T(0.25));
#pragma unroll
    for (int dj = 0; dj < 3; dj++) {
      const T wj = dj == 1 ? T(0.5) : T(0.25);
#pragma unroll
      for (int di = 0; di < 3; di++) s += wk * wj * (di == 1 ? T(0.5) : T(0.25)) * v[dk * 9 + dj * 3 + di];
    }
  }
  c[lin3(gc, I, J, K)] = s;
}

// The residual r = b - A x and its restriction in one kernel: a block forms the
// residuals that its CX x CY x CZ coarse cells read in shared memory, those of
// the rim again in its neighbours (405 for the 256 own ones; 306 for 256 when z
// is not coarsened, Z = kZSemi, 153 for 128 in 2-D, kZFlat), and no residual goes
// through memory.  A launch and a round trip less where latency is all that
// counts (rule: residual_restrict_fused).  Same operations as k_apply and
// k_restrict.  x and y are periodic and even on every level that is coarsened,
// and so is z where it is coarsened.
enum { kZFull = 0, kZSemi = 1, kZFlat = 2 };
template <int Z>
struct RrTile {
  static constexpr int CX = Z == kZFull ? 4 : 8, CY = 4, CZ = Z == kZFlat ? 1 : 2;
  static constexpr int FX = 2 * CX + 1, FY = 2 * CY + 1, FZ = Z == kZFull ? 2 * CZ + 1 : CZ;
  static constexpr int kThreads = (FX * FY * FZ + 31) / 32 * 32;
};
template <typename T, int Z>
__global__ void __launch_bounds__(RrTile<Z>::kThreads) k_residual_restrict(OpK o, GridG gc, const T *__restrict__ n,
                                                                           const T *__restrict__ coef,
                                                                           const T *__restrict__ x,
                                                                           const T *__restrict__ b, T *__restrict__ c) {
  ECS_PDL_ENTRY_FOR(T);
  typedef RrTile<Z> R;
  __shared__ T res[R::FZ][R::FY][R::FX];
  const int I0 = blockIdx.x * R::CX, J0 = blockIdx.y * R::CY, K0 = blockIdx.z * R::CZ;
  const int t = threadIdx.x, fx = t % R::FX, fy = t / R::FX % R::FY, fz = t / (R::FX * R::FY);
  if (fz < R::FZ) {
    int i = 2 * I0 - 1 + fx, j = 2 * J0 - 1 + fy, k = Z == kZFull ? 2 * K0 - 1 + fz : K0 + fz;
    if (i < o.g.nx && j < o.g.ny && k < o.g.nz) {  // past the last coarse cell: not read
      i = i < 0 ? o.g.nx - 1 : i;
      j = j < 0 ? o.g.ny - 1 : j;
      k = k < 0 ? o.g.nz - 1 : k;
      const Nbr q = nbr_of(o.g, i, j, k);
      T v[11], xe[11];
      row_coef(o, n, coef, q, v);
      row_x(x, q, xe);
      T s = T(0);
#pragma unroll
      for (int e = 0; e < 11; e++) s += v[e] * xe[e];
      res[fz][fy][fx] = b[q.c] - s;
    }
  }
  __syncthreads();
  const int ci = t % R::CX, cj = t / R::CX % R::CY, ck = t / (R::CX * R::CY);
  if (ck >= R::CZ || I0 + ci >= gc.nx || J0 + cj >= gc.ny || K0 + ck >= gc.nz) return;
  T s = T(0);
#pragma unroll
  for (int dk = Z == kZSemi ? 1 : 0; dk < (Z == kZSemi ? 2 : 3); dk++) {
    const T wk = Z == kZSemi ? T(1) : (dk == 1 ? T(0.5) : T(0.25));
    const int rk = Z == kZFull ? 2 * ck + dk : ck;  // flat: one plane is every neighbour along z
#pragma unroll
    for (int dj = 0; dj < 3; dj++) {
      const T wj = dj == 1 ? T(0.5) : T(0.25);
#pragma unroll
      for (int di = 0; di < 3; di++) s += wk * wj * (di == 1 ? T(0.5) : T(0.25)) * res[rk][2 * cj + dj][2 * ci + di];
    }
  }
  c[lin3(gc, I0 + ci, J0 + cj, K0 + ck)] = s;
}

// f += P c, trilinear: the coarse cells through the neighbour offsets of the
// coarse cell (i/2, j/2, k/2); a term of the second cell along an axis is
// added only for an odd index, x innermost, then y, then z.
template <typename T, bool SEMI>
__device__ __forceinline__ T prolonged(const GridG &gc, const T *__restrict__ c, T old, int i, int j, int k) {
  const Nbr q = nbr_of(gc, i >> 1, j >> 1, SEMI ? k : k >> 1);
  const bool t[3] = {(i & 1) != 0, (j & 1) != 0, !SEMI && (k & 1)};
  T v[8];
#pragma unroll
  for (int e = 0; e < 8; e++) {
    const bool x = e & 1, y = e & 2, z = e & 4;
    const bool has = (!x || (t[0] && q.vxp)) && (!y || (t[1] && q.vyp)) && (!z || (t[2] && q.vzp));
    v[e] = nval(c, q, (x ? q.xp : 0) + (y ? q.yp : 0) + (z ? q.zp : 0), has);
  }
  T s = T(0);
#pragma unroll
  for (int e = 0; e < 8; e++) {
    const bool add = (!(e & 1) || t[0]) && (!(e & 2) || t[1]) && (!(e & 4) || t[2]);
    s = add ? s + v[e] : s;
  }
  const T wi = t[0] ? T(0.5) : T(1), wj = t[1] ? T(0.5) : T(1), wk = t[2] ? T(0.5) : T(1);
  return old + wi * wj * wk * s;
}
template <typename T, bool SEMI>
__global__ void k_prolong_add(GridG gf, GridG gc, const T *__restrict__ c, T *__restrict__ f) {
  ECS_PDL_ENTRY_FOR(T);
  int i, j, k;
  if (!at3(gf.nx, gf.ny, i, j, k)) return;
  const unsigned e0 = lin3(gf, i, j, k);
  f[e0] = prolonged<T, SEMI>(gc, c, f[e0], i, j, k);
}

// The same transfers in FP32, two coarse cells (four fine ones) a thread: the
// cells' operands overlap, and the fine ones move as float4.
// k_restrict: coarse cells I, I + 1 (I even) from the fine columns 2I - 1 .. 2I + 3.
template <bool SEMI>
__global__ void __launch_bounds__(256) k_restrict2(GridG gf, GridG gc, const float *__restrict__ f,
                                                   float *__restrict__ c) {
  ECS_PDL_ENTRY();
  const int I = (int)(blockIdx.x * blockDim.x + threadIdx.x) * 2, J = (int)(blockIdx.y * blockDim.y + threadIdx.y),
            K = (int)blockIdx.z;
  if (I >= gc.nx || J >= gc.ny) return;
  const Nbr q = nbr_of(gf, 2 * I, 2 * J, SEMI ? K : 2 * K);
  const int oz[3] = {q.zm, 0, q.zp}, oy[3] = {q.ym, 0, q.yp};
  const bool vz[3] = {q.vzm, true, q.vzp};
  constexpr int k0 = SEMI ? 1 : 0, k1 = SEMI ? 2 : 3;
  float m[9];
  float4 v[9];
#pragma unroll
  for (int dk = k0; dk < k1; dk++)
#pragma unroll
    for (int dj = 0; dj < 3; dj++) {
      const unsigned r = (unsigned)((int)q.c + oz[dk] + oy[dj]);
      m[dk * 3 + dj] = vz[dk] ? f[(unsigned)((int)r + q.xm)] : 0.f;
      v[dk * 3 + dj] = vz[dk] ? ld4(f, r) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  float s0 = 0.f, s1 = 0.f;
#pragma unroll
  for (int dk = k0; dk < k1; dk++) {
    const float wk = SEMI ? 1.f : (dk == 1 ? 0.5f : 0.25f);
#pragma unroll
    for (int dj = 0; dj < 3; dj++) {
      const float w = wk * (dj == 1 ? 0.5f : 0.25f);
      const float4 u = v[dk * 3 + dj];
      s0 += w * 0.25f * m[dk * 3 + dj];
      s0 += w * 0.5f * u.x;
      s0 += w * 0.25f * u.y;
      s1 += w * 0.25f * u.y;
      s1 += w * 0.5f * u.z;
      s1 += w * 0.25f * u.w;
    }
  }
  *reinterpret_cast<float2 *>(c + lin3(gc, I, J, K)) = make_float2(s0, s1);
}
// k_prolong_add: the four fine cells of the coarse cells I, I + 1 (and I + 2).
template <bool SEMI>
__global__ void __launch_bounds__(256) k_prolong_add4(GridG gf, GridG gc, const float *__restrict__ c,
                                                      float *__restrict__ f) {
  ECS_PDL_ENTRY();
  const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x) * 4, j = (int)(blockIdx.y * blockDim.y + threadIdx.y),
            k = (int)blockIdx.z;
  if (i >= gf.nx || j >= gf.ny) return;
  const Nbr q = nbr_of(gc, i >> 1, j >> 1, SEMI ? k : k >> 1);
  const bool tj = j & 1, tk = !SEMI && (k & 1);
  const int x2 = (i >> 1) + 2 < gc.nx ? 2 : 2 - gc.nx;  // the coarse cell after the next
  float4 *p = reinterpret_cast<float4 *>(f + lin3(gf, i, j, k));
  float4 t = *p;
  float2 u[4];
  float w[4];
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const bool has = (!(e & 1) || tj) && (!(e & 2) || (tk && q.vzp));
    const unsigned r = (unsigned)((int)q.c + ((e & 2) ? q.zp : 0) + ((e & 1) ? q.yp : 0));
    u[e] = has ? *reinterpret_cast<const float2 *>(c + r) : make_float2(0.f, 0.f);
    w[e] = has ? c[(unsigned)((int)r + x2)] : 0.f;
  }
  float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const bool add = (!(e & 1) || tj) && (!(e & 2) || (tk && q.vzp));
    if (add) {
      s[0] += u[e].x;
      s[1] += u[e].x;
      s[1] += u[e].y;
      s[2] += u[e].y;
      s[3] += u[e].y;
      s[3] += w[e];
    }
  }
  const float wjk = (tj ? 0.5f : 1.f) * (tk ? 0.5f : 1.f);
  t.x += wjk * s[0];
  t.y += 0.5f * wjk * s[1];
  t.z += wjk * s[2];
  t.w += 0.5f * wjk * s[3];
  *p = t;
}
template <typename T>
int launch_restrict(EcsCtx *ctx, cudaStream_t s, const GridG &gf, const GridG &gc, const T *f, T *c) {
  bool wide = false;
  if constexpr (sizeof(T) == 4) {
    wide = use_row4(gf);
    if (wide) {
      const dim3 t = threads4(gf.nx);
      const dim3 b((unsigned)((gc.nx / 2 + (int)t.x - 1) / (int)t.x), (unsigned)((gc.ny + (int)t.y - 1) / (int)t.y), (unsigned)gc.nz);
      ecs_launch_pdl(semi_z(gf, gc) ? k_restrict2<true> : k_restrict2<false>, b, t, 0, s, gf, gc, f, c);
    }
  }
  if (!wide)
    ecs_launch_pdl(semi_z(gf, gc) ? k_restrict<T, true> : k_restrict<T, false>, blocks3(gc), threads3(), 0, s, gf, gc, f, c);
  ECS_LAUNCHED(ctx);
  return ECS_OK;
}
// FP32: x2 = x + P c and the right-hand side of the z-line systems, r = b - A_xy
// x2, in one kernel: a block prolongs its TX x TY x TZ cells and the rim that
// their rows read (432 values for 256 cells, 180 for 128 in 2-D) into shared
// memory.  x2 is another array than x, whose rim the neighbouring blocks read.
// Same operations as k_prolong_add and k_zline_rhs.
template <bool FLAT>
struct PrTile {
  static constexpr int TX = 16, TY = FLAT ? 8 : 4, TZ = FLAT ? 1 : 4;
  static constexpr int HX = TX + 2, HY = TY + 2;
  static constexpr int kThreads = (HX * HY * TZ + 31) / 32 * 32;
};
template <bool SEMI, bool FLAT>
__global__ void __launch_bounds__(PrTile<FLAT>::kThreads) k_prolong_rhs(OpK o, GridG gc, const float *__restrict__ n,
                                                                        const float *__restrict__ b,
                                                                        const float *__restrict__ c,
                                                                        const float *__restrict__ x,
                                                                        float *__restrict__ x2, float *__restrict__ r) {
  ECS_PDL_ENTRY();
  typedef PrTile<FLAT> R;
  __shared__ float xs[R::TZ][R::HY][R::HX];
  const int i0 = blockIdx.x * R::TX, j0 = blockIdx.y * R::TY, k0 = blockIdx.z * R::TZ;
  const int t = threadIdx.x;
  // this thread's own cell: its row is requested before the barrier
  const int oi = t % R::TX, oj = t / R::TX % R::TY, ok = t / (R::TX * R::TY);
  const bool own = ok < R::TZ && i0 + oi < o.g.nx && j0 + oj < o.g.ny && k0 + ok < o.g.nz;
  float v[11], s = 0.f;
  unsigned cell = 0;
  if (own) {
    const Nbr q = nbr_of(o.g, i0 + oi, j0 + oj, k0 + ok);
    cell = q.c;
    row11_n(n, o, q, v);
    s = b[q.c];
  }
  const int hx = t % R::HX, hy = t / R::HX % R::HY, hz = t / (R::HX * R::HY);
  const int i1 = i0 + hx - 1, j1 = j0 + hy - 1, k = k0 + hz;
  if (hz < R::TZ && i1 <= o.g.nx && j1 <= o.g.ny && k < o.g.nz) {
    const int i = i1 < 0 ? o.g.nx - 1 : (i1 == o.g.nx ? 0 : i1), j = j1 < 0 ? o.g.ny - 1 : (j1 == o.g.ny ? 0 : j1);
    const unsigned e = lin3(o.g, i, j, k);
    const float y = prolonged<float, SEMI>(gc, c, x[e], i, j, k);
    xs[hz][hy][hx] = y;
    if (hx >= 1 && hx <= R::TX && hy >= 1 && hy <= R::TY && i1 < o.g.nx && j1 < o.g.ny) x2[e] = y;
  }
  __syncthreads();
  if (!own) return;
#pragma unroll
  for (int e = 0; e < 10; e++) {
    if (e == 4 || e == 5) continue;
    s -= v[e] * xs[ok][oj + 1 + off_j(e)][oi + 1 + off_i(e)];
  }
  r[cell] = s;
}

template <typename T, int Z>
void launch_residual_restrict(EcsCtx *ctx, const OpK &o, const GridG &gc, const MgLevel<T> &L, const T *b, T *c) {
  typedef RrTile<Z> R;
  const dim3 g((unsigned)((gc.nx + R::CX - 1) / R::CX), (unsigned)((gc.ny + R::CY - 1) / R::CY),
               (unsigned)((gc.nz + R::CZ - 1) / R::CZ));
  ecs_launch_pdl(k_residual_restrict<T, Z>, g, R::kThreads, 0, ctx->stream, o, gc, (const T *)L.dens, (const T *)L.coef,
                 (const T *)L.t, b, c);
}
// Levels whose residual and restriction are one kernel (and, in FP32, their
// prolongation and right-hand side, k_prolong_rhs).  3-D: 32^3 solve 0.585 ->
// 0.561 ms, FP64 40 x 24 x 20 1.263 -> 1.216; on a 64^3 level the rim's second
// residuals cost more than the launch (64^3 solve 0.744 with two kernels, 0.760
// fused).  In 2-D the rim is smaller: 256^2 solve 0.748 -> 0.710 with the levels
// below 256^2 and 2 to 3 % more with it.  Where the line lies (whole solves;
// no level fused, this line, the line at twice and at three (2-D: eight) times
// the cells):
// 40^3 0.849, 0.786, 0.781-0.789 ms, 40 x 40 x 42 (67,200 cells) 0.957, 0.956, 0.966;
// 48^3 0.840, 0.805, 0.805; 56^3 0.909, 0.868, 0.868, 0.875; 2-D 320 x 400 1.124,
// 1.039; 400^2 1.610, 1.523, 1.511; 512^2 1.086, 1.020, 1.016, 1.029.
inline bool residual_restrict_fused(const GridG &g) {
  return g.n < (g.nz == 1 ? (size_t)1 << 17 : (size_t)1 << 16);
}
// c = restriction of b - A L.t
template <typename T>
int residual_restrict(EcsCtx *ctx, MgLevel<T> &L, const OpK &o, const GridG &gc, const T *b, T *c) {
  if (residual_restrict_fused(o.g)) {
    if (o.g.nz == 1) launch_residual_restrict<T, kZFlat>(ctx, o, gc, L, b, c);
    else if (semi_z(o.g, gc)) launch_residual_restrict<T, kZSemi>(ctx, o, gc, L, b, c);
    else launch_residual_restrict<T, kZFull>(ctx, o, gc, L, b, c);
    ECS_LAUNCHED(ctx);
    return ECS_OK;
  }
  bool row4 = false;
  if constexpr (sizeof(T) == 4) {
    row4 = use_row4(o.g);
    if (row4) ecs_launch_pdl(k_apply4, blocks4(o.g), threads4(L.nx), 0, ctx->stream, o, L.dens, L.t, b, L.r);
  }
  if (!row4) ecs_launch_pdl(k_apply<T>, blocks3(o.g), threads3(), 0, ctx->stream, o, L.dens, L.coef, L.t, b, L.r, 1);
  ECS_LAUNCHED(ctx);
  return launch_restrict<T>(ctx, ctx->stream, o.g, gc, L.r, c);
}
template <typename T>
int launch_prolong_add(EcsCtx *ctx, cudaStream_t s, const GridG &gf, const GridG &gc, const T *c, T *f) {
  bool wide = false;
  if constexpr (sizeof(T) == 4) {
    wide = use_row4(gf);
    if (wide)
      ecs_launch_pdl(semi_z(gf, gc) ? k_prolong_add4<true> : k_prolong_add4<false>, blocks4(gf), threads4(gf.nx), 0, s, gf,
                     gc, c, f);
  }
  if (!wide)
    ecs_launch_pdl(semi_z(gf, gc) ? k_prolong_add<T, true> : k_prolong_add<T, false>, blocks3(gf), threads3(), 0, s, gf, gc,
                   c, f);
  ECS_LAUNCHED(ctx);
  return ECS_OK;
}

// ---- whole V-cycle of the small levels in one thread block -------------------
// Levels of at most kSmallCells cells, all in one block of one thread a cell.
// Every level's 11 row coefficients, its neighbour offsets (packed), its
// z-line factors and its vectors live in shared memory (s* are offsets into
// it, in elements; sn in 4-byte words of the integer part): the coefficients
// and offsets are formed once per launch from the density, so that the
// residual, right-hand side and transfer phases are a few shared-memory loads
// and multiply-adds each.  The kernel runs each piece of its code once or a
// few times per launch, so instruction fetch and the phases' latency bound it.
// With the rows, wraps and index divisions redone in every phase and the
// columns' recurrences through shared memory it took 27 us for 8^3 + 4^3 (FP64
// 42) and 70 us for a 6^3 coarsest level of 21 sweeps; 11 (27) and 18 us in this
// form.
template <typename T>
struct SmallLevel {
  OpK o;
  const T *dens, *minv, *q, *a0g, *qden;  // in global memory
  int sx, sb, sr, st;                     // vectors
  int sco, sa, sc, sm, sq, s0, sqd;       // coefficients [11][n], factors (cells), column scalars
  int sn;                                 // packed neighbour offsets [3][n]
};
constexpr int kMaxSmall = 8;
template <typename T>
struct SmallCycle {
  int nl, ints;   // ints: element offset of the integer part
  const T *cinv;  // transposed inverse of the coarsest operator, or nullptr
  SmallLevel<T> lv[kMaxSmall];
};
constexpr size_t kSmallCells = 512;
constexpr size_t kSmallSmem = 200 * 1024;  // its shared memory at most
constexpr int kSmallThreads = (int)kSmallCells;
// Planes that a column's thread keeps in registers; deeper columns (a
// reflecting z is not coarsened) run their recurrences through shared memory.
constexpr int kSmallPlanes = 8;

// Neighbour offsets of a small level's cell in three words: (xm, xp, ym),
// (yp, zm, zp) as signed 10-bit fields, (i, j, k) as 10-bit fields.  Offsets
// are below 512 in magnitude; kNoNbr marks a ghost, whose value is 0.
constexpr int kNoNbr = -512;
__device__ __forceinline__ unsigned pack3(int a, int b, int c) {
  return ((unsigned)a & 1023u) | (((unsigned)b & 1023u) << 10) | (((unsigned)c & 1023u) << 20);
}
__device__ __forceinline__ int field_s(unsigned w, int f) { return (int)(w << (22 - 10 * f)) >> 22; }
__device__ __forceinline__ int field_u(unsigned w, int f) { return (int)((w >> (10 * f)) & 1023u); }
struct SmallNbr {
  int xm, xp, ym, yp, zm, zp;
};
__device__ __forceinline__ SmallNbr small_nbr(const unsigned *nb, int n, int c) {
  const unsigned w0 = nb[c], w1 = nb[n + c];
  return {field_s(w0, 0), field_s(w0, 1), field_s(w0, 2), field_s(w1, 0), field_s(w1, 1), field_s(w1, 2)};
}
template <typename T>
__device__ __forceinline__ T sval(const T *f, int c, int off, bool valid) {
  return valid ? f[c + off] : T(0);
}
// f at the row's entries, in the order of off_i/off_j/off_k; x and y are
// periodic on every grid the solver takes, so only z has ghosts.
template <typename T>
__device__ __forceinline__ void small_row(const T *f, int c, const SmallNbr &q, T xe[11]) {
  xe[0] = f[c + q.xp];
  xe[1] = f[c + q.xm];
  xe[2] = f[c + q.yp];
  xe[3] = f[c + q.ym];
  xe[4] = sval(f, c, q.zp, q.zp != kNoNbr);
  xe[5] = sval(f, c, q.zm, q.zm != kNoNbr);
  xe[6] = f[c + q.xp + q.yp];
  xe[7] = f[c + q.xp + q.ym];
  xe[8] = f[c + q.xm + q.yp];
  xe[9] = f[c + q.xm + q.ym];
  xe[10] = f[c];
}

// One column's z-line solve in shared memory: the right-hand side at rin (may
// be the same array as the substitution scratch dp), xo and xn the iterate in
// and out (all offsets into sm; xo < 0: zero).
template <typename T>
__device__ __forceinline__ void zline_col_s(const SmallLevel<T> &L, T *sm, int rin, int dp, int xo, int xn, T omega,
                                            int col) {
  const int plane = L.o.g.nx * L.o.g.ny, N = L.o.g.nz;
  const T *a = sm + L.sa + col, *cp = sm + L.sc + col, *minv = sm + L.sm + col, *q = sm + L.sq + col;
  const T *rp = sm + rin + col, *op = sm + (xo < 0 ? 0 : xo) + col;
  T *d_ = sm + dp + col, *xp = sm + xn + col;
  const T a0g = sm[L.s0 + col], qden = sm[L.sqd + col];
  if (N <= kSmallPlanes) {  // operands first, then the recurrences in registers
    T y[kSmallPlanes], av[kSmallPlanes], mv[kSmallPlanes], cv[kSmallPlanes];
#pragma unroll
    for (int k = 0; k < kSmallPlanes; k++)
      if (k < N) {
        y[k] = rp[k * plane];
        av[k] = a[k * plane];
        mv[k] = minv[k * plane];
        cv[k] = cp[k * plane];
      }
    T d = T(0);
#pragma unroll
    for (int k = 0; k < kSmallPlanes; k++)
      if (k < N) {
        d = (y[k] - av[k] * d) * mv[k];
        y[k] = d;
      }
    const T yN = d;
    T yk = d;
#pragma unroll
    for (int k = kSmallPlanes - 2; k >= 0; k--)
      if (k < N - 1) {
        yk = y[k] - cv[k] * yk;
        y[k] = yk;
      }
    const T s = (yk + a0g * yN) * qden;
#pragma unroll
    for (int k = 0; k < kSmallPlanes; k++)
      if (k < N) {
        const T ov = xo < 0 ? T(0) : op[k * plane];
        xp[k * plane] = ov + omega * ((y[k] - s * q[k * plane]) - ov);
      }
    return;
  }
  T d = T(0);
  for (int k = 0; k < N; k++) {
    d = (rp[k * plane] - a[k * plane] * d) * minv[k * plane];
    d_[k * plane] = d;
  }
  const T yN = d;
  T y = d;
  for (int k = N - 2; k >= 0; k--) {
    y = d_[k * plane] - cp[k * plane] * y;
    d_[k * plane] = y;
  }
  const T s = (y + a0g * yN) * qden;
  for (int k = 0; k < N; k++) {
    const T ov = xo < 0 ? T(0) : op[k * plane];
    xp[k * plane] = ov + omega * ((d_[k * plane] - s * q[k * plane]) - ov);
  }
}

// `sweeps` damped z-line Jacobi sweeps of level L: the first from xo (an
// offset; < 0: zero) into xn, the next ones back and forth between xn and
// alt.  Called up to three times a launch, so it is kept out of line (one copy
// of its code to fetch); the arrays go by their offsets, so that every access
// stays a shared-memory access.  A thread's coefficients and neighbour
// offsets stay in registers over the sweeps (one cell a thread).
template <typename T>
__device__ __noinline__ void blk_sweep(const SmallLevel<T> &L, int ints_off, int b, int xo, int xn, int alt,
                                       int sweeps, T omega) {
  extern __shared__ unsigned char small_smem[];
  T *sm = reinterpret_cast<T *>(small_smem);
  const unsigned *ints = reinterpret_cast<const unsigned *>(sm + ints_off);
  const int n = (int)L.o.g.n, ncol = L.o.g.nx * L.o.g.ny, c = threadIdx.x;
  const bool live = c < n;
  SmallNbr q = {0, 0, 0, 0, 0, 0};
  T v[8], bc = T(0);
  if (live) {
    q = small_nbr(ints + L.sn, n, c);
    const T *co = sm + L.sco + c;
#pragma unroll
    for (int e = 0; e < 8; e++) v[e] = co[(e < 4 ? e : e + 2) * n];
    bc = sm[b + c];
  }
#pragma unroll 1
  for (int sw = 0; sw < sweeps; sw++) {
    int rin = b;
    if (xo >= 0) {
      if (live) {
        const T *x = sm + xo + c;
        T s = bc;
        s -= v[0] * x[q.xp];
        s -= v[1] * x[q.xm];
        s -= v[2] * x[q.yp];
        s -= v[3] * x[q.ym];
        s -= v[4] * x[q.xp + q.yp];
        s -= v[5] * x[q.xp + q.ym];
        s -= v[6] * x[q.xm + q.yp];
        s -= v[7] * x[q.xm + q.ym];
        sm[L.sr + c] = s;
      }
      __syncthreads();
      rin = L.sr;
    }
    for (int col = threadIdx.x; col < ncol; col += blockDim.x) zline_col_s<T>(L, sm, rin, L.sr, xo, xn, omega, col);
    __syncthreads();
    xo = xn;
    xn = alt;
    alt = xo;
  }
}

// x_out = M(l0) b_in: V(1,1) over levels l0..l0+nl-1, all in this block.
template <typename T>
__global__ void __launch_bounds__(kSmallThreads) k_vcycle_small(SmallCycle<T> sc, const T *__restrict__ b_in,
                                                                T *__restrict__ x_out, int coarse_sweeps, T omega) {
  ECS_PDL_ENTRY_FOR(T);
  extern __shared__ unsigned char small_smem[];
  T *sm = reinterpret_cast<T *>(small_smem);
  unsigned *ints = reinterpret_cast<unsigned *>(sm + sc.ints);
  const int nl = sc.nl;
  // row coefficients, neighbour offsets and z-line factors of every level
  // (the coarsest of a direct solve needs the offsets only), and the
  // right-hand side
#pragma unroll 1
  for (int l = 0; l < nl; l++) {
    const SmallLevel<T> &L = sc.lv[l];
    const int n = (int)L.o.g.n, ncol = L.o.g.nx * L.o.g.ny;
    const bool direct = l == nl - 1 && sc.cinv;
    for (int c = threadIdx.x; c < n; c += blockDim.x) {
      int i, j, k;
      cell_ijk((unsigned)c, L.o.g, i, j, k);
      const Nbr q = nbr_of(L.o.g, i, j, k);
      ints[L.sn + c] = pack3(q.xm, q.xp, q.ym);
      ints[L.sn + n + c] = pack3(q.yp, q.vzm ? q.zm : kNoNbr, q.vzp ? q.zp : kNoNbr);
      ints[L.sn + 2 * n + c] = pack3(i, j, k);
      if (direct) continue;
      const T mi = __ldg(&L.minv[c]);
      sm[L.sm + c] = mi;
      sm[L.sq + c] = __ldg(&L.q[c]);
      T v[11];
      row11_n(L.dens, L.o, q, v);
#pragma unroll
      for (int e = 0; e < 11; e++) sm[L.sco + e * n + c] = v[e];
      sm[L.sa + c] = k == 0 ? T(0) : v[5];
      sm[L.sc + c] = (k == L.o.g.nz - 1 ? T(0) : v[4]) * mi;
    }
    if (!direct)
      for (int c = threadIdx.x; c < ncol; c += blockDim.x) {
        sm[L.s0 + c] = __ldg(&L.a0g[c]);
        sm[L.sqd + c] = __ldg(&L.qden[c]);
      }
    if (l == 0)
      for (int c = threadIdx.x; c < n; c += blockDim.x) sm[L.sb + c] = b_in[c];
  }
  __syncthreads();
  // down
#pragma unroll 1
  for (int l = 0; l < nl - 1; l++) {
    const SmallLevel<T> &L = sc.lv[l], &C = sc.lv[l + 1];
    const GridG &g = L.o.g, &gc = C.o.g;
    const int n = (int)g.n, nc = (int)gc.n;
    T *b = sm + L.sb, *t = sm + L.st, *r = sm + L.sr;
    blk_sweep(L, sc.ints, L.sb, -1, L.st, L.st, 1, omega);
    const T *co = sm + L.sco;
    for (int c = threadIdx.x; c < n; c += blockDim.x) {
      T xe[11];
      small_row((const T *)t, c, small_nbr(ints + L.sn, n, c), xe);
      T s = T(0);
#pragma unroll
      for (int e = 0; e < 11; e++) s += co[e * n + c] * xe[e];
      r[c] = b[c] - s;
    }
    __syncthreads();
    // full weighting, the terms in the order of k_restrict
    const bool semi = semi_z(g, gc);
    for (int c = threadIdx.x; c < nc; c += blockDim.x) {
      const unsigned w = ints[C.sn + 2 * nc + c];
      const int f = ((semi ? field_u(w, 2) : 2 * field_u(w, 2)) * g.ny + 2 * field_u(w, 1)) * g.nx + 2 * field_u(w, 0);
      const SmallNbr q = small_nbr(ints + L.sn, n, f);
      const int oz[3] = {q.zm, 0, q.zp}, oy[3] = {q.ym, 0, q.yp}, ox[3] = {q.xm, 0, q.xp};
      T s = T(0);
#pragma unroll
      for (int dk = 0; dk < 3; dk++) {
        if ((semi && dk != 1) || oz[dk] == kNoNbr) continue;
        const T wk = semi ? T(1) : (dk == 1 ? T(0.5) : T(0.25));
#pragma unroll
        for (int dj = 0; dj < 3; dj++)
#pragma unroll
          for (int di = 0; di < 3; di++)
            s += wk * (dj == 1 ? T(0.5) : T(0.25)) * (di == 1 ? T(0.5) : T(0.25)) * r[f + oz[dk] + oy[dj] + ox[di]];
      }
      sm[C.sb + c] = s;
    }
    __syncthreads();
  }
  // coarsest: direct solve with the precomputed inverse, else damped z-line
  // Jacobi sweeps; the result in its x
  if (sc.cinv) {  // x = inv b: each row's sum split over the 32 lanes of a warp
    const SmallLevel<T> &L = sc.lv[nl - 1];
    const int n = (int)L.o.g.n;
    const T *b = sm + L.sb;
    const int lane = threadIdx.x & 31;
    for (int r = threadIdx.x >> 5; r < n; r += blockDim.x >> 5) {
      T acc = T(0);
      for (int k = lane; k < n; k += 32) acc += __ldg(&sc.cinv[k * n + r]) * b[k];
      for (int s2 = 16; s2 >= 1; s2 >>= 1) acc += __shfl_xor_sync(ECS_FULL_MASK, acc, s2);
      if (lane == 0) sm[L.sx + r] = acc;
    }
    __syncthreads();
  } else {
    // into x after an odd number of sweeps
    const SmallLevel<T> &L = sc.lv[nl - 1];
    const int first = coarse_sweeps & 1 ? L.sx : L.st;
    blk_sweep(L, sc.ints, L.sb, -1, first, L.sx + L.st - first, coarse_sweeps, omega);
  }
  // up
#pragma unroll 1
  for (int l = nl - 2; l >= 0; l--) {
    const SmallLevel<T> &L = sc.lv[l], &C = sc.lv[l + 1];
    const GridG &g = L.o.g, &gc = C.o.g;
    const int n = (int)g.n, nc = (int)gc.n;
    T *t = sm + L.st;
    const T *cx = sm + C.sx;
    // trilinear prolongation, the terms in the order of k_prolong_add
    const bool semi = semi_z(g, gc);
    for (int c = threadIdx.x; c < n; c += blockDim.x) {
      const unsigned w = ints[L.sn + 2 * n + c];
      const int i = field_u(w, 0), j = field_u(w, 1), k = field_u(w, 2);
      const int q0 = ((semi ? k : k >> 1) * gc.ny + (j >> 1)) * gc.nx + (i >> 1);
      const SmallNbr q = small_nbr(ints + C.sn, nc, q0);
      const bool ti = i & 1, tj = j & 1, tk = !semi && (k & 1);
      T s = T(0);
#pragma unroll
      for (int e = 0; e < 8; e++) {
        if (((e & 1) && !ti) || ((e & 2) && !tj) || ((e & 4) && (!tk || q.zp == kNoNbr))) continue;
        s += cx[q0 + ((e & 4) ? q.zp : 0) + ((e & 2) ? q.yp : 0) + ((e & 1) ? q.xp : 0)];
      }
      t[c] += (ti ? T(0.5) : T(1)) * (tj ? T(0.5) : T(1)) * (tk ? T(0.5) : T(1)) * s;
    }
    __syncthreads();
    blk_sweep(L, sc.ints, L.sb, L.st, L.sx, L.sx, 1, omega);
  }
  {
    const SmallLevel<T> &L = sc.lv[0];
    for (int c = threadIdx.x; c < (int)L.o.g.n; c += blockDim.x) x_out[c] = sm[L.sx + c];
  }
}

// ---- sweeps of a coarsest level too large for the direct solve ---------------
// A grid whose axes turn odd early ends in a coarsest level of thousands of
// cells, solved by kCoarseSweeps damped z-line sweeps.  As two launches a sweep
// (right-hand side, z-line solve) the sweeps are launch latency, some 5 us
// each and half of a solve and more.  Here one
// thread-block cluster runs them all: the rows of the level are split over
// its CTAs, the density, the iterate and its halo rows live in shared memory,
// the right-hand side and the factors in registers, and each CTA writes its
// edge rows into its neighbours' halos through distributed shared memory
// before the cluster barrier that ends a sweep.  Thread (p, column) owns
// segment p of the column, as in k_zline_seg, with the same operations in the
// same order.  FP32 only: sixteen SMs hold too few FP64 units (the launches
// over all SMs are faster there).  Bound by the latency of a sweep's three
// barriers and, from some 20,000 cells on, by instruction issue on sixteen
// SMs: solves of 30^3 (coarsest 15^3) 1.19 -> 0.90 ms, 66 x 54 x 42 (33 x 27 x
// 21) 2.20 -> 1.68 ms, 100 x 72 x 50 (50 x 36 x 25) 3.50 -> 3.42 ms.
constexpr int kClusterMax = 16;
constexpr int kClusterSeg = 8;
constexpr size_t kClusterSmem = 220 * 1024;
__host__ __device__ __forceinline__ int row_begin(int ny, int ctas, int r) { return (int)((long long)ny * r / ctas); }

// Planes of the iterate are EW elements apart (its columns and halo rows,
// rounded up to a constant, so that a column's loads differ by immediates).
template <typename T, int EW, int kThreads>
__global__ void __launch_bounds__(kThreads, 1)
    k_coarse_sweeps(OpK o, ZCoup<T> zc, const T *__restrict__ dens, ZlP<T> z, const T *__restrict__ b,
                    T *__restrict__ xout, int rows, int sweeps, T omega) {
  ECS_PDL_ENTRY_FOR(T);
  constexpr int S = kClusterSeg;
  extern __shared__ __align__(16) unsigned char coarse_smem[];
  cg::cluster_group cl = cg::this_cluster();
  const int ctas = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int nx = o.g.nx, ny = o.g.ny, N = o.g.nz;
  const int W = rows * nx;  // columns of a CTA
  const int P = (N + S - 1) / S, NP = P * S;
  float4 *C = reinterpret_cast<float4 *>(coarse_smem);  // [2][N][W]: in-plane row entries 0-3 and 6-9
  T *X = reinterpret_cast<T *>(C + 2 * N * W);          // [2][NP][EW]: rows -1 .. R, planes past N stay 0
  T *sA = X + 2 * NP * EW, *sB = sA + P * W, *sC = sB + P * W, *sD = sC + P * W, *sLast = sD + P * W;
  const int r0 = row_begin(ny, ctas, rank), R = row_begin(ny, ctas, rank + 1) - r0;
  const int prev = rank ? rank - 1 : ctas - 1, next = rank + 1 < ctas ? rank + 1 : 0;
  T *Xprev = cl.map_shared_rank(X, prev), *Xnext = cl.map_shared_rank(X, next);
  const int prev_rows = row_begin(ny, ctas, prev + 1) - row_begin(ny, ctas, prev);
  const unsigned plane = (unsigned)(nx * ny);
  const int p = (int)threadIdx.x / W, lc = (int)threadIdx.x - p * W, lr = lc / nx, i = lc - lr * nx;
  const bool act = p < P && lr < R;
  const int k0 = p * S;
  const int j = r0 + lr, col = j * nx + i;
  auto in = [&](int q) { return act && k0 + q < N; };
  // the segment's operands; a cell past the last plane changes nothing:
  // mv = 0, fv = 0 and cv = -1 keep its d and y at 0 and the products as they are
  T bv[S], av[S], mv[S], cv[S], fv[S], qv[S], xv[S];
  {
    T nv[S + 2];
    nv[0] = in(0) && k0 > 0 ? dens[(unsigned)(k0 - 1) * plane + col] : T(0);
#pragma unroll
    for (int q = 0; q <= S; q++) nv[q + 1] = in(q) ? dens[(unsigned)(k0 + q) * plane + col] : T(0);
    T fprod = T(1);
#pragma unroll
    for (int q = 0; q < S; q++) {
      bv[q] = av[q] = mv[q] = fv[q] = qv[q] = xv[q] = T(0);
      cv[q] = T(-1);
      if (in(q)) {
        const int k = k0 + q;
        const Nbr nb = nbr_of(o.g, i, j, k);
        T v[11];
        row11_n(dens, o, nb, v);
        C[k * W + lc] = make_float4(v[0], v[1], v[2], v[3]);
        C[(N + k) * W + lc] = make_float4(v[6], v[7], v[8], v[9]);
        const unsigned c = (unsigned)k * plane + col;
        bv[q] = b[c];
        mv[q] = z.minv[c];
        qv[q] = z.q[c];
        av[q] = k == 0 ? T(0) : zc(nv[q + 1], nv[q]);
        cv[q] = (k == N - 1 ? T(0) : zc(nv[q + 1], nv[q + 2])) * mv[q];
        fprod *= -(av[q] * mv[q]);
        fv[q] = fprod;
      }
    }
    if (p < P) sB[p * W + lc] = fprod;
    T bprod = T(1);
#pragma unroll
    for (int q = S - 1; q >= 0; q--) bprod *= -cv[q];
    if (p < P) sD[p * W + lc] = bprod;
  }
  const T a0g = act ? z.a0g[col] : T(0), qden = act ? z.qden[col] : T(0);
  // element offsets of this segment's first cell and its in-plane neighbours
  const int at = k0 * EW + nx + lc, xm = i > 0 ? -1 : nx - 1, xp = i < nx - 1 ? 1 : 1 - nx;
  cl.sync();  // every CTA runs before it is written to
#pragma unroll 1
  for (int sw = 0; sw < sweeps; sw++) {
    const int buf = (sw & 1) * NP * EW, nbuf = NP * EW - buf;
    T rv[S];
#pragma unroll
    for (int q = 0; q < S; q++) rv[q] = bv[q];
    if (sw > 0 && act) {  // b - A_xy x, the entries in the order of k_zline_rhs
      const T *x0 = X + buf + at;
      const T *e0 = x0 + xp, *e1 = x0 + xm, *e2 = x0 + nx, *e3 = x0 - nx;
      const T *e6 = e0 + nx, *e7 = e0 - nx, *e8 = e1 + nx, *e9 = e1 - nx;
      const float4 *cu = C + k0 * W + lc, *cw = cu + N * W;
#pragma unroll
      for (int q = 0; q < S; q++) {
        const float4 u = *cu, w = *cw;
        const int step = k0 + q + 1 < N ? W : 0;  // past the last plane: its entries times 0
        cu += step;
        cw += step;
        T s = rv[q];
        s -= u.x * e0[q * EW];
        s -= u.y * e1[q * EW];
        s -= u.z * e2[q * EW];
        s -= u.w * e3[q * EW];
        s -= w.x * e6[q * EW];
        s -= w.y * e7[q * EW];
        s -= w.z * e8[q * EW];
        s -= w.w * e9[q * EW];
        rv[q] = s;
      }
    }
    {
      T d = T(0);
#pragma unroll
      for (int q = 0; q < S; q++) {
        d = (rv[q] - av[q] * d) * mv[q];
        rv[q] = d;
      }
      if (p < P) sA[p * W + lc] = d;
    }
    __syncthreads();
    {
      T din = T(0);
      for (int pp = 0; pp < p; pp++) din = sA[pp * W + lc] + sB[pp * W + lc] * din;
      T y = T(0), yl = T(0);
#pragma unroll
      for (int q = S - 1; q >= 0; q--) {
        y = (rv[q] + fv[q] * din) - cv[q] * y;
        rv[q] = y;
        if (k0 + q == N - 1) yl = y;
      }
      if (p < P) sC[p * W + lc] = y;
      if (p == P - 1) sLast[lc] = yl;
    }
    __syncthreads();
    if (act) {
      T yin = T(0), run = T(0);
      for (int pp = P - 1; pp >= 0; pp--) {
        if (pp == p) yin = run;
        run = sC[pp * W + lc] + sD[pp * W + lc] * run;
      }
      const T s = (run + a0g * sLast[lc]) * qden;  // run = y_0
      T bprod = T(1);
#pragma unroll
      for (int q = S - 1; q >= 0; q--) {
        bprod *= -cv[q];
        const T yk = rv[q] + bprod * yin;
        xv[q] = xv[q] + omega * ((yk - s * qv[q]) - xv[q]);
      }
      if (sw == sweeps - 1) {
#pragma unroll
        for (int q = 0; q < S; q++)
          if (in(q)) xout[(unsigned)(k0 + q) * plane + col] = xv[q];
      } else {
        T *xn = X + nbuf + at;
#pragma unroll
        for (int q = 0; q < S; q++) xn[q * EW] = xv[q];
        if (lr == 0) {
          T *h = Xprev + nbuf + k0 * EW + (prev_rows + 1) * nx + i;
#pragma unroll
          for (int q = 0; q < S; q++) h[q * EW] = xv[q];
        }
        if (lr == R - 1) {
          T *h = Xnext + nbuf + k0 * EW + i;
#pragma unroll
          for (int q = 0; q < S; q++) h[q * EW] = xv[q];
        }
      }
    }
    cl.sync();  // the halos are in place (and nothing is written after a CTA's end)
  }
}

// Cluster of the sweeps of an nx x ny x nz level: one CTA up to 2048 cells,
// then a CTA for each 2048 (a sweep of that many cells takes about as long as
// the cluster barrier), at most sixteen and one a row; 0 CTAs when the level
// does not fit (or its columns are cut into longer segments).  Solves with
// 1024, 2048 and 4096 cells a CTA: 20 x 18 x 22 0.736, 0.736, 0.736 ms; 26^3 0.740,
// 0.751, 0.836; 30^3 0.741, 0.801, 0.925; 34^3 0.953, 0.948, 1.109; 42 x 38 x 34
// 1.011, 1.209, 1.428; 66 x 54 x 42 1.496, 1.493, 1.659; 100 x 72 x 50 2.55 each.
static CoarseShape coarse_shape(int nx, int ny, int nz) {
  CoarseShape s;
  if (nz > kClusterSeg * kMaxSeg) return s;
  const int P = (nz + kClusterSeg - 1) / kClusterSeg, NP = P * kClusterSeg;
  for (int c = 1; c <= kClusterMax && c <= ny; c *= 2) {
    const int rows = (ny + c - 1) / c, ew = (rows + 2) * nx;
    const long long threads = (long long)rows * nx * P;
    const int EW = ew <= 128 ? 128 : (ew <= 256 ? 256 : 512);
    const size_t words = (size_t)8 * nz * rows * nx + (size_t)2 * NP * EW + (size_t)(4 * P + 1) * rows * nx;
    const bool fits = threads <= 640 && ew <= EW && words * sizeof(float) <= kClusterSmem;
    if (fits) {
      s.ctas = c;
      s.rows = rows;
      s.threads = (int)((threads + 31) / 32 * 32);
      s.ew = EW;
      s.smem = words * sizeof(float);
      if ((size_t)nx * ny * nz <= (size_t)2048 * c) break;
    }
  }
  return s;
}
// The instantiation for a shape's plane stride.
template <typename T>
using CoarseKernel = void (*)(OpK, ZCoup<T>, const T *, ZlP<T>, const T *, T *, int, int, T);
template <typename T>
static CoarseKernel<T> coarse_kernel(const CoarseShape &s) {
  return s.ew == 128 ? k_coarse_sweeps<T, 128, 640> : (s.ew == 256 ? k_coarse_sweeps<T, 256, 640> : k_coarse_sweeps<T, 512, 640>);
}

// ---- direct solve of the coarsest level -----------------------------------------
constexpr int kDirectMax = 128;  // largest coarsest level solved directly
constexpr int kInvTpr = 8;       // threads a row up to 64 cells

// Order-preserving integer of |a|: 0 for a NaN, which is never a pivot.
__device__ __forceinline__ unsigned pivot_key(float a) {
  return isnan(a) ? 0u : (__float_as_uint(a) & 0x7fffffffu) + 1u;
}
__device__ __forceinline__ unsigned long long pivot_key(double a) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(a) & 0x7fffffffffffffffull;
  return b > 0x7ff0000000000000ull ? 0ull : b + 1ull;
}
__device__ __forceinline__ unsigned warp_max_key(unsigned k) { return __reduce_max_sync(ECS_FULL_MASK, k); }
__device__ __forceinline__ unsigned long long warp_max_key(unsigned long long k) {
  const unsigned hi = __reduce_max_sync(ECS_FULL_MASK, (unsigned)(k >> 32));
  const unsigned lo = __reduce_max_sync(ECS_FULL_MASK, (unsigned)(k >> 32) == hi ? (unsigned)k : 0u);
  return ((unsigned long long)hi << 32) | lo;
}

// invT = (A + sigma 1 1^T)^-1, transposed (invT[k n + r] = inv[r][k]), by
// Gauss-Jordan elimination with partial pivoting, one block, the matrix in
// registers: row r belongs to the TPR threads tid / TPR == r, thread jr
// holding columns jr + TPR u (u < COLS).  sigma = mean |A_rr| / n removes the
// constant null space of a fully periodic operator (regularize = 1); without
// it the operator is regular.
// The elimination is in place: when row pr is the pivot of column c, the
// column has served its purpose, and its slot takes the column of the inverse
// that starts there (identity column pr).  Pivoting is implicit: the pivot of
// column c is the largest |M[r][c]| among rows not yet used; the row used at
// step c ends up holding row c of the inverse.  Ties go to the lowest row
// (SWAP: to the lowest position, as if rows c and pr were exchanged at each
// step), so the result is reproducible.
// A step needs two barriers: column c and the scaled pivot row pass through
// shared memory (double-buffered by the parity of c), and every warp finds the
// pivot for itself, with integer compares of |a|'s bits and warp maxima.  In
// FP64 that matters most: compares and a reciprocal in all 32 warps, and the
// half of [A | I] that is known to be zero or done, kept the one FP64 pipe
// busy for 644 us at 64 cells (157 us now; FP32 74 -> 35 us).
template <typename T, int ROWS, int TPR, bool SWAP>
__global__ void __launch_bounds__(ROWS *TPR) k_coarse_inverse(OpK o, const T *__restrict__ dens, int regularize,
                                                              T *__restrict__ invT) {
  ECS_PDL_ENTRY_FOR(T);
  constexpr int COLS = ROWS / TPR, RPL = ROWS / 32;  // columns a thread, rows a lane (pivot search)
  __shared__ T colbuf[2][ROWS];
  __shared__ T prow[2][ROWS];
  __shared__ int rowpos[ROWS], colrow[ROWS];  // step at which a row was the pivot, and the other way round
  __shared__ T wsum[32];
  __shared__ T sigma;
  const GridG &g = o.g;
  const int n = (int)g.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r = tid / TPR, jr = tid % TPR;
  const bool live = r < n;
  // Every access to M below has a compile-time index (u), so M stays in
  // registers.
  T M[COLS];
#pragma unroll
  for (int u = 0; u < COLS; u++) M[u] = T(0);
  if (live) {  // row r: the operator's entries in the reference's order
    int i, j, k;
    cell_ijk((unsigned)r, g, i, j, k);
    T v[11];
    int tc[11];
    row11(dens, o, i, j, k, v);
#pragma unroll
    for (int e = 0; e < 11; e++) {
      int ii = i + off_i(e), jj = j + off_j(e), kk = k + off_k(e);
      bool out = false;
      if (ii < 0 || ii >= g.nx) { if (g.bc[0]) out = true; else ii = ii < 0 ? ii + g.nx : ii - g.nx; }
      if (jj < 0 || jj >= g.ny) { if (g.bc[1]) out = true; else jj = jj < 0 ? jj + g.ny : jj - g.ny; }
      if (kk < 0 || kk >= g.nz) { if (g.bc[2]) out = true; else kk = kk < 0 ? kk + g.nz : kk - g.nz; }
      tc[e] = out ? -1 : (kk * g.ny + jj) * g.nx + ii;
    }
#pragma unroll
    for (int u = 0; u < COLS; u++) {
      const int q = jr + TPR * u;
#pragma unroll
      for (int e = 0; e < 11; e++)
        if (tc[e] == q) M[u] += v[e];
    }
  }
  if (regularize) {  // sigma = sum |A_rr| / n^2 over the diagonal, added to every entry of A
#pragma unroll
    for (int u = 0; u < COLS; u++)
      if (live && jr + TPR * u == r) colbuf[0][r] = fabs(M[u]);
    __syncthreads();
    T t = tid < n ? colbuf[0][tid] : T(0);
    for (int s2 = 16; s2 >= 1; s2 >>= 1) t += __shfl_xor_sync(ECS_FULL_MASK, t, s2);
    if (lane == 0) wsum[warp] = t;
    __syncthreads();
    if (tid == 0) {
      T u2 = T(0);
      for (int q = 0; q < ROWS * TPR / 32; q++) u2 += wsum[q];
      sigma = u2 / (T(n) * T(n));
    }
    __syncthreads();
    const T sg = sigma;
#pragma unroll
    for (int u = 0; u < COLS; u++)
      if (live && jr + TPR * u < n) M[u] += sg;
  }
  __syncthreads();  // colbuf[0] is free again
  if (live && jr == 0) colbuf[0][r] = M[0];  // column 0
  // the lane's rows lane + 32 g2 in the pivot search: their positions, -1 once used
  int pos[RPL];
#pragma unroll
  for (int g2 = 0; g2 < RPL; g2++) pos[g2] = lane + 32 * g2 < n ? lane + 32 * g2 : -1;
  // step c = j0 + TPR u0: column c is column u0 of the threads jr == j0
#pragma unroll
  for (int u0 = 0; u0 < COLS; u0++) {
#pragma unroll 1
    for (int j0 = 0; j0 < TPR; j0++) {
      const int c = j0 + TPR * u0;
      if (c >= n) break;
      const int b = c & 1;
      __syncthreads();  // column c complete
      decltype(pivot_key(T(0))) key[RPL], best = 0;
#pragma unroll
      for (int g2 = 0; g2 < RPL; g2++) {
        key[g2] = pos[g2] >= 0 ? pivot_key(colbuf[b][lane + 32 * g2]) : 0;
        best = key[g2] > best ? key[g2] : best;
      }
      best = warp_max_key(best);
      // the lowest position among the candidates (all unused rows if every one is NaN)
      unsigned cand = 0xffffffffu;  // position << 8 | row
#pragma unroll
      for (int g2 = 0; g2 < RPL; g2++)
        if (pos[g2] >= 0 && key[g2] == best) cand = min(cand, ((unsigned)pos[g2] << 8) | (unsigned)(lane + 32 * g2));
      cand = __reduce_min_sync(ECS_FULL_MASK, cand);
      const int pr = (int)(cand & 255u), ppos = (int)(cand >> 8);
#pragma unroll
      for (int g2 = 0; g2 < RPL; g2++) {
        if (SWAP && pos[g2] == c) pos[g2] = ppos;  // the row at position c moves to the pivot's
        if (lane + 32 * g2 == pr) pos[g2] = -1;
      }
      if (tid == 0) {
        rowpos[pr] = c;
        colrow[c] = pr;
      }
      if (r == pr) {
        const T pv = colbuf[b][pr];
        const T ip = pv != T(0) ? T(1) / pv : T(0);
        if (jr == j0) M[u0] = T(1);
#pragma unroll
        for (int u = 0; u < COLS; u++) {
          M[u] *= ip;
          prow[b][jr + TPR * u] = M[u];
        }
      }
      __syncthreads();  // scaled pivot row complete
      if (live && r != pr) {
        const T f = colbuf[b][r];
        if (jr == j0) M[u0] = T(0);
        if (f != T(0)) {
#pragma unroll
          for (int u = 0; u < COLS; u++) M[u] -= f * prow[b][jr + TPR * u];
        }
      }
      // column c + 1 for the next step: column u0 of j0 + 1, or column
      // u0 + 1 of thread 0 of the row
      if (live && c + 1 < n) {
        if (j0 + 1 < TPR) {
          if (jr == j0 + 1) colbuf[b ^ 1][r] = M[u0];
        } else if (u0 + 1 < COLS) {
          if (jr == 0) colbuf[b ^ 1][r] = M[u0 + 1 < COLS ? u0 + 1 : u0];
        }
      }
    }
  }
  __syncthreads();
  if (live) {
    const int row = rowpos[r];
#pragma unroll
    for (int u = 0; u < COLS; u++) {
      const int q = jr + TPR * u;
      if (q < n) invT[(size_t)colrow[q] * n + row] = M[u];
    }
  }
}

// ---- vectors ----------------------------------------------------------------------
// Sums of one thread use compensated (Kahan) summation in FP32; a warp adds
// its 32 lanes in T (fixed tree); from there on (warps of a block, blocks)
// the sums are FP64 in a fixed order.  FP32 sums thus need no FP64
// instruction per element, which matters on sm_103 where FP64 issues on a
// narrow pipe.  An FP64 thread sum (a dozen terms or so) is plain, one
// multiply-add a term for the norms: compensation would add four FP64
// operations a term for digits beyond what a norm or a mean needs.
template <typename T>
struct KSum {
  T s, c;
  __device__ __forceinline__ KSum() : s(T(0)), c(T(0)) {}
  __device__ __forceinline__ void add(T x) {
    const T y = x - c;
    const T t = s + y;
    c = (t - s) - y;
    s = t;
  }
  __device__ __forceinline__ T value() const { return s - c; }
};
template <>
struct KSum<double> {
  double s;
  __device__ __forceinline__ KSum() : s(0.0) {}
  __device__ __forceinline__ void add(double x) { s += x; }
  __device__ __forceinline__ double value() const { return s; }
};
template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
  for (int s = 16; s >= 1; s >>= 1) v += __shfl_xor_sync(ECS_FULL_MASK, v, s);
  return v;
}

// W consecutive elements of a vector.  W = kPack<T> (4 floats, 2 doubles)
// moves them with one 16-byte access: the caller guarantees the alignment
// (a basis vector of n cells starts on a 16-byte boundary when n % 4 == 0);
// W = 1 is the plain form.
template <typename T>
constexpr int kPack = 16 / (int)sizeof(T);
template <typename T, int W>
struct Pack {
  T v[W];
};
template <typename T, int W>
__device__ __forceinline__ Pack<T, W> ld_pack(const T *__restrict__ p) {
  Pack<T, W> r;
  if constexpr (W == 4 && sizeof(T) == 4) {
    const float4 f = *reinterpret_cast<const float4 *>(p);
    r.v[0] = f.x; r.v[1] = f.y; r.v[2] = f.z; r.v[3] = f.w;
  } else if constexpr (W == 2 && sizeof(T) == 8) {
    const double2 a = *reinterpret_cast<const double2 *>(p);
    r.v[0] = a.x; r.v[1] = a.y;
  } else {
#pragma unroll
    for (int i = 0; i < W; i++) r.v[i] = p[i];
  }
  return r;
}
template <typename T, int W>
__device__ __forceinline__ void st_pack(T *__restrict__ p, const Pack<T, W> &r) {
  if constexpr (W == 4 && sizeof(T) == 4) {
    *reinterpret_cast<float4 *>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
  } else if constexpr (W == 2 && sizeof(T) == 8) {
    *reinterpret_cast<double2 *>(p) = make_double2(r.v[0], r.v[1]);
  } else {
#pragma unroll
    for (int i = 0; i < W; i++) p[i] = r.v[i];
  }
}

// Completion ticket of a grid-wide reduction: true in the block that
// finishes last, to which every block's partials (written before the call)
// are then visible; it reads them through L2 (__ldcg).  That block puts the
// counter back to 0 for the next launch.  No block waits on another.
__device__ __forceinline__ bool last_block(unsigned int *ticket) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned int t = atomicAdd(ticket, 1u);
    last = t == gridDim.x - 1;
    if (last) {
      *ticket = 0u;
      __threadfence();
    }
  }
  __syncthreads();
  return last != 0;
}

// partial[blockIdx.x] = the block's sum of the threads' values (Kahan runs
// in T, warps in T, the block's warps in FP64).
template <typename T>
__device__ __forceinline__ void block_partial(const KSum<T> &acc, double *__restrict__ partial) {
  __shared__ double sh[32];
  const T t = warp_sum(acc.value());
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = (double)t;
  __syncthreads();
  if (threadIdx.x == 0) {
    double u = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); q++) u += sh[q];
    partial[blockIdx.x] = u;
  }
}

// Sum of partial[0..nb) in a fixed order, valid in thread 0 (the last block).
__device__ __forceinline__ double partials_total(const double *partial, int nb) {
  __shared__ double sh[32];
  double t = 0.0;
  for (int q = threadIdx.x; q < nb; q += blockDim.x) t += __ldcg(partial + q);
  t = warp_sum(t);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = t;
  __syncthreads();
  double u = 0.0;
  if (threadIdx.x == 0)
    for (int q = 0; q < (int)(blockDim.x >> 5); q++) u += sh[q];
  return u;
}

// out[q] = sum over blocks of slot q's partials (partial[q * nb + b]), one
// warp a slot, for slots 0..ns.
__device__ __forceinline__ void slot_totals(const double *partial, int ns, int nb, double *out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int q = warp; q < ns; q += (int)(blockDim.x >> 5)) {
    double t = 0.0;
    for (int b = lane; b < nb; b += 32) t += __ldcg(partial + (size_t)q * nb + b);
    t = warp_sum(t);
    if (lane == 0) out[q] = t;
  }
}

// v -= value[0]
template <typename T>
__global__ void k_sub_value(size_t n, T *__restrict__ v, const double *__restrict__ value) {
  ECS_PDL_ENTRY_FOR(T);
  const double m = value[0];
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
    v[e] = (T)((double)v[e] - m);
}

// ---- FGMRES on the device -----------------------------------------------------------
// Dot products are formed 8 slots at a time, then a fixed-order block
// reduction; slot q of block b goes to partial[q * gridDim.x + b].
constexpr int kChunk = 8;
// The warp's 8 sums at once: each exchange halves the slots a lane carries
// (4 + 2 + 1 + 1 + 1 additions instead of 8 trees of 5, the same tree for every
// slot).  In FP64 the trees held the pipe for longer than the products: dots of
// a 64^3 basis 22.9 -> 13.2 us.
template <typename T>
__device__ __forceinline__ T warp_sum8(T (&a)[kChunk], int &slot) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = kChunk / 2, s = 16; h >= 1; h /= 2, s /= 2) {
    const bool up = lane & s;
#pragma unroll
    for (int i = 0; i < kChunk / 2; i++)
      if (i < h) {
        const T send = up ? a[i] : a[i + h], keep = up ? a[i + h] : a[i];
        a[i] = keep + __shfl_xor_sync(ECS_FULL_MASK, send, s);
      }
  }
  a[0] += __shfl_xor_sync(ECS_FULL_MASK, a[0], 2);
  a[0] += __shfl_xor_sync(ECS_FULL_MASK, a[0], 1);
  slot = (lane & 16 ? 4 : 0) + (lane & 8 ? 2 : 0) + (lane & 4 ? 1 : 0);
  return a[0];
}
template <typename T>
__device__ __forceinline__ void block_chunk(const KSum<T> (&acc)[kChunk], int v0, int nslot,
                                            double *__restrict__ partial) {
  __shared__ double sh[kB / 32][kChunk];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T v[kChunk];
#pragma unroll
  for (int q = 0; q < kChunk; q++) v[q] = acc[q].value();
  int slot;
  const T t = warp_sum8(v, slot);
  if ((lane & 3) == 0) sh[warp][slot] = (double)t;
  __syncthreads();
  if (threadIdx.x < kChunk && v0 + (int)threadIdx.x < nslot) {
    double u = 0.0;
    for (int w = 0; w < kB / 32; w++) u += sh[w][threadIdx.x];
    partial[(size_t)(v0 + threadIdx.x) * gridDim.x + blockIdx.x] = u;
  }
  __syncthreads();
}

// Packs e of V_{v0}..V_{v0 + kHalf - 1} (zeros past the last vector): a few
// loads are requested before the first is used, where a load a vector inside
// the sums waited for each in turn.
constexpr int kHalf = 4;
template <typename T, int W>
__device__ __forceinline__ void ld_half(const T *__restrict__ V, size_t n, int v0, int nv, size_t e,
                                        Pack<T, W> (&v)[kHalf]) {
#pragma unroll
  for (int q = 0; q < kHalf; q++) {
#pragma unroll
    for (int i = 0; i < W; i++) v[q].v[i] = T(0);
    if (v0 + q < nv) v[q] = ld_pack<T, W>(V + (size_t)(v0 + q) * n + e * W);
  }
}

// Pass 1 of classical Gram-Schmidt: dots of V_0..V_j with w = V_{j+1}.
// Block partials, then the last block forms h1[q] (one warp a slot).  Packs
// of W cells; one resident wave of blocks (4 an SM).
template <typename T, int W>
__global__ void __launch_bounds__(kB, 4) k_dots1(size_t n, const T *__restrict__ V, KrylovDev *__restrict__ kd,
                                                 double *__restrict__ partial) {
  ECS_PDL_ENTRY_FOR(T);
  const int nv = kd->j + 1;
  const T *w = V + (size_t)nv * n;
  const size_t nw = n / W, stride = (size_t)gridDim.x * blockDim.x;
  for (int v0 = 0; v0 < nv; v0 += kChunk) {
    KSum<T> acc[kChunk];
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < nw; e += stride) {
      const Pack<T, W> we = ld_pack<T, W>(w + e * W);
#pragma unroll
      for (int h = 0; h < kChunk; h += kHalf) {
        if (v0 + h >= nv) break;
        Pack<T, W> v[kHalf];
        ld_half<T, W>(V, n, v0 + h, nv, e, v);
#pragma unroll
        for (int q = 0; q < kHalf; q++)
          if (v0 + h + q < nv) {
#pragma unroll
            for (int i = 0; i < W; i++) acc[h + q].add(v[q].v[i] * we.v[i]);
          }
      }
    }
    block_chunk(acc, v0, nv, partial);
  }
  if (!last_block(&kd->ticket[0])) return;
  slot_totals(partial, nv, (int)gridDim.x, kd->h1);
}

// Arnoldi bookkeeping of step j.  Its first part, in the last block of the
// pass-2 launch, is what the next kernel waits for: the pass-2 partials
// reduced into h2 and w.w, and the norm of the new basis vector.
__device__ __noinline__ void arnoldi_norm(KrylovDev *kd, int nb, const double *partial) {
  __shared__ double red[kSlots];
  if (kd->done) return;  // stopped before this step (b = 0): keep the state
  const int j = kd->j, nv = j + 1;
  slot_totals(partial, nv + 1, nb, red);
  __syncthreads();
  if (threadIdx.x <= j) kd->h2[threadIdx.x] = red[threadIdx.x];
  if (threadIdx.x != 0) return;
  double ss = 0.0;
  for (int q = 0; q <= j; q++) ss += red[q] * red[q];
  const double hn = sqrt(fmax(red[nv] - ss, 0.0));
  kd->hn = hn;
  kd->inv_scale = hn > 0 ? 1.0 / hn : 0.0;
  kd->jprev = j;
}

// The rest, in a block of its own beside the blocks that scale the new basis
// vector (it takes about as long as they do): column j of the Hessenberg
// matrix, the previous Givens rotations and a new one, the residual estimate
// and the decision whether the cycle stops; when it does, the solve of H y = g
// (upper triangular).  One thread works through the column, a chain of FP64
// operations, on shared memory that the block filled.
__device__ __noinline__ void arnoldi_rotate(KrylovDev *kd, cudaGraphConditionalHandle cond, int use_graph) {
  constexpr int m = kKrylovMax;
  __shared__ double col[kSlots], scs[m], ssn[m], g[m + 1], y[m];
  __shared__ double Hs[m * m];  // Hs[r * m + c]: the upper triangle's earlier columns
  __shared__ int stop;
  const int done0 = kd->done, j = kd->j, tid = threadIdx.x;
  if (done0) {  // stopped before this step (b = 0): keep the state
    if (tid == 0 && use_graph) cudaGraphSetConditional(cond, 0u);
    return;
  }
  for (int e = tid; e < j; e += blockDim.x) {
    scs[e] = kd->cs[e];
    ssn[e] = kd->sn[e];
  }
  for (int e = tid; e <= j; e += blockDim.x) {
    g[e] = kd->g[e];
    col[e] = kd->h1[e] + kd->h2[e];
  }
  for (int e = tid; e < j * j; e += blockDim.x) Hs[(e / j) * m + e % j] = kd->H[(e / j) * m + e % j];
  __syncthreads();
  if (tid == 0) {
    const double hn = kd->hn;
    col[j + 1] = hn;
    for (int q = 0; q < j; q++) {
      const double a = col[q], c = col[q + 1];
      col[q] = fma(scs[q], a, ssn[q] * c);
      col[q + 1] = fma(scs[q], c, -ssn[q] * a);
    }
    const double a = col[j], c = hn;
    const double r = sqrt(fma(a, a, c * c));
    const double cs = r > 0 ? a / r : 1.0, sn = r > 0 ? c / r : 0.0;
    kd->cs[j] = cs;
    kd->sn[j] = sn;
    col[j] = r;
    const double g1 = -sn * g[j], g0 = cs * g[j];
    kd->g[j + 1] = g1;
    kd->g[j] = g0;
    g[j] = g0;
    const double res = fabs(g1);
    kd->res = res;
    kd->nits = j + 1;
    const int done = (res <= kd->tol_rel * kd->beta) || hn == 0.0 || (j + 1 >= kd->maxit) ||
                     (j + 1 >= kKrylovMax) || !isfinite(res);
    kd->done = done;
    if (!done) kd->j = j + 1;
    if (use_graph) cudaGraphSetConditional(cond, done ? 0u : 1u);
    stop = done;
    if (done)
      for (int q = j; q >= 0; q--) {
        double t = g[q];
        for (int r2 = q + 1; r2 <= j; r2++) t -= (r2 == j ? col[q] : Hs[q * m + r2]) * y[r2];
        y[q] = t / (q == j ? col[j] : Hs[q * m + q]);
      }
  }
  __syncthreads();
  if (tid <= j) {
    kd->H[tid * m + j] = col[tid];
    if (stop) kd->y[tid] = y[tid];
  }
}

// w = V_{j+1} - sum_q h1[q] V_q (stored, in the first slot chunk), then
// pass 2: partial dots of V_0..V_j with the new w (slots 0..j) and of w with
// itself (slot j+1); the last block forms the new vector's norm.
template <typename T, int W>
__global__ void __launch_bounds__(kB, 4) k_orth1_dots2(size_t n, T *__restrict__ V, KrylovDev *__restrict__ kd,
                                                       double *__restrict__ partial) {
  ECS_PDL_ENTRY_FOR(T);
  __shared__ T hs[kSlots];
  const int nv = kd->j + 1, nslot = nv + 1;
  if (threadIdx.x < kSlots) hs[threadIdx.x] = (int)threadIdx.x < nv ? (T)kd->h1[threadIdx.x] : T(0);
  __syncthreads();
  T *w = V + (size_t)nv * n;
  const size_t nw = n / W, stride = (size_t)gridDim.x * blockDim.x;
  for (int v0 = 0; v0 < nslot; v0 += kChunk) {
    KSum<T> acc[kChunk];
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < nw; e += stride) {
      Pack<T, W> s = ld_pack<T, W>(w + e * W);
      if (v0 == 0) {
        for (int h = 0; h < nv; h += kHalf) {
          Pack<T, W> v[kHalf];
          ld_half<T, W>(V, n, h, nv, e, v);
#pragma unroll
          for (int q = 0; q < kHalf; q++)
            if (h + q < nv) {
              const T hq = hs[h + q];
#pragma unroll
              for (int i = 0; i < W; i++) s.v[i] -= hq * v[q].v[i];
            }
        }
        st_pack<T, W>(w + e * W, s);
      }
#pragma unroll
      for (int h = 0; h < kChunk; h += kHalf) {
        if (v0 + h > nv) break;
        Pack<T, W> v[kHalf];
        ld_half<T, W>(V, n, v0 + h, nv, e, v);
#pragma unroll
        for (int q = 0; q < kHalf; q++) {
          if (v0 + h + q < nv) {
#pragma unroll
            for (int i = 0; i < W; i++) acc[h + q].add(v[q].v[i] * s.v[i]);
          } else if (v0 + h + q == nv) {
#pragma unroll
            for (int i = 0; i < W; i++) acc[h + q].add(s.v[i] * s.v[i]);
          }
        }
      }
    }
    block_chunk(acc, v0, nslot, partial);
  }
  if (!last_block(&kd->ticket[1])) return;
  arnoldi_norm(kd, (int)gridDim.x, partial);
}

// V_{j+1} = (w - sum_q h2[q] V_q) / h_{j+1,j}, also copied to the
// preconditioner input vin (j = the step that just finished: the fields read
// here are those of arnoldi_norm).  Block 0 does the rest of the bookkeeping
// meanwhile.
template <typename T, int W>
__global__ void k_orth2_scale(size_t n, T *__restrict__ V, KrylovDev *kd, T *__restrict__ vin,
                              cudaGraphConditionalHandle cond, int use_graph) {
  ECS_PDL_ENTRY_FOR(T);
  if (blockIdx.x == 0) {
    arnoldi_rotate(kd, cond, use_graph);
    return;
  }
  __shared__ T h[kSlots + 1];
  const int j = kd->jprev, nv = j + 1;
  if (threadIdx.x < kSlots) h[threadIdx.x] = (int)threadIdx.x < nv ? (T)kd->h2[threadIdx.x] : T(0);
  if (threadIdx.x == kSlots) h[kSlots] = (T)kd->inv_scale;
  __syncthreads();
  T *w = V + (size_t)(j + 1) * n;
  const T sc = h[kSlots];
  const size_t nw = n / W, stride = (size_t)(gridDim.x - 1) * blockDim.x;
  for (size_t e = (size_t)(blockIdx.x - 1) * blockDim.x + threadIdx.x; e < nw; e += stride) {
    Pack<T, W> s = ld_pack<T, W>(w + e * W);
    for (int v0 = 0; v0 < nv; v0 += kHalf) {
      Pack<T, W> v[kHalf];
      ld_half<T, W>(V, n, v0, nv, e, v);
#pragma unroll
      for (int q = 0; q < kHalf; q++)
        if (v0 + q < nv) {
          const T hq = h[v0 + q];
#pragma unroll
          for (int i = 0; i < W; i++) s.v[i] -= hq * v[q].v[i];
        }
    }
#pragma unroll
    for (int i = 0; i < W; i++) s.v[i] *= sc;
    st_pack<T, W>(w + e * W, s);
    st_pack<T, W>(vin + e * W, s);
  }
}

// Z_j = x - mean (mean = nullptr: x) and V_{j+1} = A Z_j.  Z_j is formed
// at every stencil point on the fly, with the rounding of the stored value;
// a mean is removed only on fully periodic grids, which have no ghosts.
template <typename T>
__global__ void k_apply_dyn(OpK o, const T *__restrict__ n, const T *__restrict__ coef, const T *__restrict__ x,
                            const double *__restrict__ mean, T *__restrict__ Z, T *__restrict__ V,
                            const KrylovDev *__restrict__ kd) {
  ECS_PDL_ENTRY_FOR(T);
  int i, j, k;
  if (!at3(o.g.nx, o.g.ny, i, j, k)) return;
  const int jj = kd->j;
  const T m = mean ? (T)mean[0] : T(0);
  const Nbr q = nbr_of(o.g, i, j, k);
  const unsigned c = q.c;
  T v[11], xe[11];
  row_coef(o, n, coef, q, v);
  row_x(x, q, xe);
  T s = T(0);
#pragma unroll
  for (int e = 0; e < 11; e++) s += v[e] * (xe[e] - m);
  Z[(size_t)jj * o.g.n + c] = x[c] - m;
  V[(size_t)(jj + 1) * o.g.n + c] = s;
}

// Device state of the iterative-refinement loop.
struct RefineDev {
  double bnorm, rel;
  int its, sweeps;
  int done;  // converged, out of iterations, stalled or non-finite
  int nonfinite;
};

// Refinement sweeps in one solve: each sweep runs at least one FGMRES step
// (or ends the solve), so max_it bounds them; this caps the loop regardless.
constexpr int kMaxSweeps = 64;

// What the norm that ends a refinement sweep (or starts the solve) decides.
struct RefineArgs {
  RefineDev *rd;
  double rtol, tol_floor;
  int max_it;
  int decide;  // 0: set the state up only
  int after;   // 1: the residual is that of a finished sweep
};
// Relative residual of the current sweep from its norm; decides whether
// another correction follows (condition `cond` of the sweep loop) and sets
// the FGMRES tolerance and step limit of that correction.
__device__ __forceinline__ void refine_decide(const RefineArgs &ra, KrylovDev *kd, double norm,
                                              cudaGraphConditionalHandle cond) {
  RefineDev *rd = ra.rd;
  if (ra.after) {
    rd->its += kd->nits;
    rd->sweeps += 1;
    if (kd->nits == 0) rd->done = 1;
  }
  if (rd->bnorm > 0.0) {
    const double rel = norm / rd->bnorm;
    rd->rel = rel;
    if (!isfinite(rel)) rd->nonfinite = 1;
  }
  const bool stop = rd->done || rd->nonfinite || rd->rel <= ra.rtol || rd->its >= ra.max_it || rd->sweeps >= kMaxSweeps;
  if (stop) {
    rd->done = 1;
  } else {
    const double tol = fmax(fmax(0.5 * ra.rtol / rd->rel, 1e-14), ra.tol_floor);
    kd->tol_rel = tol;
    kd->maxit = min(kKrylovMax, max(ra.max_it - rd->its, 1));
  }
  cudaGraphSetConditional(cond, stop ? 0u : 1u);
}

// Start of an FGMRES cycle on a vector of norm sqrt(u2).  In a graph it also
// (re)arms the Arnoldi loop's condition, which keeps its last value between
// cycles of one launch.
__device__ __forceinline__ void cycle_begin(KrylovDev *kd, double u2, cudaGraphConditionalHandle cond, int use_graph) {
  const double beta = sqrt(u2);
  kd->beta = beta;
  kd->res = beta;
  kd->j = 0;
  kd->jprev = 0;
  kd->nits = 0;
  kd->done = !(beta > 0.0) || kd->maxit < 1;
  kd->inv_scale = beta > 0.0 ? 1.0 / beta : 0.0;
  for (int q = 0; q <= kKrylovMax; q++) kd->g[q] = 0.0;
  kd->g[0] = beta;
  if (use_graph) cudaGraphSetConditional(cond, kd->done ? 0u : 1u);
}

// Grid-wide sums of a vector in packs of W, finished by the last block:
//   kRedMean   out[0] = sum(v) / div
//   kRedNorm   out[0] = ||v||, out[1] = 1 / ||v|| (0 for v = 0)
//   kRedBeta   start of an FGMRES cycle: beta = ||v|| into the control block
//   kRedInit   kRedNorm of the right-hand side, which sets the refinement
//              state up (and decides on the first correction: ra.decide)
//   kRedCheck  kRedNorm of a residual, and the refinement loop's decision
// The decisions ride on the reductions because a one-thread kernel of their
// own costs a launch (2 to 3 us) each.
enum { kRedMean = 0, kRedNorm = 1, kRedBeta = 2, kRedInit = 3, kRedCheck = 4 };
template <typename T, int W, int M>
__global__ void __launch_bounds__(kB) k_reduce(size_t nw, const T *__restrict__ v, double *__restrict__ partial,
                                               double div, double *out, KrylovDev *kd,
                                               cudaGraphConditionalHandle cond, int use_graph, RefineArgs ra) {
  ECS_PDL_ENTRY_FOR(T);
  KSum<T> acc;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < nw; e += (size_t)gridDim.x * blockDim.x) {
    const Pack<T, W> p = ld_pack<T, W>(v + e * W);
#pragma unroll
    for (int i = 0; i < W; i++) acc.add(M == kRedMean ? p.v[i] : p.v[i] * p.v[i]);
  }
  block_partial(acc, partial);
  if (!last_block(&kd->ticket[2 + M])) return;
  const double u = partials_total(partial, (int)gridDim.x);
  if (threadIdx.x != 0) return;
  if (M == kRedMean) {
    out[0] = u / div;
  } else if (M == kRedBeta) {
    cycle_begin(kd, u, cond, use_graph);
  } else {
    const double norm = sqrt(u);
    out[0] = norm;
    out[1] = u > 0.0 ? 1.0 / sqrt(u) : 0.0;
    if (M == kRedInit) {
      RefineDev *rd = ra.rd;
      rd->bnorm = norm;
      rd->rel = 0.0;
      rd->its = 0;
      rd->sweeps = 0;
      rd->done = !(norm > 0.0);
      rd->nonfinite = 0;
    }
    if ((M == kRedInit && ra.decide) || M == kRedCheck) refine_decide(ra, kd, norm, cond);
  }
}

// The normalised FP64 residual to FP32, d = s scale[0], and the cycle's
// beta = ||d||, with the sums of k_reduce.  The first sweep from phi = 0
// (rd, its s0) takes the right-hand side for the residual.
template <int W>
__global__ void __launch_bounds__(kB) k_scale_beta(size_t nw, const double *__restrict__ s0,
                                                   const double *__restrict__ s1, const RefineDev *rd,
                                                   const double *__restrict__ scale, float *__restrict__ d,
                                                   double *__restrict__ partial, KrylovDev *kd,
                                                   cudaGraphConditionalHandle cond, int use_graph) {
  ECS_PDL_ENTRY();
  const double *s = rd && rd->sweeps == 0 ? s0 : s1;
  const float a = (float)scale[0];
  KSum<float> acc;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < nw; e += (size_t)gridDim.x * blockDim.x) {
    Pack<float, W> p;
    if constexpr (W == 4) {
      const Pack<double, 2> lo = ld_pack<double, 2>(s + e * 4), hi = ld_pack<double, 2>(s + e * 4 + 2);
      p.v[0] = (float)lo.v[0] * a;
      p.v[1] = (float)lo.v[1] * a;
      p.v[2] = (float)hi.v[0] * a;
      p.v[3] = (float)hi.v[1] * a;
    } else {
      p.v[0] = (float)s[e] * a;
    }
    st_pack<float, W>(d + e * W, p);
#pragma unroll
    for (int i = 0; i < W; i++) acc.add(p.v[i] * p.v[i]);
  }
  block_partial(acc, partial);
  if (!last_block(&kd->ticket[7])) return;
  const double u = partials_total(partial, (int)gridDim.x);
  if (threadIdx.x == 0) cycle_begin(kd, u, cond, use_graph);
}

// V_0 = b / beta, vin = V_0
template <typename T>
__global__ void k_cycle_start(size_t n, const T *__restrict__ b, T *__restrict__ V, T *__restrict__ vin,
                              const KrylovDev *__restrict__ kd) {
  ECS_PDL_ENTRY_FOR(T);
  const T sc = (T)kd->inv_scale;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const T v = b[e] * sc;
    V[e] = v;
    vin[e] = v;
  }
}

// End of a cycle, one pass over Z and phi: phi += scale[0] sum_q y[q] Z_q
// (scale nullptr: 1), and with MEAN also mean[0] = the mean of the new phi,
// with the sums of k_reduce (packs of W cells).
template <typename T, int W, bool MEAN>
__global__ void __launch_bounds__(kB) k_cycle_finish(size_t nw, size_t n, const T *__restrict__ Z, KrylovDev *kd,
                                                     const double *__restrict__ scale, double *__restrict__ phi,
                                                     double *__restrict__ partial, double *mean) {
  ECS_PDL_ENTRY_FOR(T);
  __shared__ T y[kKrylovMax];
  const int nj = kd->nits;
  const double a = scale ? scale[0] : 1.0;
  if (threadIdx.x < kKrylovMax) y[threadIdx.x] = (int)threadIdx.x < nj ? (T)kd->y[threadIdx.x] : T(0);
  __syncthreads();
  KSum<double> acc;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < nw; e += (size_t)gridDim.x * blockDim.x) {
    Pack<double, W> p = ld_pack<double, W>(phi + e * W);
    T s[W];
#pragma unroll
    for (int i = 0; i < W; i++) s[i] = T(0);
#pragma unroll 4
    for (int q = 0; q < nj; q++) {
      const T yq = y[q], *zq = Z + (size_t)q * n + e * W;
      T zv[W];
      if constexpr (W == 2 && sizeof(T) == 4) {
        const float2 f = *reinterpret_cast<const float2 *>(zq);
        zv[0] = f.x;
        zv[1] = f.y;
      } else {
        const Pack<T, W> f = ld_pack<T, W>(zq);
#pragma unroll
        for (int i = 0; i < W; i++) zv[i] = f.v[i];
      }
#pragma unroll
      for (int i = 0; i < W; i++) s[i] += yq * zv[i];
    }
#pragma unroll
    for (int i = 0; i < W; i++) {
      p.v[i] += a * (double)s[i];
      if (MEAN) acc.add(p.v[i]);
    }
    st_pack<double, W>(phi + e * W, p);
  }
  if constexpr (MEAN) {
    block_partial(acc, partial);
    if (!last_block(&kd->ticket[2 + kRedMean])) return;
    const double u = partials_total(partial, (int)gridDim.x);
    if (threadIdx.x == 0) mean[0] = u / (double)n;
  }
}

// ---- host side -----------------------------------------------------------------------
unsigned int blocks_for(const EcsCtx *ctx, size_t n) {
  size_t want = (n + kB - 1) / kB;
  size_t cap = (size_t)ctx->nsm * 8;
  if (want > cap) want = cap;
  return (unsigned int)(want ? want : 1);
}
// Grid of a reduction over `units` packs: at most one resident wave (4
// blocks of kB threads an SM), so that no block starts after another's end.
unsigned int dot_blocks(const EcsCtx *ctx, size_t units) {
  size_t want = (units + kB - 1) / kB;
  want = std::min(want, std::min((size_t)ctx->nsm * 4, (size_t)kDotBlocks));
  return (unsigned int)(want ? want : 1);
}
// Vectors go in packs of 4 cells (16-byte accesses) when every basis vector
// starts on a 16-byte boundary, i.e. when the cell count is a multiple of 4.
inline bool packed4(size_t n) { return (n & 3) == 0; }

// A grid-wide sum of v (kRed* mode M) on the context's stream.
template <typename T, int M>
int launch_reduce(EcsCtx *ctx, size_t n, const T *v, double div, double *out, cudaGraphConditionalHandle cond,
                  int use_graph, const RefineArgs &ra = RefineArgs()) {
  KrylovDev *kd = (KrylovDev *)ctx->kdev;
  constexpr int W = kPack<T>;
  if (packed4(n))
    ecs_launch_pdl(k_reduce<T, W, M>, dot_blocks(ctx, n / W), kB, 0, ctx->stream, n / W, v, ctx->red, div, out, kd, cond, use_graph, ra);
  else
    ecs_launch_pdl(k_reduce<T, 1, M>, dot_blocks(ctx, n), kB, 0, ctx->stream, n, v, ctx->red, div, out, kd, cond, use_graph, ra);
  ECS_LAUNCHED(ctx);
  return ECS_OK;
}

bool fully_periodic(const EcsCtx *ctx) {
  return ctx->p.bc[0] == ECS_BC_PERIODIC && ctx->p.bc[1] == ECS_BC_PERIODIC && ctx->p.bc[2] == ECS_BC_PERIODIC;
}

// The density the operator is built from (-lhs laplacian ignores it: see
// make_op).
const double *op_density(const EcsCtx *ctx) { return ctx->mom; }
bool identity_lhs(const EcsCtx *ctx) { return ctx->p.lhs_type == ECS_LHS_IDENTITY; }

template <typename T>
Multigrid<T> &mg_of(EcsCtx *ctx);
template <>
Multigrid<double> &mg_of<double>(EcsCtx *ctx) { return ctx->mg64; }
template <>
Multigrid<float> &mg_of<float>(EcsCtx *ctx) { return ctx->mg32; }

template <typename T>
int coarse_attrs(EcsCtx *ctx, CoarseShape &cs);

// The levels of the hierarchy, finest first.
std::vector<MgDims> mg_dims(const EcsParams &p) {
  std::vector<MgDims> lv;
  int nx = p.Nx, ny = p.Ny, nz = p.Nz;
  double hx = p.dx, hy = p.dy, hz = p.dz;
  for (;;) {
    lv.push_back({nx, ny, nz, hx, hy, hz});
    // A 2-D grid (nz = 1) coarsens in x and y only.  So does a grid with a
    // reflecting z: its ghost planes one spacing outside the walls do not
    // nest under z coarsening, and the z-line smoother resolves z on every
    // level, so the levels keep all planes down to one column (x y = 1 x 1,
    // whose Nz cells the coarsest inverse solves directly).
    const bool flat = nz == 1;
    const bool semi = !flat && p.bc[2] != ECS_BC_PERIODIC;
    if (semi) {
      if (nx % 2 || ny % 2 || lv.size() >= 12) break;
    } else {
      bool even = (nx % 2 == 0) && (ny % 2 == 0) && (flat || nz % 2 == 0);
      if (!even || std::min(nx, std::min(ny, flat ? nx : nz)) < 8 || lv.size() >= 12) break;
    }
    nx /= 2; ny /= 2;
    hx *= 2; hy *= 2;
    if (!flat && !semi) {
      nz /= 2;
      hz *= 2;
    }
  }
  return lv;
}

// What mg_alloc allocates for these levels.
template <typename T>
void mg_bytes(const std::vector<MgDims> &lv, DeviceBytes &b) {
  for (size_t l = 0; l < lv.size(); l++) {
    const int64_t plane = (int64_t)lv[l].nx * lv[l].ny, n = plane * lv[l].nz;
    for (int q = 0; q < (zl_stored<T>(seg_len<T>(lv[l].nz)) ? 11 : 7); q++) b.add(n * sizeof(T));
    for (int q = 0; q < 2; q++) b.add(plane * sizeof(T));
    if (sizeof(T) == 8 && l > 0) b.add(11 * n * sizeof(T));
  }
  const MgDims &c = lv.back();
  const int64_t nc = (int64_t)c.nx * c.ny * c.nz;
  if (nc <= kDirectMax) b.add(nc * nc * sizeof(T));
}

template <typename T>
void free_mg(Multigrid<T> &mg);

// An array added here goes into mg_bytes too.
template <typename T>
int mg_alloc_levels(EcsCtx *ctx, Multigrid<T> &mg) {
  int rc;
  for (const MgDims &d : mg_dims(ctx->p)) {
    mg.lv.emplace_back();
    MgLevel<T> &L = mg.lv.back();
    L.nx = d.nx; L.ny = d.ny; L.nz = d.nz;
    L.n = (size_t)d.nx * d.ny * d.nz;
    L.hx = d.hx; L.hy = d.hy; L.hz = d.hz;
    T **arr[] = {&L.dens, &L.x, &L.b, &L.r, &L.t, &L.zl_minv, &L.zl_q};
    for (auto a : arr)
      if ((rc = ecs_dev_alloc(ctx, *a, L.n * sizeof(T)))) return rc;
    if constexpr (sizeof(T) == 8) {
      if (mg.lv.size() == 1) L.coef = ctx->coef64;
      else if ((rc = ecs_dev_alloc(ctx, L.coef, 11 * L.n * sizeof(T)))) return rc;
    }
    if (zl_stored<T>(seg_len<T>(L.nz))) {
      T **more[] = {&L.zl_a, &L.zl_cp, &L.zl_fb, &L.zl_bb};
      for (auto a : more)
        if ((rc = ecs_dev_alloc(ctx, *a, L.n * sizeof(T)))) return rc;
    }
    for (auto a : {&L.zl_a0g, &L.zl_qden})
      if ((rc = ecs_dev_alloc(ctx, *a, (size_t)L.nx * L.ny * sizeof(T)))) return rc;
  }
  const size_t nc = mg.lv.back().n;
  if (nc <= (size_t)kDirectMax) {
    if ((rc = ecs_dev_alloc(ctx, mg.cinv, nc * nc * sizeof(T)))) return rc;
  } else if constexpr (sizeof(T) == 4) {
    const MgLevel<T> &C = mg.lv.back();
    CoarseShape cs = coarse_shape(C.nx, C.ny, C.nz);
    if (cs.ctas > 0) {
      rc = coarse_attrs<T>(ctx, cs);
      if (rc) return rc;
    }
    mg.cluster = cs;
  }
  return ECS_OK;
}

// The whole hierarchy or, when an allocation fails, none of it: a later call
// starts anew.
template <typename T>
int mg_alloc(EcsCtx *ctx) {
  Multigrid<T> &mg = mg_of<T>(ctx);
  if (mg.built) return ECS_OK;
  // on the device of every context: a flag for the process would leave others out
  ECS_CUDA(ctx, cudaFuncSetAttribute(k_vcycle_small<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmem));
  const int rc = mg_alloc_levels<T>(ctx, mg);
  if (rc) free_mg(mg);
  else mg.built = true;
  return rc;
}

template <typename T>
ZlP<T> zl_of(MgLevel<T> &L) {
  ZlP<T> z;
  z.a = L.zl_a; z.cp = L.zl_cp; z.minv = L.zl_minv; z.q = L.zl_q; z.fb = L.zl_fb; z.bb = L.zl_bb;
  z.a0g = L.zl_a0g; z.qden = L.zl_qden;
  return z;
}
template <typename T>
OpK op_level(const EcsCtx *ctx, const MgLevel<T> &L) {
  return make_op(ctx->p, L.nx, L.ny, L.nz, L.hx, L.hy, L.hz);
}
GridG grid_level(const EcsCtx *ctx, int nx, int ny, int nz) { return make_grid(ctx->p, nx, ny, nz); }

constexpr int kColBlock = 32;  // one warp a block: the columns spread over the SMs
constexpr int kCoarseSweeps = 21;
template <typename T>
constexpr T kOmega() { return T(0.8); }

// Level densities (level 0 from the deposited density, coarser ones by full
// weighting) and the z-line factorisation of every level.
template <typename T>
__global__ void k_density_in(size_t n, const double *__restrict__ mom, T *__restrict__ d) {
  ECS_PDL_ENTRY_FOR(T);
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
    d[e] = (T)mom[e];
}

int ensure_setup_streams(EcsCtx *ctx) {
  for (auto &c : ctx->sst)
    if (!c) ECS_CUDA(ctx, cudaStreamCreateWithFlags(&c, cudaStreamNonBlocking));
  for (auto &e : ctx->sev)
    if (!e) ECS_CUDA(ctx, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  return ECS_OK;
}

// The 11 FP64 row coefficients of every cell, coef[e * n + c] (e in the
// order of off_i/off_j/off_k), computed once per operator set-up: FP64
// arithmetic runs at a small fraction of the FP32 rate on this GPU, and the
// coefficients take about three quarters of a residual's FP64 operations.
// Densities that are whole quanta 2^-S (S given for those of a mixed deposit)
// have their sums formed in integers: 33 -> 15 FP64 operations a cell (128^3:
// 140 -> 70 us).
__global__ void k_coef64(OpK o, int S, const double *__restrict__ n, double *__restrict__ coef) {
  ECS_PDL_ENTRY();
  int i, j, k;
  if (!at3(o.g.nx, o.g.ny, i, j, k)) return;
  const Nbr q = nbr_of(o.g, i, j, k);
  const double m[7] = {n[q.c],
                       nval(n, q, q.xm, q.vxm), nval(n, q, q.xp, q.vxp), nval(n, q, q.ym, q.vym),
                       nval(n, q, q.yp, q.vyp), nval(n, q, q.zm, q.vzm), nval(n, q, q.zp, q.vzp)};
  long long a[7];
  bool whole = S != kNoQuanta && !o.unit && quanta_of(m[0], S, a[0]);  // other densities mostly end here
  if (whole) {
#pragma unroll
    for (int e = 1; e < 7; e++) whole &= quanta_of(m[e], S, a[e]);
  }
  double v[11];
  if (whole) row11_quanta(o, S, a[0], a[1], a[2], a[3], a[4], a[5], a[6], v);
  else row11_vals(o, m[0], m[1], m[2], m[3], m[4], m[5], m[6], v);
#pragma unroll
  for (int e = 0; e < 11; e++) coef[(size_t)e * o.g.n + q.c] = v[e];
}

// z-line rows and factors of level L on stream s.
template <typename T>
int zline_factor(EcsCtx *ctx, MgLevel<T> &L, cudaStream_t s) {
  const int ncol = L.nx * L.ny;
  const OpK o = op_level(ctx, L);
  if constexpr (sizeof(T) == 8) {
    if (&L != &mg_of<T>(ctx).lv[0]) {  // the finest level's are computed beside this
      ecs_launch_pdl(k_coef64, blocks3(o.g), threads3(), 0, s, o, kNoQuanta, (const double *)L.dens, L.coef);
      ECS_LAUNCHED(ctx);
    }
  }
  ecs_launch_pdl(k_zline_rows<T>, blocks3(o.g), threads3(), 0, s, o, L.dens, L.r);  // r is free here
  ECS_LAUNCHED(ctx);
  ecs_launch_pdl(k_zline_setup<T>, ecs_div_up(ncol, kColBlock), kColBlock, 0, s, o.g, z_coupling<T>(o), L.dens, L.r, zl_of(L), seg_len<T>(L.nz));
  ECS_LAUNCHED(ctx);
  return ECS_OK;
}

// Operator set-up of the multigrid levels: level densities, z-line factors,
// coarsest inverse, and the FP64 row coefficients of the refinement
// residuals.  The pieces are latency-bound small launches with few
// dependencies (and one FP64-bound kernel), so they run on four streams
// (also inside a graph capture, where the fork and join become graph edges):
//   context stream: fine density, fine z-line factors
//   sst[0]:         restriction chain of the densities, then the coarse inverse
//   sst[1]:         z-line factors of the coarse levels (after the chain)
//   sst[2]:         FP64 row coefficients
// and the context stream waits for the side streams at the end.
template <typename T>
int mg_setup(EcsCtx *ctx) {
  int rc = mg_alloc<T>(ctx);
  if (rc) return rc;
  if ((rc = ensure_setup_streams(ctx))) return rc;
  Multigrid<T> &mg = mg_of<T>(ctx);
  cudaStream_t s0 = ctx->stream, sa = ctx->sst[0], sb = ctx->sst[1], sc = ctx->sst[2];
  MgLevel<T> &L0 = mg.lv[0];
  ECS_CUDA(ctx, cudaEventRecord(ctx->sev[4], s0));
  ECS_CUDA(ctx, cudaStreamWaitEvent(sc, ctx->sev[4], 0));
  {
    const EcsParams &p = ctx->p;
    const OpK o64 = make_op(p, p.Nx, p.Ny, p.Nz, p.dx, p.dy, p.dz);
    ecs_launch_pdl(k_coef64, blocks3(o64.g), threads3(), 0, sc, o64,
                   ctx->mom_quanta ? ctx->shift_n : kNoQuanta, op_density(ctx), ctx->coef64);
    ECS_LAUNCHED(ctx);
  }
  ECS_CUDA(ctx, cudaEventRecord(ctx->sev[5], sc));
  ecs_launch_pdl(k_density_in<T>, blocks_for(ctx, L0.n), kB, 0, s0, L0.n, op_density(ctx), L0.dens);
  ECS_LAUNCHED(ctx);
  ECS_CUDA(ctx, cudaEventRecord(ctx->sev[0], s0));
  ECS_CUDA(ctx, cudaStreamWaitEvent(sa, ctx->sev[0], 0));
  for (size_t l = 1; l < mg.lv.size(); l++) {
    MgLevel<T> &F = mg.lv[l - 1], &C = mg.lv[l];
    if ((rc = launch_restrict<T>(ctx, sa, grid_level(ctx, F.nx, F.ny, F.nz), grid_level(ctx, C.nx, C.ny, C.nz), F.dens, C.dens)))
      return rc;
  }
  ECS_CUDA(ctx, cudaEventRecord(ctx->sev[1], sa));
  ECS_CUDA(ctx, cudaStreamWaitEvent(sb, ctx->sev[1], 0));
  for (size_t l = 1; l < mg.lv.size(); l++)
    if ((rc = zline_factor<T>(ctx, mg.lv[l], sb))) return rc;
  ECS_CUDA(ctx, cudaEventRecord(ctx->sev[2], sb));
  if (mg.cinv) {
    MgLevel<T> &C = mg.lv.back();
    const int reg = fully_periodic(ctx) ? 1 : 0;
    if (C.n <= 64)
      ecs_launch_pdl(k_coarse_inverse<T, 64, kInvTpr, false>, 1, 64 * kInvTpr, 0, sa, op_level(ctx, C), C.dens, reg, mg.cinv);
    else
      ecs_launch_pdl(k_coarse_inverse<T, 128, 8, true>, 1, 1024, 0, sa, op_level(ctx, C), C.dens, reg, mg.cinv);
    ECS_LAUNCHED(ctx);
  }
  ECS_CUDA(ctx, cudaEventRecord(ctx->sev[3], sa));
  if ((rc = zline_factor<T>(ctx, L0, s0))) return rc;
  ECS_CUDA(ctx, cudaStreamWaitEvent(s0, ctx->sev[2], 0));
  ECS_CUDA(ctx, cudaStreamWaitEvent(s0, ctx->sev[3], 0));
  ECS_CUDA(ctx, cudaStreamWaitEvent(s0, ctx->sev[5], 0));
  return ECS_OK;
}

// One sweep xn = xo + omega (...); `rhs_done`: its right-hand side is in L.r.
template <typename T>
int sweep(EcsCtx *ctx, MgLevel<T> &L, const T *b, const T *xo, T *xn, bool rhs_done = false) {
  const OpK o = op_level(ctx, L);
  const T *r = b;
  bool row4 = false;
  if constexpr (sizeof(T) == 4) row4 = use_row4(o.g);
  if (rhs_done) {
    r = L.r;
  } else if (xo && row4) {
    if constexpr (sizeof(T) == 4)
      ecs_launch_pdl(k_zline_rhs4, blocks4(o.g), threads4(L.nx), 0, ctx->stream, o, L.dens, b, xo, L.r);
    ECS_LAUNCHED(ctx);
    r = L.r;
  } else if (xo) {
    ecs_launch_pdl(k_zline_rhs<T>, blocks3(o.g), threads3(), 0, ctx->stream, o, L.dens, L.coef, b, xo, L.r);
    ECS_LAUNCHED(ctx);
    r = L.r;
  }
  const int S = seg_len<T>(L.nz);
  const ZCoup<T> zc = z_coupling<T>(o);
  const dim3 grid((unsigned)((L.nx + 31) / 32), (unsigned)L.ny);
  const dim3 block(32, (unsigned)((L.nz + S - 1) / S));
  if (S == 8)
    ecs_launch_pdl(k_zline_seg<T, 8>, grid, block, 0, ctx->stream, o.g, zc, L.dens, zl_of(L), r, xo, xn, kOmega<T>());
  else if (S == 16)
    ecs_launch_pdl(k_zline_seg<T, 16>, grid, block, 0, ctx->stream, o.g, zc, L.dens, zl_of(L), r, xo, xn, kOmega<T>());
  else if (S == 32)
    ecs_launch_pdl(k_zline_seg<T, 32>, grid, block, 0, ctx->stream, o.g, zc, L.dens, zl_of(L), r, xo, xn, kOmega<T>());
  else
    ecs_launch_pdl(k_zline_seg<T, 64>, grid, block, 0, ctx->stream, o.g, zc, L.dens, zl_of(L), r, xo, xn, kOmega<T>());
  ECS_LAUNCHED(ctx);
  return ECS_OK;
}

// Layout of a single-block cycle over levels l.. in shared memory (offsets in
// sc, if given): per level 4 vectors, 11 row coefficients and 4 z-line factor
// arrays, 2 column arrays, and 3 words a cell of neighbour offsets at the end.
// Returns its bytes: at most 164 B a cell and 16 B a column in FP64, for the
// at most 683 cells that such levels have together.
template <typename T>
size_t small_layout(const Multigrid<T> &mg, size_t l, SmallCycle<T> *sc) {
  int off = 0, ni = 0;
  for (size_t q = l; q < mg.lv.size(); q++) {
    const int n = (int)mg.lv[q].n, nc = mg.lv[q].nx * mg.lv[q].ny;
    if (sc) {
      SmallLevel<T> &S = sc->lv[q - l];
      S.sx = off; S.sb = off + n; S.sr = off + 2 * n; S.st = off + 3 * n;
      S.sco = off + 4 * n;
      S.sa = off + 15 * n; S.sc = off + 16 * n; S.sm = off + 17 * n; S.sq = off + 18 * n;
      S.s0 = off + 19 * n; S.sqd = off + 19 * n + nc;
      S.sn = ni;
    }
    off += 19 * n + 2 * nc;
    ni += 3 * n;
  }
  if (sc) sc->ints = off;
  return (size_t)off * sizeof(T) + (size_t)ni * sizeof(unsigned);
}

// Sizes the cluster of the coarsest level's sweeps (no CTAs: two launches a
// sweep), checking that the device can place it.
template <typename T>
int coarse_attrs(EcsCtx *ctx, CoarseShape &cs) {
  auto kernel = coarse_kernel<T>(cs);
  ECS_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClusterSmem));
  ECS_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)cs.ctas);
  cfg.blockDim = dim3((unsigned)cs.threads);
  cfg.dynamicSmemBytes = cs.smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs.ctas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
    cudaGetLastError();
    cs.ctas = 0;
  }
  return ECS_OK;
}
template <typename T>
int launch_coarse_sweeps(EcsCtx *ctx, MgLevel<T> &L, const CoarseShape &cs, const T *b, T *xout) {
  const OpK o = op_level(ctx, L);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)cs.ctas);
  cfg.blockDim = dim3((unsigned)cs.threads);
  cfg.dynamicSmemBytes = cs.smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs.ctas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const ZCoup<T> zc = z_coupling<T>(o);
  const ZlP<T> z = zl_of(L);
  cudaLaunchKernelEx(&cfg, coarse_kernel<T>(cs), o, zc, (const T *)L.dens, z, b, xout, cs.rows, kCoarseSweeps, kOmega<T>());
  ECS_LAUNCHED(ctx);
  return ECS_OK;
}

// x2 = L.x, the coarse correction xc added to L.t, and the right-hand side in L.r.
int launch_prolong_rhs(EcsCtx *ctx, MgLevel<float> &L, const OpK &o, const GridG &gc, const float *b, const float *xc) {
  const bool flat = o.g.nz == 1;
  const auto kernel = flat ? k_prolong_rhs<false, true> : (semi_z(o.g, gc) ? k_prolong_rhs<true, false> : k_prolong_rhs<false, false>);
  const int ty = flat ? PrTile<true>::TY : PrTile<false>::TY, tz = flat ? PrTile<true>::TZ : PrTile<false>::TZ;
  const dim3 g((unsigned)((L.nx + PrTile<true>::TX - 1) / PrTile<true>::TX), (unsigned)((L.ny + ty - 1) / ty),
               (unsigned)((L.nz + tz - 1) / tz));
  ecs_launch_pdl(kernel, g, flat ? PrTile<true>::kThreads : PrTile<false>::kThreads, 0, ctx->stream, o, gc,
                 (const float *)L.dens, b, xc, (const float *)L.t, L.x, L.r);
  ECS_LAUNCHED(ctx);
  return ECS_OK;
}

// One V(1,1) cycle on level l: *x = M(l) b (one of the level's arrays), zero
// initial guess.  Levels of at most kSmallCells cells run as one single-block
// kernel.
template <typename T>
int vcycle(EcsCtx *ctx, size_t l, const T *b, const T **x) {
  Multigrid<T> &mg = mg_of<T>(ctx);
  MgLevel<T> &L = mg.lv[l];
  T *xout = L.x;
  *x = xout;
  int rc;
  if (L.n <= kSmallCells && mg.lv.size() - l <= (size_t)kMaxSmall && small_layout<T>(mg, l, nullptr) <= kSmallSmem) {
    SmallCycle<T> sc;
    sc.nl = (int)(mg.lv.size() - l);
    sc.cinv = mg.cinv;
    const size_t bytes = small_layout<T>(mg, l, &sc);
    for (int q = 0; q < sc.nl; q++) {
      MgLevel<T> &M = mg.lv[l + q];
      SmallLevel<T> &S = sc.lv[q];
      S.o = op_level(ctx, M);
      S.dens = M.dens;
      S.minv = M.zl_minv; S.q = M.zl_q; S.a0g = M.zl_a0g; S.qden = M.zl_qden;
    }
    ecs_launch_pdl(k_vcycle_small<T>, 1, kSmallThreads, bytes, ctx->stream, sc, b, xout, kCoarseSweeps, kOmega<T>());
    ECS_LAUNCHED(ctx);
    return ECS_OK;
  }
  if (l + 1 == mg.lv.size()) {
    if constexpr (sizeof(T) == 4) {
      if (mg.cluster.ctas > 0) return launch_coarse_sweeps<T>(ctx, L, mg.cluster, b, xout);
    }
    if ((rc = sweep<T>(ctx, L, b, nullptr, xout))) return rc;
    for (int s = 0; s < (kCoarseSweeps - 1) / 2; s++) {
      if ((rc = sweep<T>(ctx, L, b, xout, L.t))) return rc;
      if ((rc = sweep<T>(ctx, L, b, L.t, xout))) return rc;
    }
    return ECS_OK;
  }
  MgLevel<T> &C = mg.lv[l + 1];
  const OpK o = op_level(ctx, L);
  if ((rc = sweep<T>(ctx, L, b, nullptr, L.t))) return rc;
  const GridG gc = grid_level(ctx, C.nx, C.ny, C.nz);
  if ((rc = residual_restrict<T>(ctx, L, o, gc, b, C.b))) return rc;
  const T *xc = nullptr;
  if ((rc = vcycle<T>(ctx, l + 1, C.b, &xc))) return rc;
  // FP32: one kernel where the residual and its restriction are (32^3 solve 0.536
  // -> 0.513 ms, 64^3 0.746 -> 0.738, 256^2 in 2-D 0.673 -> 0.656).  FP64 would lose
  // (64^3 1.633 -> 1.642): the rim's sums cost its narrow pipe what the launch does.
  if constexpr (sizeof(T) == 4) {
    if (residual_restrict_fused(o.g)) {
      if ((rc = launch_prolong_rhs(ctx, L, o, gc, b, xc))) return rc;
      *x = L.t;
      return sweep<T>(ctx, L, b, L.x, L.t, true);
    }
  }
  if ((rc = launch_prolong_add<T>(ctx, ctx->stream, o.g, gc, xc, L.t))) return rc;
  return sweep<T>(ctx, L, b, L.t, xout);
}

template <typename T>
T *basis_v(EcsCtx *ctx);
template <>
double *basis_v<double>(EcsCtx *ctx) { return ctx->kv64; }
template <>
float *basis_v<float>(EcsCtx *ctx) { return ctx->kv32; }
template <typename T>
T *basis_z(EcsCtx *ctx);
template <>
double *basis_z<double>(EcsCtx *ctx) { return ctx->kz64; }
template <>
float *basis_z<float>(EcsCtx *ctx) { return ctx->kz32; }
// right-hand side of the FGMRES cycle in precision T
template <typename T>
T *cycle_b(EcsCtx *ctx);
template <>
double *cycle_b<double>(EcsCtx *ctx) { return ctx->r64; }
template <>
float *cycle_b<float>(EcsCtx *ctx) { return ctx->kz32 + (size_t)ctx->krylov_m * ctx->ncell; }
// Kernels before the Arnoldi loop: the cycle's right-hand side (mixed: the
// normalised FP64 residual, r64 or, with first = rhs in a graph's first sweep,
// the right-hand side), its norm, V_0.
template <typename T>
int cycle_pre(EcsCtx *ctx, const double *first, cudaGraphConditionalHandle cond, int use_graph) {
  const size_t n = ctx->ncell;
  KrylovDev *kd = (KrylovDev *)ctx->kdev;
  Multigrid<T> &mg = mg_of<T>(ctx);
  T *b = cycle_b<T>(ctx);
  if constexpr (sizeof(T) == 4) {
    const RefineDev *rd = first ? (const RefineDev *)ctx->rdev : nullptr;
    if (packed4(n))
      ecs_launch_pdl(k_scale_beta<4>, dot_blocks(ctx, n / 4), kB, 0, ctx->stream, n / 4, first, ctx->r64, rd, ctx->dots + 1, b, ctx->red, kd, cond, use_graph);
    else
      ecs_launch_pdl(k_scale_beta<1>, dot_blocks(ctx, n), kB, 0, ctx->stream, n, first, ctx->r64, rd, ctx->dots + 1, b, ctx->red, kd, cond, use_graph);
    ECS_LAUNCHED(ctx);
  } else {
    int rc = launch_reduce<T, kRedBeta>(ctx, n, b, 1.0, nullptr, cond, use_graph);
    if (rc) return rc;
  }
  ecs_launch_pdl(k_cycle_start<T>, blocks_for(ctx, n), kB, 0, ctx->stream, n, b, basis_v<T>(ctx), mg.lv[0].b, kd);
  ECS_LAUNCHED(ctx);
  return ECS_OK;
}

// One Arnoldi step j (j read from the control block).
template <typename T>
int cycle_step(EcsCtx *ctx, cudaGraphConditionalHandle cond, int use_graph) {
  const size_t n = ctx->ncell;
  KrylovDev *kd = (KrylovDev *)ctx->kdev;
  Multigrid<T> &mg = mg_of<T>(ctx);
  MgLevel<T> &L0 = mg.lv[0];
  const OpK o0 = op_level(ctx, L0);
  T *V = basis_v<T>(ctx), *Z = basis_z<T>(ctx);
  int rc;
  // z = M v_j  (vin = L0.b holds v_j)
  const T *zv = nullptr;
  if ((rc = vcycle<T>(ctx, 0, L0.b, &zv))) return rc;
  const double *mean = nullptr;
  if (fully_periodic(ctx)) {  // the operator's null space: project out the mean
    if ((rc = launch_reduce<T, kRedMean>(ctx, n, zv, (double)n, &kd->mean, cond, use_graph))) return rc;
    mean = &kd->mean;
  }
  bool row4 = false;
  if constexpr (sizeof(T) == 4) {
    row4 = use_row4(o0.g);
    if (row4) ecs_launch_pdl(k_apply_dyn4, blocks4(o0.g), threads4(L0.nx), 0, ctx->stream, o0, L0.dens, zv, mean, Z, V, kd);
  }
  if (!row4) ecs_launch_pdl(k_apply_dyn<T>, blocks3(o0.g), threads3(), 0, ctx->stream, o0, L0.dens, L0.coef, zv, mean, Z, V, kd);
  ECS_LAUNCHED(ctx);
  // classical Gram-Schmidt, two passes
  constexpr int W = kPack<T>;
  if (packed4(n)) {
    const unsigned nb = dot_blocks(ctx, n / W);
    ecs_launch_pdl(k_dots1<T, W>, nb, kB, 0, ctx->stream, n, V, kd, ctx->red);
    ECS_LAUNCHED(ctx);
    ecs_launch_pdl(k_orth1_dots2<T, W>, nb, kB, 0, ctx->stream, n, V, kd, ctx->red);
    ECS_LAUNCHED(ctx);
  } else {
    const unsigned nb = dot_blocks(ctx, n);
    ecs_launch_pdl(k_dots1<T, 1>, nb, kB, 0, ctx->stream, n, V, kd, ctx->red);
    ECS_LAUNCHED(ctx);
    ecs_launch_pdl(k_orth1_dots2<T, 1>, nb, kB, 0, ctx->stream, n, V, kd, ctx->red);
    ECS_LAUNCHED(ctx);
  }
  if (packed4(n))
    ecs_launch_pdl(k_orth2_scale<T, W>, blocks_for(ctx, n / W) + 1, kB, 0, ctx->stream, n, V, kd, L0.b, cond, use_graph);
  else
    ecs_launch_pdl(k_orth2_scale<T, 1>, blocks_for(ctx, n) + 1, kB, 0, ctx->stream, n, V, kd, L0.b, cond, use_graph);
  ECS_LAUNCHED(ctx);
  return ECS_OK;
}

// Kernels after the loop: phi += (||r||) sum_q y_q Z_q, mean projection.
template <typename T, int W, bool MEAN>
void launch_finish(EcsCtx *ctx) {
  const size_t n = ctx->ncell;
  ecs_launch_pdl(k_cycle_finish<T, W, MEAN>, dot_blocks(ctx, n / W), kB, 0, ctx->stream, n / W, n, basis_z<T>(ctx),
                 (KrylovDev *)ctx->kdev, sizeof(T) == 4 ? ctx->dots : nullptr, ctx->phi, ctx->red, ctx->dots + 2);
}
template <typename T>
int cycle_post(EcsCtx *ctx) {
  const size_t n = ctx->ncell;
  constexpr int W = kPack<double>;
  const bool mean = fully_periodic(ctx);
  if (packed4(n)) {
    if (mean) launch_finish<T, W, true>(ctx);
    else launch_finish<T, W, false>(ctx);
  } else {
    if (mean) launch_finish<T, 1, true>(ctx);
    else launch_finish<T, 1, false>(ctx);
  }
  ECS_LAUNCHED(ctx);
  if (mean) {
    ecs_launch_pdl(k_sub_value<double>, blocks_for(ctx, n), kB, 0, ctx->stream, n, ctx->phi, ctx->dots + 2);
    ECS_LAUNCHED(ctx);
  }
  return ECS_OK;
}

// One FGMRES cycle on r64 with tolerance tol (relative to its norm) and at
// most maxit steps, launched from the host step by step (the host reads the
// stop flag after each step), its correction added to phi; the control block
// ends up in ctx->kdev_host.
template <typename T>
int fgmres_cycle(EcsCtx *ctx, double tol, int maxit) {
  KrylovDev *kd = (KrylovDev *)ctx->kdev;
  KrylovDev *ctl = (KrylovDev *)ctx->kctl_host;
  ctl->tol_rel = tol;
  ctl->maxit = std::min(std::min(ctx->krylov_m, kKrylovMax), std::max(maxit, 1));
  ECS_CUDA(ctx, cudaMemcpyAsync(kd, ctl, offsetof(KrylovDev, j), cudaMemcpyHostToDevice, ctx->stream));
  int rc;
  cudaGraphConditionalHandle none = 0;
  if ((rc = cycle_pre<T>(ctx, nullptr, none, 0))) return rc;
  KrylovDev *hk = (KrylovDev *)ctx->kdev_host;
  for (int s = 0; s < kKrylovMax; s++) {
    ECS_CUDA(ctx, cudaMemcpyAsync(&hk->done, &kd->done, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    ECS_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (hk->done) break;
    if ((rc = cycle_step<T>(ctx, none, 0))) return rc;
  }
  return cycle_post<T>(ctx);
}

// ||v||_2 of an FP64 vector into out2[0], its inverse into out2[1], on the device.
int norm64_dev(EcsCtx *ctx, const double *v, double *out2) {
  return launch_reduce<double, kRedNorm>(ctx, ctx->ncell, v, 1.0, out2, 0, 0);
}

// ---- the whole solve on the device ------------------------------------------
// Mixed-precision residual: r64 = b64 - A64(n64) x64.
// r = b - A x in FP64 from the stored coefficients (the same products and
// sum as computing them in place).
__global__ void k_residual64(OpK o, const double *__restrict__ coef, const double *__restrict__ x,
                             const double *__restrict__ b, double *__restrict__ r) {
  ECS_PDL_ENTRY();
  int i, j, k;
  if (!at3(o.g.nx, o.g.ny, i, j, k)) return;
  const Nbr q = nbr_of(o.g, i, j, k);
  double xe[11];
  row_x(x, q, xe);
  double s = 0.0;
#pragma unroll
  for (int e = 0; e < 11; e++) s += __ldg(&coef[(size_t)e * o.g.n + q.c]) * xe[e];
  r[q.c] = b[q.c] - s;
}

template <typename T>
void free_mg(Multigrid<T> &mg) {
  for (size_t l = 0; l < mg.lv.size(); l++) {
    MgLevel<T> &L = mg.lv[l];
    if (l > 0 && L.coef) cudaFree(L.coef);  // the finest level's are the context's
    T *arr[] = {L.dens, L.x, L.b, L.r, L.t, L.zl_a, L.zl_cp, L.zl_minv, L.zl_q, L.zl_fb, L.zl_bb, L.zl_a0g, L.zl_qden};
    for (T *a : arr)
      if (a) cudaFree(a);
  }
  mg.lv.clear();
  if (mg.cinv) cudaFree(mg.cinv);
  mg.cinv = nullptr;
  mg.built = false;
}

void free_graph(SolverGraph &sg) {
  if (sg.exec) cudaGraphExecDestroy(sg.exec);
  if (sg.graph) cudaGraphDestroy(sg.graph);
  sg = SolverGraph();
}

// ---- graph construction ----------------------------------------------------------
// Conditional node appended to the graph being captured on stream s (after
// its current dependencies); the node's body graph is returned, to be
// captured on another stream.
int capture_conditional(EcsCtx *ctx, cudaStream_t s, cudaGraphConditionalHandle h, cudaGraphConditionalNodeType type,
                        cudaGraph_t *body) {
  cudaStreamCaptureStatus cs;
  cudaGraph_t g = nullptr;
  const cudaGraphNode_t *deps = nullptr;
  const cudaGraphEdgeData *edges = nullptr;
  size_t nd = 0;
  ECS_CUDA(ctx, cudaStreamGetCaptureInfo(s, &cs, nullptr, &g, &deps, &edges, &nd));
  // zero-initialised storage (the parameter union has no default constructor)
  alignas(cudaGraphNodeParams) unsigned char cp_store[sizeof(cudaGraphNodeParams)];
  memset(cp_store, 0, sizeof cp_store);
  cudaGraphNodeParams *cp = reinterpret_cast<cudaGraphNodeParams *>(cp_store);
  cp->type = cudaGraphNodeTypeConditional;
  cp->conditional.handle = h;
  cp->conditional.type = type;
  cp->conditional.size = 1;
  cudaGraphNode_t node;
  ECS_CUDA(ctx, cudaGraphAddNode(&node, g, deps, edges, nd, cp));
  ECS_CUDA(ctx, cudaStreamUpdateCaptureDependencies(s, &node, nullptr, 1, cudaStreamSetCaptureDependencies));
  *body = cp->conditional.phGraph_out[0];
  return ECS_OK;
}
// The graph being captured on stream s.
int capture_graph(EcsCtx *ctx, cudaStream_t s, cudaGraph_t *g) {
  cudaStreamCaptureStatus cs;
  ECS_CUDA(ctx, cudaStreamGetCaptureInfo(s, &cs, nullptr, g, nullptr, nullptr, nullptr));
  return ECS_OK;
}

template <typename T>
RefineArgs refine_args(EcsCtx *ctx, double rtol, int max_it, int decide, int after) {
  return {(RefineDev *)ctx->rdev, rtol, sizeof(T) == 4 ? 2e-6 : 0.0, max_it, decide, after};
}

// Residual of the current phi, its norm and the check that sets the sweep
// loop's condition h (on ctx->stream).
template <typename T>
int refine_check(EcsCtx *ctx, double rtol, int max_it, int after, cudaGraphConditionalHandle h) {
  const EcsParams &p = ctx->p;
  const OpK o64 = make_op(p, p.Nx, p.Ny, p.Nz, p.dx, p.dy, p.dz);
  ecs_launch_pdl(k_residual64, blocks3(o64.g), threads3(), 0, ctx->stream, o64, (const double *)ctx->coef64, ctx->phi, ctx->rhs, ctx->r64);
  ECS_LAUNCHED(ctx);
  return launch_reduce<double, kRedCheck>(ctx, ctx->ncell, ctx->r64, 1.0, ctx->dots, h, 1,
                                          refine_args<T>(ctx, rtol, max_it, 1, after));
}

// The correction of one sweep: the FGMRES cycle (the Arnoldi loop as a WHILE
// node captured on capture stream `lvl`), phi update, mean projection.
template <typename T>
int refine_correct(EcsCtx *ctx, int lvl, int warm) {
  int rc;
  cudaGraph_t g = nullptr, body = nullptr;
  if ((rc = capture_graph(ctx, ctx->stream, &g))) return rc;
  cudaGraphConditionalHandle hw;
  ECS_CUDA(ctx, cudaGraphConditionalHandleCreate(&hw, g, 0, 0));
  if ((rc = cycle_pre<T>(ctx, warm ? nullptr : ctx->rhs, hw, 1))) return rc;
  if ((rc = capture_conditional(ctx, ctx->stream, hw, cudaGraphCondTypeWhile, &body))) return rc;
  cudaStream_t outer = ctx->stream;
  ctx->stream = ctx->capst[lvl];
  ECS_CUDA(ctx, cudaStreamBeginCaptureToGraph(ctx->stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
  const int64_t l0 = ctx->launches;
  rc = cycle_step<T>(ctx, hw, 1);
  ctx->sgraph.k_step = ctx->launches - l0;
  cudaError_t ce = cudaStreamEndCapture(ctx->stream, &body);
  ctx->stream = outer;
  if (rc) return rc;
  ECS_CUDA(ctx, ce);
  return cycle_post<T>(ctx);
}

// The nodes of one solve, appended to the graph being captured on
// ctx->stream:
//   [phi = 0, r = b | r = b - A phi]  ||r||, init, check
//   WHILE( scale, beta  cycle(WHILE Arnoldi)  phi += e  residual  norm, check )
// The checks set the sweep loop's condition; everything stays on the device.
// The kernel counts of the head, a sweep and an Arnoldi step go to sgraph.
template <typename T>
int capture_solve(EcsCtx *ctx, double rtol, int max_it, int warm) {
  SolverGraph &sg = ctx->sgraph;
  const size_t n = ctx->ncell;
  const int64_t launches0 = ctx->launches;
  int rc;
  cudaError_t ce;
  cudaGraph_t top = nullptr;
  if ((rc = capture_graph(ctx, ctx->stream, &top))) return rc;
  const bool identity = identity_lhs(ctx);
  cudaGraphConditionalHandle hs = 0;
  if (!identity) ECS_CUDA(ctx, cudaGraphConditionalHandleCreate(&hs, top, 0, cudaGraphCondAssignDefault));
  // ||b||; from phi = 0 the residual is b, and the same norm decides
  rc = launch_reduce<double, kRedInit>(ctx, n, ctx->rhs, 1.0, ctx->dots, hs, 1,
                                       refine_args<T>(ctx, rtol, max_it, !warm && !identity, 0));
  if (rc) return rc;
  if (identity) {  // -lhs identity (ComputeIdentityLHS, src/lhs.c:11-23): phi = b exactly
    ECS_CUDA(ctx, cudaMemcpyAsync(ctx->phi, ctx->rhs, n * sizeof(double), cudaMemcpyDeviceToDevice, ctx->stream));
    sg.k_head = ctx->launches - launches0;
    sg.k_sweep = sg.k_step = 0;
    return ECS_OK;
  }
  if (!warm) {
    ECS_CUDA(ctx, cudaMemsetAsync(ctx->phi, 0, n * sizeof(double), ctx->stream));
    if (sizeof(T) == 8)  // the mixed cycle reads b itself in its first sweep
      ECS_CUDA(ctx, cudaMemcpyAsync(ctx->r64, ctx->rhs, n * sizeof(double), cudaMemcpyDeviceToDevice, ctx->stream));
  } else {
    rc = refine_check<T>(ctx, rtol, max_it, 0, hs);
  }
  if (rc) return rc;
  sg.k_head = ctx->launches - launches0;
  cudaGraph_t body = nullptr;
  if ((rc = capture_conditional(ctx, ctx->stream, hs, cudaGraphCondTypeWhile, &body))) return rc;
  cudaStream_t outer = ctx->stream;
  ctx->stream = ctx->capst[1];
  ce = cudaStreamBeginCaptureToGraph(ctx->stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
  if (ce != cudaSuccess) {
    ctx->stream = outer;
    return ecs_cuda_check(ctx, ce, "sweep capture");
  }
  const int64_t l1 = ctx->launches;
  rc = refine_correct<T>(ctx, 2, warm);
  if (!rc) rc = refine_check<T>(ctx, rtol, max_it, 1, hs);
  sg.k_sweep = ctx->launches - l1 - sg.k_step;
  ce = cudaStreamEndCapture(ctx->stream, &body);
  ctx->stream = outer;
  if (rc) return rc;
  ECS_CUDA(ctx, ce);
  return ECS_OK;
}

int ensure_capture_streams(EcsCtx *ctx) {
  for (auto &c : ctx->capst)
    if (!c) ECS_CUDA(ctx, cudaStreamCreateWithFlags(&c, cudaStreamNonBlocking));
  return ECS_OK;
}

// The right-hand side (FP64-bound) on sst[3] beside the operator set-up
// (latency-bound) on the context's stream and sst[0..2]; both need only the
// moments, and the context's stream waits for both.
template <typename T>
int rhs_beside_setup(EcsCtx *ctx) {
  int rc = ensure_setup_streams(ctx);
  if (rc) return rc;
  if (identity_lhs(ctx)) return ecs_grid_rhs(ctx);
  cudaStream_t s0 = ctx->stream;
  ECS_CUDA(ctx, cudaEventRecord(ctx->sev[6], s0));
  ECS_CUDA(ctx, cudaStreamWaitEvent(ctx->sst[3], ctx->sev[6], 0));
  ctx->stream = ctx->sst[3];
  rc = ecs_grid_rhs(ctx);
  ctx->stream = s0;
  if (rc) return rc;
  ECS_CUDA(ctx, cudaEventRecord(ctx->sev[7], ctx->sst[3]));
  if ((rc = mg_setup<T>(ctx))) return rc;
  ECS_CUDA(ctx, cudaStreamWaitEvent(s0, ctx->sev[7], 0));
  return ECS_OK;
}

// One solve as one graph (see capture_solve), built for (rtol, max_it, warm).
template <typename T>
int build_solve_graph(EcsCtx *ctx, double rtol, int max_it, int warm, int setup) {
  SolverGraph &sg = ctx->sgraph;
  if (sg.exec && sg.rtol == rtol && sg.max_it == max_it && sg.warm == warm && sg.setup == setup) return ECS_OK;
  free_graph(sg);
  int rc = ensure_capture_streams(ctx);
  if (rc) return rc;
  if (setup) {  // allocations happen before the capture
    if ((rc = ecs_solver_alloc(ctx))) return rc;
    if (!identity_lhs(ctx) && (rc = mg_alloc<T>(ctx))) return rc;
    if ((rc = ensure_setup_streams(ctx))) return rc;
  }
  const int64_t launches0 = ctx->launches;
  cudaStream_t user = ctx->stream;
  ctx->stream = ctx->capst[0];
  cudaGraph_t g = nullptr;
  cudaError_t ce = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal);
  if (ce != cudaSuccess) {
    ctx->stream = user;
    return ecs_cuda_check(ctx, ce, "solve graph capture");
  }
  rc = ECS_OK;
  sg.k_pre = 0;
  if (setup) {
    rc = rhs_beside_setup<T>(ctx);
    sg.k_pre = ctx->launches - launches0;
  }
  if (!rc) rc = capture_solve<T>(ctx, rtol, max_it, warm);
  ce = cudaStreamEndCapture(ctx->stream, &g);
  ctx->stream = user;
  ctx->launches = launches0;
  if (rc) {
    if (g) cudaGraphDestroy(g);
    return rc;
  }
  ECS_CUDA(ctx, ce);
  sg.graph = g;
  ECS_CUDA(ctx, cudaGraphInstantiate(&sg.exec, g, 0));
  sg.rtol = rtol;
  sg.max_it = max_it;
  sg.warm = warm;
  sg.setup = setup;
  return ECS_OK;
}

// Launch the solve graph (asynchronous).
int solve_graph_launch(EcsCtx *ctx, double rtol, int max_it, int warm, int setup) {
  int rc = ctx->prec == ECS_PREC_FP64 ? build_solve_graph<double>(ctx, rtol, max_it, warm, setup)
                                      : build_solve_graph<float>(ctx, rtol, max_it, warm, setup);
  if (rc) return rc;
  ECS_CUDA(ctx, cudaGraphLaunch(ctx->sgraph.exec, ctx->stream));
  return ECS_OK;
}

// ---- stand-alone solve request ----------------------------------------------
// Fluxes of a loaded density (src/file-io.c:51-59: VecAXPY into a zeroed
// vector, so G_d = 0 + flux_scale_d * n), into the SoA moment planes 1..3.
__global__ void k_density_flux(size_t n, double f0, double f1, double f2, double *__restrict__ mom) {
  ECS_PDL_ENTRY();
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
    const double d = mom[c];
    mom[n + c] = __dadd_rn(0.0, __dmul_rn(f0, d));
    mom[2 * n + c] = __dadd_rn(0.0, __dmul_rn(f1, d));
    mom[3 * n + c] = __dadd_rn(0.0, __dmul_rn(f2, d));
  }
}

// The node that the last call captured on stream s.
int last_captured(EcsCtx *ctx, cudaStream_t s, cudaGraphNode_t *node) {
  cudaStreamCaptureStatus cs;
  const cudaGraphNode_t *deps = nullptr;
  size_t nd = 0;
  ECS_CUDA(ctx, cudaStreamGetCaptureInfo(s, &cs, nullptr, nullptr, &deps, nullptr, &nd));
  if (nd != 1) return ecs_fail(ctx, ECS_ERR_CUDA, "capture: expected one tail node, found %zu", nd);
  *node = deps[0];
  return ECS_OK;
}

void free_request_graph(RequestGraph &rg) {
  if (rg.exec) cudaGraphExecDestroy(rg.exec);
  if (rg.graph) cudaGraphDestroy(rg.graph);
  rg.exec = nullptr;
  rg.graph = nullptr;
  rg.in_node = rg.out_node = nullptr;
}

// density -> moments -> RHS -> operator set-up -> solve -> phi, as one graph.
template <typename T>
int build_request_graph(EcsCtx *ctx, const double fs[3], double rtol, int max_it) {
  RequestGraph &rg = ctx->rgraph;
  if (rg.exec && rg.rtol == rtol && rg.max_it == max_it && rg.flux_scale[0] == fs[0] && rg.flux_scale[1] == fs[1] &&
      rg.flux_scale[2] == fs[2])
    return ECS_OK;
  free_request_graph(rg);
  const size_t n = ctx->ncell, bytes = n * sizeof(double);
  int rc;
  if ((rc = ecs_pinned_alloc(ctx, rg.h_in, bytes)) || (rc = ecs_pinned_alloc(ctx, rg.h_out, bytes))) return rc;
  // allocations and one-time attributes outside the capture
  if ((rc = ecs_solver_alloc(ctx))) return rc;
  if (!identity_lhs(ctx) && (rc = mg_alloc<T>(ctx))) return rc;
  if ((rc = ensure_capture_streams(ctx))) return rc;
  if ((rc = ensure_setup_streams(ctx))) return rc;  // the set-up forks onto them inside the capture
  const int64_t launches0 = ctx->launches;
  cudaStream_t user = ctx->stream;
  ctx->stream = ctx->capst[0];
  cudaGraph_t g = nullptr;
  cudaError_t ce = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal);
  if (ce != cudaSuccess) {
    ctx->stream = user;
    return ecs_cuda_check(ctx, ce, "request graph capture");
  }
  do {
    if ((ce = cudaMemcpyAsync(ctx->mom, rg.h_in, bytes, cudaMemcpyHostToDevice, ctx->stream)) != cudaSuccess) {
      rc = ecs_cuda_check(ctx, ce, "density copy");
      break;
    }
    if ((rc = last_captured(ctx, ctx->stream, &rg.in_node))) break;
    ecs_launch_pdl(k_density_flux, blocks_for(ctx, n), kB, 0, ctx->stream, n, fs[0], fs[1], fs[2], ctx->mom);
    if ((ce = cudaGetLastError()) != cudaSuccess) {
      rc = ecs_cuda_check(ctx, ce, "kernel launch");
      break;
    }
    ctx->launches++;
    if ((rc = rhs_beside_setup<T>(ctx))) break;
    rg.k_pre = ctx->launches - launches0;
    if ((rc = capture_solve<T>(ctx, rtol, max_it, 0))) break;
    if ((ce = cudaMemcpyAsync(rg.h_out, ctx->phi, bytes, cudaMemcpyDeviceToHost, ctx->stream)) != cudaSuccess) {
      rc = ecs_cuda_check(ctx, ce, "potential copy");
      break;
    }
    if ((rc = last_captured(ctx, ctx->stream, &rg.out_node))) break;
    if ((ce = cudaMemcpyAsync(ctx->rdev_host, ctx->rdev, sizeof(RefineDev), cudaMemcpyDeviceToHost, ctx->stream)) !=
        cudaSuccess) {
      rc = ecs_cuda_check(ctx, ce, "status copy");
      break;
    }
  } while (0);
  ce = cudaStreamEndCapture(ctx->stream, &g);
  ctx->stream = user;
  ctx->launches = launches0;
  if (rc) {
    if (g) cudaGraphDestroy(g);
    rg.in_node = rg.out_node = nullptr;
    return rc;
  }
  ECS_CUDA(ctx, ce);
  rg.graph = g;
  ECS_CUDA(ctx, cudaGraphInstantiate(&rg.exec, g, 0));
  rg.rtol = rtol;
  rg.max_it = max_it;
  for (int d = 0; d < 3; d++) rg.flux_scale[d] = fs[d];
  return ECS_OK;
}

// Page-locked (or registered) host memory: the copy engines read and write it
// directly.
bool host_pinned(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost;
}

}  // namespace

// ============================================================================
// entry points used by ecs_api.cu and ecs_grid.cu
// ============================================================================
void ecs_mg_bytes(const EcsParams &p, int precision, DeviceBytes &b) {
  const std::vector<MgDims> lv = mg_dims(p);
  if (precision == ECS_PREC_FP64) mg_bytes<double>(lv, b);
  else mg_bytes<float>(lv, b);
}

// Each buffer that is not there yet (after a failure, the rest of them).
int ecs_solver_alloc(EcsCtx *ctx) {
  const size_t n = ctx->ncell, m = (size_t)ctx->krylov_m;
  int rc;
  ctx->nred = kSlots * 4096;
  if ((rc = ecs_dev_alloc(ctx, ctx->red, (size_t)ctx->nred * sizeof(double))) ||
      (rc = ecs_dev_alloc(ctx, ctx->dots, (m + 2) * sizeof(double))) ||
      (rc = ecs_pinned_alloc(ctx, ctx->h_dots, (m + 2) * sizeof(double))) ||
      (rc = ecs_dev_alloc(ctx, ctx->r64, n * sizeof(double))))
    return rc;
  if (!identity_lhs(ctx) && (rc = ecs_dev_alloc(ctx, ctx->coef64, 11 * n * sizeof(double)))) return rc;
  // zeroed on the context's stream: the default stream is not ordered with
  // it, and behind a host step's transfers its memset ran during the first solve
  if (!ctx->kdev) {
    if ((rc = ecs_dev_alloc(ctx, ctx->kdev, sizeof(KrylovDev)))) return rc;
    ECS_CUDA(ctx, cudaMemsetAsync(ctx->kdev, 0, sizeof(KrylovDev), ctx->stream));
  }
  if (!ctx->rdev) {
    if ((rc = ecs_dev_alloc(ctx, ctx->rdev, sizeof(RefineDev)))) return rc;
    ECS_CUDA(ctx, cudaMemsetAsync(ctx->rdev, 0, sizeof(RefineDev), ctx->stream));
  }
  struct {
    void *&p;
    size_t bytes;
  } host[] = {{ctx->kdev_host, sizeof(KrylovDev)}, {ctx->kctl_host, sizeof(KrylovDev)}, {ctx->rdev_host, sizeof(RefineDev)}};
  for (auto &h : host)
    if (!h.p) {
      if ((rc = ecs_pinned_alloc(ctx, h.p, h.bytes))) return rc;
      memset(h.p, 0, h.bytes);
    }
  if (ctx->prec == ECS_PREC_FP64) {
    if ((rc = ecs_dev_alloc(ctx, ctx->kv64, (m + 1) * n * sizeof(double))) ||
        (rc = ecs_dev_alloc(ctx, ctx->kz64, m * n * sizeof(double))))
      return rc;
  } else {
    // V, Z and the normalised residual
    if ((rc = ecs_dev_alloc(ctx, ctx->kv32, (m + 1) * n * sizeof(float))) ||
        (rc = ecs_dev_alloc(ctx, ctx->kz32, (m + 1) * n * sizeof(float))))
      return rc;
  }
  return ECS_OK;
}

int ecs_solver_setup(EcsCtx *ctx) {
  int rc = ecs_solver_alloc(ctx);
  if (rc) return rc;
  if (!identity_lhs(ctx)) rc = ctx->prec == ECS_PREC_FP64 ? mg_setup<double>(ctx) : mg_setup<float>(ctx);
  if (rc) return rc;
  ctx->lhs_ready = true;
  return ECS_OK;
}

// Iterative refinement around FGMRES cycles.  Per refinement the host waits
// once, for the FP64 residual norm and the finished cycle's control block.
int ecs_solver_run(EcsCtx *ctx, double rtol, int max_it, int warm, EcsSolveStats *st, int setup,
                   EcsHostHook between, void *arg) {
  const bool graphs = ctx->use_graphs || identity_lhs(ctx);
  if (between && !graphs) {  // the host-driven loop waits on the device from its start
    const int rc_h = between(ctx, arg);
    if (rc_h) return rc_h;
    between = nullptr;
  }
  if (setup && !graphs) {  // the host-driven loop: RHS and set-up launched one by one
    int rc0 = ecs_grid_rhs(ctx);
    if (!rc0) rc0 = ecs_solver_setup(ctx);
    if (rc0) return rc0;
    setup = 0;
  }
  if (!setup && !ctx->lhs_ready) return ecs_fail(ctx, ECS_ERR_STATE, "solve called before lhs");
  const size_t n = ctx->ncell;
  const EcsParams &p = ctx->p;
  const OpK o64 = make_op(p, p.Nx, p.Ny, p.Nz, p.dx, p.dy, p.dz);
  KrylovDev *hk = (KrylovDev *)ctx->kdev_host;
  if (!ctx->ev_solve[0]) {
    ECS_CUDA(ctx, cudaEventCreate(&ctx->ev_solve[0]));
    ECS_CUDA(ctx, cudaEventCreate(&ctx->ev_solve[1]));
  }
  ECS_CUDA(ctx, cudaEventRecord(ctx->ev_solve[0], ctx->stream));
  int rc;
  if (graphs) {  // the whole solve as one graph launch, one wait
    if ((rc = solve_graph_launch(ctx, rtol, max_it, warm, setup))) return rc;
    if (setup) ctx->lhs_ready = true;  // the graph sets the operator up before it solves
    RefineDev *hr = (RefineDev *)ctx->rdev_host;
    ECS_CUDA(ctx, cudaMemcpyAsync(hr, ctx->rdev, sizeof(RefineDev), cudaMemcpyDeviceToHost, ctx->stream));
    ECS_CUDA(ctx, cudaEventRecord(ctx->ev_solve[1], ctx->stream));
    const int rc_h = between ? between(ctx, arg) : ECS_OK;
    ECS_CUDA(ctx, cudaEventSynchronize(ctx->ev_solve[1]));
    if (rc_h) return rc_h;
    const SolverGraph &sg = ctx->sgraph;
    ctx->launches += sg.k_pre + sg.k_head + hr->sweeps * sg.k_sweep + (int64_t)hr->its * sg.k_step;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ctx->ev_solve[0], ctx->ev_solve[1]);
    if (st) {
      st->iterations = hr->its;
      st->refinements = hr->sweeps;
      st->relres = hr->rel;
      st->seconds = ms * 1e-3;
    }
    if (hr->nonfinite) return ecs_fail(ctx, ECS_ERR_NONFINITE, "non-finite residual in solve");
    if (hr->bnorm > 0.0 && hr->rel > rtol)
      return ecs_fail(ctx, ECS_ERR_NOT_CONVERGED, "solve stopped at relres %.3e > %.3e after %d iterations", hr->rel,
                      rtol, hr->its);
    return ECS_OK;
  }
  if (!warm) ECS_CUDA(ctx, cudaMemsetAsync(ctx->phi, 0, n * sizeof(double), ctx->stream));
  // ||b|| -> dots[0], 1/||b|| -> dots[1]
  if ((rc = norm64_dev(ctx, ctx->rhs, ctx->dots))) return rc;
  ECS_CUDA(ctx, cudaMemcpyAsync(ctx->h_dots, ctx->dots, 2 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  ECS_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  const double bnorm = ctx->h_dots[0];
  int its = 0, sweeps = 0;
  double rel = 0.0;
  bool cycle_pending = false;
  bool zero_guess = !warm;
  if (bnorm > 0.0) {
    for (;;) {
      if (zero_guess) {  // phi = 0: the residual is b, its norm (dots[0..1]) is known
        ECS_CUDA(ctx, cudaMemcpyAsync(ctx->r64, ctx->rhs, n * sizeof(double), cudaMemcpyDeviceToDevice, ctx->stream));
        zero_guess = false;
      } else {
        ecs_launch_pdl(k_residual64, blocks3(o64.g), threads3(), 0, ctx->stream, o64, (const double *)ctx->coef64, ctx->phi, ctx->rhs, ctx->r64);
        ECS_LAUNCHED(ctx);
        if ((rc = norm64_dev(ctx, ctx->r64, ctx->dots))) return rc;
        ECS_CUDA(ctx, cudaMemcpyAsync(ctx->h_dots, ctx->dots, 2 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
        if (cycle_pending)
          ECS_CUDA(ctx, cudaMemcpyAsync(hk, ctx->kdev, sizeof(KrylovDev), cudaMemcpyDeviceToHost, ctx->stream));
        ECS_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
      }
      if (cycle_pending) {
        its += hk->nits;
        sweeps++;
        cycle_pending = false;
        if (hk->nits == 0) {
          rel = ctx->h_dots[0] / bnorm;
          break;
        }
      }
      const double rn = ctx->h_dots[0];
      rel = rn / bnorm;
      if (!isfinite(rel)) return ecs_fail(ctx, ECS_ERR_NONFINITE, "non-finite residual in solve");
      if (rel <= rtol || its >= max_it) break;
      const double tol_cycle = std::max(0.5 * rtol / rel, 1e-14);
      if (ctx->prec == ECS_PREC_FP64) {
        // the cycle solves A e = r64 directly (beta = ||r64||)
        rc = fgmres_cycle<double>(ctx, tol_cycle, max_it - its);
      } else {
        rc = fgmres_cycle<float>(ctx, std::max(tol_cycle, 2e-6), max_it - its);
      }
      if (rc) return rc;
      cycle_pending = true;
    }
  }
  ECS_CUDA(ctx, cudaEventRecord(ctx->ev_solve[1], ctx->stream));
  ECS_CUDA(ctx, cudaEventSynchronize(ctx->ev_solve[1]));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, ctx->ev_solve[0], ctx->ev_solve[1]);
  if (st) {
    st->iterations = its;
    st->refinements = sweeps;
    st->relres = rel;
    st->seconds = ms * 1e-3;
  }
  if (bnorm > 0.0 && rel > rtol)
    return ecs_fail(ctx, ECS_ERR_NOT_CONVERGED, "solve stopped at relres %.3e > %.3e after %d iterations", rel, rtol, its);
  return ECS_OK;
}

int ecs_operator_apply64(EcsCtx *ctx, const double *x, double *y) {
  const EcsParams &p = ctx->p;
  const OpK o64 = make_op(p, p.Nx, p.Ny, p.Nz, p.dx, p.dy, p.dz);
  if (identity_lhs(ctx)) {
    ECS_CUDA(ctx, cudaMemcpyAsync(y, x, ctx->ncell * sizeof(double), cudaMemcpyDeviceToDevice, ctx->stream));
    return ECS_OK;
  }
  ecs_launch_pdl(k_apply<double>, blocks3(o64.g), threads3(), 0, ctx->stream, o64, op_density(ctx), nullptr, x, nullptr, y, 0);
  ECS_LAUNCHED(ctx);
  return ECS_OK;
}

int ecs_solver_free(EcsCtx *ctx) {
  free_graph(ctx->sgraph);
  free_request_graph(ctx->rgraph);
  if (ctx->rgraph.h_in) cudaFreeHost(ctx->rgraph.h_in);
  if (ctx->rgraph.h_out) cudaFreeHost(ctx->rgraph.h_out);
  for (auto &c : ctx->capst)
    if (c) cudaStreamDestroy(c);
  for (auto &c : ctx->sst)
    if (c) cudaStreamDestroy(c);
  for (auto &e : ctx->sev)
    if (e) cudaEventDestroy(e);
  free_mg(ctx->mg64);
  free_mg(ctx->mg32);
  void *ptrs[] = {ctx->kv64, ctx->kz64, ctx->kv32, ctx->kz32, ctx->r64, ctx->coef64, ctx->dots, ctx->red,
                  ctx->kdev, ctx->rdev};
  for (void *q : ptrs)
    if (q) cudaFree(q);
  if (ctx->h_dots) cudaFreeHost(ctx->h_dots);
  if (ctx->kdev_host) cudaFreeHost(ctx->kdev_host);
  if (ctx->kctl_host) cudaFreeHost(ctx->kctl_host);
  if (ctx->rdev_host) cudaFreeHost(ctx->rdev_host);
  for (auto &e : ctx->ev_solve)
    if (e) cudaEventDestroy(e);
  return ECS_OK;
}

// ---- stand-alone solve requests ---------------------------------------------
int ecs_request_launch(EcsCtx *ctx, const double *density, double *phi, const double flux_scale[3], double rtol,
                       int max_it) {
  // before the graph is built: it keeps the kernels that this picks, and a
  // request's density is no deposit's
  ctx->mom_quanta = false;
  int rc = ctx->prec == ECS_PREC_FP64 ? build_request_graph<double>(ctx, flux_scale, rtol, max_it)
                                      : build_request_graph<float>(ctx, flux_scale, rtol, max_it);
  if (rc) return rc;
  RequestGraph &rg = ctx->rgraph;
  const size_t bytes = ctx->ncell * sizeof(double);
  const double *src = density;
  if (!host_pinned(density)) {
    memcpy(rg.h_in, density, bytes);
    src = rg.h_in;
  }
  rg.staged_out = !host_pinned(phi);
  rg.dst = phi;
  double *dst = rg.staged_out ? rg.h_out : phi;
  ECS_CUDA(ctx, cudaGraphExecMemcpyNodeSetParams1D(rg.exec, rg.in_node, ctx->mom, src, bytes, cudaMemcpyHostToDevice));
  ECS_CUDA(ctx, cudaGraphExecMemcpyNodeSetParams1D(rg.exec, rg.out_node, dst, ctx->phi, bytes, cudaMemcpyDeviceToHost));
  if (!ctx->ev_solve[0]) {
    ECS_CUDA(ctx, cudaEventCreate(&ctx->ev_solve[0]));
    ECS_CUDA(ctx, cudaEventCreate(&ctx->ev_solve[1]));
  }
  ECS_CUDA(ctx, cudaEventRecord(ctx->ev_solve[0], ctx->stream));
  ECS_CUDA(ctx, cudaGraphLaunch(rg.exec, ctx->stream));
  ECS_CUDA(ctx, cudaEventRecord(ctx->ev_solve[1], ctx->stream));
  ctx->moments_ready = true;
  ctx->lhs_ready = true;
  ctx->eext_ready = false;
  return ECS_OK;
}

int ecs_request_finish(EcsCtx *ctx, EcsSolveStats *st) {
  RequestGraph &rg = ctx->rgraph;
  const RefineDev *hr = (const RefineDev *)ctx->rdev_host;
  if (rg.staged_out) memcpy(rg.dst, rg.h_out, ctx->ncell * sizeof(double));
  const SolverGraph &sg = ctx->sgraph;
  ctx->launches += rg.k_pre + sg.k_head + hr->sweeps * sg.k_sweep + (int64_t)hr->its * sg.k_step;
  float ms = 0.f;
  cudaEventElapsedTime(&ms, ctx->ev_solve[0], ctx->ev_solve[1]);
  if (st) {
    st->iterations = hr->its;
    st->refinements = hr->sweeps;
    st->relres = hr->rel;
    st->seconds = ms * 1e-3;
  }
  if (hr->nonfinite) return ecs_fail(ctx, ECS_ERR_NONFINITE, "non-finite residual in solve");
  if (hr->bnorm > 0.0 && hr->rel > rg.rtol)
    return ecs_fail(ctx, ECS_ERR_NOT_CONVERGED, "solve stopped at relres %.3e > %.3e after %d iterations", hr->rel,
                    rg.rtol, hr->its);
  return ECS_OK;
}
