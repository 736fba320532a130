// Structured-grid helpers shared by the grid and solver translation units:
// grid shape, ghost-aware loads, 3-D launch indexing (no integer division)
// and the 11-coefficient operator row of src/lhs.c:366-423.
#pragma once

#include <math.h>

#include "ecs_internal.cuh"

// FP64 arithmetic with every operation separately rounded (no contraction),
// for kernels that must match the reference's FP64 results operand for
// operand.
struct rd {
  double v;
};
__device__ __forceinline__ rd operator+(rd a, rd b) { return {__dadd_rn(a.v, b.v)}; }
__device__ __forceinline__ rd operator-(rd a, rd b) { return {__dsub_rn(a.v, b.v)}; }
__device__ __forceinline__ rd operator*(rd a, rd b) { return {__dmul_rn(a.v, b.v)}; }

struct GridG {
  int nx, ny, nz;
  int bc[3];  // 0 periodic, else ghosted (value 0 outside)
  size_t n;   // nx*ny*nz (at most 2^30)
};

// Value at (k,j,i) with the reference's ghost semantics: periodic wrap, or 0
// outside a ghosted (non-periodic) dimension.  Offsets are at most one grid
// length.
template <typename T>
__device__ __forceinline__ T gval(const T *__restrict__ F, const GridG &g, int k, int j, int i) {
  if (i < 0 || i >= g.nx) { if (g.bc[0]) return T(0); i = i < 0 ? i + g.nx : i - g.nx; }
  if (j < 0 || j >= g.ny) { if (g.bc[1]) return T(0); j = j < 0 ? j + g.ny : j - g.ny; }
  if (k < 0 || k >= g.nz) { if (g.bc[2]) return T(0); k = k < 0 ? k + g.nz : k - g.nz; }
  return F[((unsigned)k * g.ny + j) * g.nx + i];
}

// ---- 3-D launches: one thread per cell, (x, y) tiles of kTx x kTy, z from
// blockIdx.z.  No division anywhere in the index arithmetic.
constexpr int kTx = 32, kTy = 8;
static inline dim3 threads3() { return dim3(kTx, kTy, 1); }
static inline dim3 blocks3(int nx, int ny, int nz) {
  return dim3((unsigned)((nx + kTx - 1) / kTx), (unsigned)((ny + kTy - 1) / kTy), (unsigned)nz);
}
static inline dim3 blocks3(const GridG &g) { return blocks3(g.nx, g.ny, g.nz); }
__device__ __forceinline__ bool at3(int nx, int ny, int &i, int &j, int &k) {
  i = blockIdx.x * kTx + threadIdx.x;
  j = blockIdx.y * kTy + threadIdx.y;
  k = blockIdx.z;
  return i < nx && j < ny;
}
__device__ __forceinline__ unsigned lin3(const GridG &g, int i, int j, int k) {
  return ((unsigned)k * g.ny + j) * g.nx + i;
}
// Linear block index and thread index of a 3-D launch (for block partials).
__device__ __forceinline__ unsigned block_lin() {
  return (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
}
__device__ __forceinline__ int thread_lin() { return threadIdx.y * blockDim.x + threadIdx.x; }

// (i, j, k) of linear cell c, 32-bit (single-block loops over small levels).
__device__ __forceinline__ void cell_ijk(unsigned c, const GridG &g, int &i, int &j, int &k) {
  i = (int)(c % (unsigned)g.nx);
  unsigned r = c / (unsigned)g.nx;
  j = (int)(r % (unsigned)g.ny);
  k = (int)(r / (unsigned)g.ny);
}

// ---- operator (src/lhs.c:366-423), templated on the arithmetic type --------
struct OpK {
  GridG g;
  double sxx, syy, szz, sod;
  float fxx, fyy, fzz, fod;  // the same scales rounded to FP32 (FP32 rows)
  int unit;                  // density 1 at every stencil point, ghosts included (-lhs laplacian)
};
__device__ __forceinline__ void op_scales(const OpK &o, double &a, double &b, double &c, double &d) {
  a = o.sxx; b = o.syy; c = o.szz; d = o.sod;
}
__device__ __forceinline__ void op_scales(const OpK &o, float &a, float &b, float &c, float &d) {
  a = o.fxx; b = o.fyy; c = o.fzz; d = o.fod;
}

// Stencil offsets (di, dj, dk) of the 11 row entries, in the reference's
// order: x+, x-, y+, y-, z+, z-, (x+,y+), (x+,y-), (x-,y+), (x-,y-), centre.
__device__ __forceinline__ int off_i(int e) { return (e == 0 || e == 6 || e == 7) ? 1 : ((e == 1 || e == 8 || e == 9) ? -1 : 0); }
__device__ __forceinline__ int off_j(int e) { return (e == 2 || e == 6 || e == 8) ? 1 : ((e == 3 || e == 7 || e == 9) ? -1 : 0); }
__device__ __forceinline__ int off_k(int e) { return e == 4 ? 1 : (e == 5 ? -1 : 0); }

// A product that is rounded by itself, and a fused multiply-add.
__device__ __forceinline__ float mul_r(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_r(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float fma_r(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_r(double a, double b, double c) { return __fma_rn(a, b, c); }

// ---- exact sums in integers ------------------------------------------------
// FP64 adds issue at 1/64 of the FP32 rate.  Moments that come from the mixed
// deposit are whole multiples of 2^-S, and sums and differences of a few of
// them are exact in FP64 too; so they can be formed in int64 and converted
// (exactly: below 2^53) on the integer units, with the same bits.  Any other
// value takes the FP64 operations (all of them where S is kNoQuanta).
constexpr int kNoQuanta = -1;
constexpr int kQuantaBits = 50;  // |a| < 2^50: sums of up to four stay below 2^52
// a = v 2^S; false unless that is whole and below 2^kQuantaBits.
__device__ __forceinline__ bool quanta_of(double v, int S, long long &a) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const int r = 1075 - S - (int)((hi >> 20) & 0x7ffu);  // the significand's right shift
  const unsigned mh = (hi & 0xfffffu) | 0x100000u;
  const int tz = lo ? __ffs((int)lo) - 1 : 31 + __ffs((int)mh);
  const unsigned long long m = (((unsigned long long)mh << 32) | lo) >> (r & 63);
  const bool zero = (hi | lo) == 0u;  // -0 is left to the FP64 operations
  a = zero ? 0 : ((int)hi < 0 ? -(long long)m : (long long)m);
  return zero || (r >= 53 - kQuantaBits && r <= tz);
}
// a 2^-S for |a| < 2^53.
__device__ __forceinline__ double from_quanta(long long a, int S) {
  const unsigned long long m = a < 0 ? 0ull - (unsigned long long)a : (unsigned long long)a;
  const int lz = __clzll((long long)m);
  // the leading bit adds one to the exponent field
  const unsigned long long b = ((unsigned long long)(1023 + 62 - lz - S) << 52) + ((m << (lz & 63)) >> 11);
  return m == 0 ? 0.0 : __longlong_as_double((long long)(b | ((unsigned long long)a & 0x8000000000000000ull)));
}

// 11 coefficients of a row in the order above, from the density at the
// centre and its six face neighbours: the sums and differences (RowSums),
// then their products.  The roundings are written out, so that
// every kernel forms the same bits however the compiler shares the products
// of neighbouring rows.
template <typename T>
struct RowSums {
  T dy, dx;                      // n(y+) - n(y-), n(x+) - n(x-)
  T d6, d7, d8, d9;              // of the four off-diagonals
  T xp, xm, yp, ym, zp, zm;      // face sums
  T x2, y2, z2;                  // n+ + 2 n + n-
};
template <typename T>
__device__ __forceinline__ void row11_products(const OpK &o, const RowSums<T> &u, T v[11]) {
  T sxx, syy, szz, sod;
  op_scales(o, sxx, syy, szz, sod);
  const T ty = mul_r(sod, u.dy), tx = mul_r(sod, u.dx);
  v[6] = mul_r(sod, u.d6);
  v[7] = mul_r(sod, u.d7);
  v[8] = mul_r(sod, u.d8);
  v[9] = mul_r(sod, u.d9);
  v[0] = fma_r(sxx, u.xp, ty);
  v[1] = fma_r(sxx, u.xm, -ty);
  v[2] = fma_r(syy, u.yp, -tx);
  v[3] = fma_r(syy, u.ym, tx);
  v[4] = mul_r(szz, u.zp);
  v[5] = mul_r(szz, u.zm);
  v[10] = -fma_r(szz, u.z2, fma_r(sxx, u.x2, mul_r(syy, u.y2)));
}
template <typename T>
__device__ __forceinline__ void row11_vals(const OpK &o, T nijk, T nmjk, T npjk, T nimk, T nipk, T nijm, T nijp,
                                           T v[11]) {
  if (o.unit) nijk = nmjk = npjk = nimk = nipk = nijm = nijp = T(1);
  RowSums<T> u;
  u.dy = nipk - nimk;
  u.dx = npjk - nmjk;
  u.d6 = nipk - npjk;
  u.d7 = npjk - nimk;
  u.d8 = nmjk - nipk;
  u.d9 = nimk - nmjk;
  u.xp = npjk + nijk;
  u.xm = nijk + nmjk;
  u.yp = nipk + nijk;
  u.ym = nijk + nimk;
  u.zp = nijp + nijk;
  u.zm = nijk + nijm;
  u.x2 = npjk + T(2) * nijk + nmjk;
  u.y2 = nipk + T(2) * nijk + nimk;
  u.z2 = nijp + T(2) * nijk + nijm;
  row11_products(o, u, v);
}
// The same from densities a 2^-S.
__device__ __forceinline__ void row11_quanta(const OpK &o, int S, long long a, long long xm, long long xp, long long ym,
                                             long long yp, long long zm, long long zp, double v[11]) {
  RowSums<double> u;
  u.dy = from_quanta(yp - ym, S);
  u.dx = from_quanta(xp - xm, S);
  u.d6 = from_quanta(yp - xp, S);
  u.d7 = from_quanta(xp - ym, S);
  u.d8 = from_quanta(xm - yp, S);
  u.d9 = from_quanta(ym - xm, S);
  u.xp = from_quanta(xp + a, S);
  u.xm = from_quanta(a + xm, S);
  u.yp = from_quanta(yp + a, S);
  u.ym = from_quanta(a + ym, S);
  u.zp = from_quanta(zp + a, S);
  u.zm = from_quanta(a + zm, S);
  u.x2 = from_quanta(xp + 2 * a + xm, S);
  u.y2 = from_quanta(yp + 2 * a + ym, S);
  u.z2 = from_quanta(zp + 2 * a + zm, S);
  row11_products(o, u, v);
}

// 11 coefficients of row (k,j,i) in the order above.
template <typename T>
__device__ __forceinline__ void row11(const T *__restrict__ n, const OpK &o, int i, int j, int k, T v[11]) {
  const GridG &g = o.g;
  row11_vals(o, gval(n, g, k, j, i), gval(n, g, k, j, i - 1), gval(n, g, k, j, i + 1), gval(n, g, k, j - 1, i),
             gval(n, g, k, j + 1, i), gval(n, g, k - 1, j, i), gval(n, g, k + 1, j, i), v);
}

// The neighbours of cell (i,j,k) as offsets from its linear index, with the
// ghost semantics of gval: a periodic axis wraps, a ghosted one reads 0 past
// its edge (valid flag false).  Computed once per cell, so that the row's 18
// loads need no wrap logic of their own.
struct Nbr {
  unsigned c;                   // linear index of the cell
  int xm, xp, ym, yp, zm, zp;   // offsets of the six face neighbours
  bool vxm, vxp, vym, vyp, vzm, vzp;
};
__device__ __forceinline__ Nbr nbr_of(const GridG &g, int i, int j, int k) {
  Nbr q;
  const int sy = g.nx, sz = g.nx * g.ny;
  q.c = ((unsigned)k * g.ny + j) * g.nx + i;
  q.xm = i > 0 ? -1 : g.nx - 1;
  q.xp = i < g.nx - 1 ? 1 : 1 - g.nx;
  q.ym = j > 0 ? -sy : (g.ny - 1) * sy;
  q.yp = j < g.ny - 1 ? sy : (1 - g.ny) * sy;
  q.zm = k > 0 ? -sz : (g.nz - 1) * sz;
  q.zp = k < g.nz - 1 ? sz : (1 - g.nz) * sz;
  q.vxm = i > 0 || !g.bc[0];
  q.vxp = i < g.nx - 1 || !g.bc[0];
  q.vym = j > 0 || !g.bc[1];
  q.vyp = j < g.ny - 1 || !g.bc[1];
  q.vzm = k > 0 || !g.bc[2];
  q.vzp = k < g.nz - 1 || !g.bc[2];
  return q;
}
template <typename T>
__device__ __forceinline__ T nval(const T *__restrict__ F, const Nbr &q, int off, bool valid) {
  return valid ? F[(unsigned)((int)q.c + off)] : T(0);
}
// The 11 coefficients of the row (the same operands as row11).
template <typename T>
__device__ __forceinline__ void row11_n(const T *__restrict__ n, const OpK &o, const Nbr &q, T v[11]) {
  row11_vals(o, n[q.c], nval(n, q, q.xm, q.vxm), nval(n, q, q.xp, q.vxp), nval(n, q, q.ym, q.vym),
             nval(n, q, q.yp, q.vyp), nval(n, q, q.zm, q.vzm), nval(n, q, q.zp, q.vzp), v);
}
// x at the row's 11 entries, in the order of off_i/off_j/off_k.
template <typename T>
__device__ __forceinline__ void row_x(const T *__restrict__ x, const Nbr &q, T xe[11]) {
  xe[0] = nval(x, q, q.xp, q.vxp);
  xe[1] = nval(x, q, q.xm, q.vxm);
  xe[2] = nval(x, q, q.yp, q.vyp);
  xe[3] = nval(x, q, q.ym, q.vym);
  xe[4] = nval(x, q, q.zp, q.vzp);
  xe[5] = nval(x, q, q.zm, q.vzm);
  xe[6] = nval(x, q, q.xp + q.yp, q.vxp && q.vyp);
  xe[7] = nval(x, q, q.xp + q.ym, q.vxp && q.vym);
  xe[8] = nval(x, q, q.xm + q.yp, q.vxm && q.vyp);
  xe[9] = nval(x, q, q.xm + q.ym, q.vxm && q.vym);
  xe[10] = x[q.c];
}

// Operator scale factors for spacing (hx, hy, hz), src/lhs.c:366-375.  The
// constant-coefficient Laplacian of -lhs laplacian (ComputeLaplacianLHS3D,
// src/lhs.c:101-191: 1/h^2 off the diagonal, minus their sum on it, the same
// in boundary rows whose out-of-range columns are dropped) is this operator
// with kappa = 0, scale = 1 and the density 1 everywhere, ghost points
// included (`unit`): 2 * (1/(2 h^2)) equals 1/h^2 exactly.
static inline OpK make_op(const EcsParams &p, int nx, int ny, int nz, double hx, double hy, double hz) {
  OpK o;
  o.g.nx = nx; o.g.ny = ny; o.g.nz = nz;
  for (int d = 0; d < 3; d++) o.g.bc[d] = p.bc[d] == ECS_BC_PERIODIC ? 0 : 1;
  o.g.n = (size_t)nx * ny * nz;
  const bool lap = p.lhs_type == ECS_LHS_LAPLACIAN;
  double kappa = lap ? 0.0 : p.kappa_e, scale = lap ? 1.0 : p.scale;
  double hxx = 1.0 / (2.0 * hx * hx), hyy = 1.0 / (2.0 * hy * hy), hzz = 1.0 / (2.0 * hz * hz);
  double hod = 1.0 / (8.0 * hy * hx);
  o.sxx = scale * hxx;
  o.syy = scale * hyy;
  // 2-D (ComputeFullLHS2D src/lhs.c:194-335, ComputeLaplacianLHS2D
  // src/lhs.c:26-97): the same in-plane entries, no z coupling
  o.szz = p.ndim == 2 ? 0.0 : scale * (1 + kappa * kappa) * hzz;
  o.sod = scale * kappa * hod;
  o.fxx = (float)o.sxx; o.fyy = (float)o.syy; o.fzz = (float)o.szz; o.fod = (float)o.sod;
  o.unit = lap ? 1 : 0;
  return o;
}
static inline GridG make_grid(const EcsParams &p, int nx, int ny, int nz) {
  return make_op(p, nx, ny, nz, 1.0, 1.0, 1.0).g;
}

// ---- right-hand side (src/rhs.c:321-354) -------------------------------------
// The reference's operation order, every operation separately rounded.  The
// row is bound by the FP64 pipe (1/64 of the FP32 rate), so what FP64
// arithmetic cannot change runs on the integer units: products with a power of
// two (1/(2 dx), 1/dx^2 of a power-of-two spacing, 2 n) are exponent
// additions, 1 + kappa^2 is formed on the host, and without a background field
// its term, an exact zero for finite densities, is left out.  128^3 and
// dx = 1: 42 -> 25 FP64 operations a cell.
constexpr int kNoPow2 = 1 << 20;
struct RhsK {
  double kappa, opk2, hx, hy, hz, hxx, hyy, hzz, E0, cth, cG, scale;
  int px, py, pz, pxx, pyy, pzz;  // h = 2^p exactly, or kNoPow2
};
static inline int pow2_of(double h) {
  int e = 0;
  return frexp(h, &e) == 0.5 && e >= -62 && e <= 64 ? e - 1 : kNoPow2;
}
static inline RhsK make_rhs(const EcsParams &p, double dz) {
  RhsK r;
  volatile double k2 = p.kappa_e * p.kappa_e;  // rounded by itself
  r.kappa = p.kappa_e;
  r.opk2 = 1.0 + k2;
  r.hx = 1.0 / (2.0 * p.dx); r.hy = 1.0 / (2.0 * p.dy); r.hz = 1.0 / (2.0 * dz);
  r.hxx = 1.0 / (p.dx * p.dx); r.hyy = 1.0 / (p.dy * p.dy); r.hzz = 1.0 / (dz * dz);
  r.px = pow2_of(r.hx); r.py = pow2_of(r.hy); r.pz = pow2_of(r.hz);
  r.pxx = pow2_of(r.hxx); r.pyy = pow2_of(r.hyy); r.pzz = pow2_of(r.hzz);
  r.E0 = p.E0; r.cth = p.cth; r.cG = p.cG; r.scale = p.scale;
  return r;
}
// h v for h = 2^p (any h when p is kNoPow2).
__device__ __forceinline__ rd scale2(double h, int p, rd v) {
  const int hi = __double2hiint(v.v), e = (hi >> 20) & 0x7ff;
  if (p == kNoPow2 || (unsigned)(e - 128) > 1792u) return e == 0 && ((hi << 1) | __double2loint(v.v)) == 0 ? v : rd{h} * v;
  return rd{__hiloint2double(hi + p * (1 << 20), __double2loint(v.v))};
}
// b from the derivatives; with a background field also those of the density
// along x and y (dndx(), dndy()).
template <typename X, typename Y>
__device__ __forceinline__ double rhs_combine(const RhsK &r, rd d2ndxx, rd d2ndyy, rd d2ndzz, rd dGxdx, rd dGydy,
                                              rd dGzdz, X dndx, Y dndy) {
  rd t = rd{r.cth} * ((d2ndxx + d2ndyy) + rd{r.opk2} * d2ndzz);
  if (r.E0 != 0.0) t = (dndy() - rd{r.kappa} * dndx()) * rd{r.E0} + t;
  const rd Gterm = rd{r.cG} * ((dGxdx + dGydy) + dGzdz);
  return (rd{r.scale} * (t + Gterm)).v;
}
// b from the density at the node and its six neighbours and the flux at the
// two neighbours along its own axis.
__device__ __forceinline__ double rhs_value(const RhsK &r, rd nijk, rd npjk, rd nmjk, rd nipk, rd nimk, rd nijp, rd nijm,
                                            rd gxp, rd gxm, rd gyp, rd gym, rd gzp, rd gzm) {
  const rd n2 = scale2(2.0, 1, nijk);
  const rd d2ndxx = scale2(r.hxx, r.pxx, (npjk - n2) + nmjk);
  const rd d2ndyy = scale2(r.hyy, r.pyy, (nipk - n2) + nimk);
  const rd d2ndzz = scale2(r.hzz, r.pzz, (nijp - n2) + nijm);
  const rd dGxdx = scale2(r.hx, r.px, gxp - gxm);
  const rd dGydy = scale2(r.hy, r.py, gyp - gym);
  const rd dGzdz = scale2(r.hz, r.pz, gzp - gzm);
  return rhs_combine(r, d2ndxx, d2ndyy, d2ndzz, dGxdx, dGydy, dGzdz, [&] { return scale2(r.hx, r.px, npjk - nmjk); },
                     [&] { return scale2(r.hy, r.py, nipk - nimk); });
}
