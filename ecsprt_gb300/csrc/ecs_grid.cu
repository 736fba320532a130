// Grid phase of the ECSPRT hot path on sm_103a (everything but the solver):
//   difference numerators of phi on the extended node grid (input to push)
//   fixed-point -> FP64 moments                       src/moments.c:208-211
//   RHS of the quasineutral potential equation         src/rhs.c:259-373
// All kernels are 3-D launches over (x, y) tiles and z (no index division);
// the RHS mean is a fixed-order reduction, so results repeat run to run.
#include <math.h>

#include <algorithm>

#include "ecs_stencil.cuh"

namespace {

// ---- difference numerators on the extended (N+1)^3 node grid -------------
// src/vector-math.c:619-712: central difference at every node index < N, the
// backward formula at index N (reached only as the high corner of the last
// cell).  FP64, separately rounded.
__device__ __forceinline__ double dnum(const double *F, const GridG &g, int axis, int k, int j, int i) {
  int N = axis == 0 ? g.nx : (axis == 1 ? g.ny : g.nz);
  int h = axis == 0 ? i : (axis == 1 ? j : k);
  auto at = [&](int o) -> rd {
    return rd{axis == 0 ? gval(F, g, k, j, i + o) : (axis == 1 ? gval(F, g, k, j + o, i) : gval(F, g, k + o, j, i))};
  };
  if (h < N) return (at(1) - at(-1)).v;
  return ((rd{3.0} * at(0) - rd{4.0} * at(-1)) + rd{1.0} * at(-2)).v;
}

__global__ void k_eext(GridG g, const double *__restrict__ phi, double4_32a *__restrict__ e64,
                       float4 *__restrict__ e32) {
  const int sx = g.nx + 1, sy = g.ny + 1;
  int i, j, k;
  if (!at3(sx, sy, i, j, k)) return;
  const unsigned e = ((unsigned)k * sy + j) * sx + i;
  double dx = dnum(phi, g, 0, k, j, i), dy = dnum(phi, g, 1, k, j, i), dz = dnum(phi, g, 2, k, j, i);
  if (e64) e64[e] = make_double4_32a(dx, dy, dz, 0.0);
  if (e32) e32[e] = make_float4((float)dx, (float)dy, (float)dz, 0.0f);
}

// ---- moments -----------------------------------------------------------------
// a 2^-S rounded to nearest even, in integers: the conversion and the product
// would take two slots of the FP64 pipe, 1/64 of the FP32 rate, which bound
// this kernel (256 x 256 x 128: 154 -> 83 us; bandwidth bounds it now).
__device__ __forceinline__ double fix_value(long long a, int S) {
  const unsigned long long m = a < 0 ? 0ull - (unsigned long long)a : (unsigned long long)a;
  if (m == 0) return 0.0;
  const int lz = __clzll((long long)m);
  const unsigned long long t = m << lz, q = t >> 11;  // 53 bits and what is rounded off
  const unsigned up = ((unsigned)(t & 0x7ffu) + 0x3ffu + (unsigned)(q & 1u)) >> 11;
  // q carries the leading bit: one more in the exponent field
  const unsigned long long v = ((unsigned long long)(1023 + 62 - lz - S) << 52) + q + up;
  return __longlong_as_double((long long)(v | ((unsigned long long)a & 0x8000000000000000ull)));
}

// mom[f][c] from acc[4 c + f] (INTERLEAVED) or acc[f][c]; a thread takes all
// four fields of a cell.
template <bool INTERLEAVED>
__global__ void k_moments(size_t n, const long long *__restrict__ acc, double *__restrict__ mom, int shift_n,
                          int shift_f, EcsDevStatus *st) {
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
    long long a[4];
    if (INTERLEAVED) {
      const longlong2 lo = reinterpret_cast<const longlong2 *>(acc)[2 * c], hi = reinterpret_cast<const longlong2 *>(acc)[2 * c + 1];
      a[0] = lo.x; a[1] = lo.y; a[2] = hi.x; a[3] = hi.y;
    } else {
#pragma unroll
      for (int f = 0; f < 4; f++) a[f] = acc[f * n + c];
    }
    bool out = false;
#pragma unroll
    for (int f = 0; f < 4; f++) {
      out |= a[f] > (1ll << 62) || a[f] < -(1ll << 62);
      mom[f * n + c] = fix_value(a[f], f == 0 ? shift_n : shift_f);
    }
    if (out) atomicOr(&st->flags, ECS_FLAG_RANGE);
  }
}

// ---- RHS: src/rhs.c:321-354 (rhs_value) ---------------------------------------
// Fixed-order sum of `local` over the block into partial[block].
__device__ __forceinline__ void block_partial(double local, double *sh, double *__restrict__ partial) {
  for (int s = 16; s >= 1; s >>= 1) local += __shfl_xor_sync(ECS_FULL_MASK, local, s);
  const int t = thread_lin();
  if ((t & 31) == 0) sh[t >> 5] = local;
  __syncthreads();
  if (t == 0) {
    double u = 0.0;
    for (int w = 0; w < kTx * kTy / 32; w++) u += sh[w];
    partial[block_lin()] = u;
  }
}

// b at every cell; each block writes the sum of its cells to partial[block]
// (z loop with stride gridDim.z, so the block count stays bounded).
__global__ void k_rhs(GridG g, RhsK r, const double *__restrict__ mom, double *__restrict__ b,
                      double *__restrict__ partial) {
  __shared__ double sh[kTx * kTy / 32];
  double local = 0.0;
  const double *n = mom, *Gx = mom + g.n, *Gy = mom + 2 * g.n, *Gz = mom + 3 * g.n;
  int i, j, k0;
  if (at3(g.nx, g.ny, i, j, k0)) {
    for (int k = k0; k < g.nz; k += gridDim.z) {
      const Nbr q = nbr_of(g, i, j, k);  // the neighbours' offsets (gval's wrap and ghosts)
      const double v = rhs_value(
          r, rd{n[q.c]}, rd{nval(n, q, q.xp, q.vxp)}, rd{nval(n, q, q.xm, q.vxm)}, rd{nval(n, q, q.yp, q.vyp)},
          rd{nval(n, q, q.ym, q.vym)}, rd{nval(n, q, q.zp, q.vzp)}, rd{nval(n, q, q.zm, q.vzm)},
          rd{nval(Gx, q, q.xp, q.vxp)}, rd{nval(Gx, q, q.xm, q.vxm)}, rd{nval(Gy, q, q.yp, q.vyp)},
          rd{nval(Gy, q, q.ym, q.vym)}, rd{nval(Gz, q, q.zp, q.vzp)}, rd{nval(Gz, q, q.zm, q.vzm)});
      b[q.c] = v;
      local += v;
    }
  }
  block_partial(local, sh, partial);
}

// The same with the differences of moments that are whole quanta (2^-Sn,
// 2^-Sf) formed in integers: 25 -> 16 FP64 operations a cell.  Launched for
// moments of a mixed deposit (EcsCtx::mom_quanta); a cell with any other value
// takes the FP64 operations here too, at a loss (the whole ecs_rhs at 128^3,
// dx = 1: 134 -> 111 us; moments without quanta 145 against k_rhs's 134).
__global__ void __launch_bounds__(kTx * kTy, 4) k_rhs_quanta(GridG g, RhsK r, int Sn, int Sf,
                                                             const double *__restrict__ mom, double *__restrict__ b,
                                                             double *__restrict__ partial) {
  __shared__ double sh[kTx * kTy / 32];
  double local = 0.0;
  const double *n = mom, *Gx = mom + g.n, *Gy = mom + 2 * g.n, *Gz = mom + 3 * g.n;
  int i, j, k0;
  if (at3(g.nx, g.ny, i, j, k0)) {
    for (int k = k0; k < g.nz; k += gridDim.z) {
      const Nbr q = nbr_of(g, i, j, k);
      // centre, then + and - along x, y, z
      const double m[7] = {n[q.c],
                           nval(n, q, q.xp, q.vxp), nval(n, q, q.xm, q.vxm), nval(n, q, q.yp, q.vyp),
                           nval(n, q, q.ym, q.vym), nval(n, q, q.zp, q.vzp), nval(n, q, q.zm, q.vzm)};
      const double G[6] = {nval(Gx, q, q.xp, q.vxp), nval(Gx, q, q.xm, q.vxm), nval(Gy, q, q.yp, q.vyp),
                           nval(Gy, q, q.ym, q.vym), nval(Gz, q, q.zp, q.vzp), nval(Gz, q, q.zm, q.vzm)};
      long long a[7], f[6];
      bool whole = true;
#pragma unroll
      for (int e = 0; e < 7; e++) whole &= quanta_of(m[e], Sn, a[e]);
#pragma unroll
      for (int e = 0; e < 6; e++) whole &= quanta_of(G[e], Sf, f[e]);
      double v;
      if (whole) {
        auto dif = [&](double h, int p, long long c, int S) { return scale2(h, p, rd{from_quanta(c, S)}); };
        v = rhs_combine(
            r, dif(r.hxx, r.pxx, a[1] - 2 * a[0] + a[2], Sn), dif(r.hyy, r.pyy, a[3] - 2 * a[0] + a[4], Sn),
            dif(r.hzz, r.pzz, a[5] - 2 * a[0] + a[6], Sn), dif(r.hx, r.px, f[0] - f[1], Sf),
            dif(r.hy, r.py, f[2] - f[3], Sf), dif(r.hz, r.pz, f[4] - f[5], Sf),
            [&] { return dif(r.hx, r.px, a[1] - a[2], Sn); }, [&] { return dif(r.hy, r.py, a[3] - a[4], Sn); });
      } else {
        v = rhs_value(r, rd{m[0]}, rd{m[1]}, rd{m[2]}, rd{m[3]}, rd{m[4]}, rd{m[5]}, rd{m[6]}, rd{G[0]}, rd{G[1]},
                      rd{G[2]}, rd{G[3]}, rd{G[4]}, rd{G[5]});
      }
      b[q.c] = v;
      local += v;
    }
  }
  block_partial(local, sh, partial);
}

// -rhs sinusoidal (ComputeSinusoidalRHS3D, src/rhs.c:82-148): b = n0 cos(2 pi
// x) cos(2 pi y) cos(2 pi z) scale at the cell centres x = (i + 1/2) dx (in
// the grid's own units, as the reference), block partials for the mean that
// MatNullSpaceRemove takes out (src/rhs.c:138-141).
__global__ void k_rhs_sin(GridG g, int ndim, double dx, double dy, double dz, double n0, double scale,
                          double *__restrict__ b, double *__restrict__ partial) {
  __shared__ double sh[kTx * kTy / 32];
  double local = 0.0;
  int i, j, k0;
  if (at3(g.nx, g.ny, i, j, k0)) {
    const double twopi = 2 * M_PI;
    const double cx = cos(__dmul_rn(twopi, __dmul_rn(__dadd_rn((double)i, 0.5), dx)));
    const double cy = cos(__dmul_rn(twopi, __dmul_rn(__dadd_rn((double)j, 0.5), dy)));
    for (int k = k0; k < g.nz; k += gridDim.z) {
      // 2-D (ComputeSinusoidalRHS2D src/rhs.c:26-79): n0 Cx Cy scale
      const double cxy = __dmul_rn(cx, cy);
      const double val =
          ndim == 2 ? cxy : __dmul_rn(cxy, cos(__dmul_rn(twopi, __dmul_rn(__dadd_rn((double)k, 0.5), dz))));
      const double v = __dmul_rn(__dmul_rn(n0, val), scale);
      b[lin3(g, i, j, k)] = v;
      local += v;
    }
  }
  block_partial(local, sh, partial);
}

// -rhs constant (ComputeConstantRHS, src/rhs.c:6-23): b = n0 * scale, no
// projection.
__global__ void k_fill(size_t n, double v, double *__restrict__ b) {
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) b[c] = v;
}

// out[0] = (sum of partial[0..nb)) / div, one block, fixed order.
__global__ void __launch_bounds__(1024) k_sum_final(int nb, const double *__restrict__ partial, double div,
                                                    double *__restrict__ out) {
  __shared__ double sh[32];
  double t = 0.0;
  for (int q = threadIdx.x; q < nb; q += blockDim.x) t += partial[q];
  for (int s = 16; s >= 1; s >>= 1) t += __shfl_xor_sync(ECS_FULL_MASK, t, s);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    double u = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); q++) u += sh[q];
    out[0] = u / div;
  }
}

// v -= mean (src/rhs.c:363-366)
__global__ void k_sub_value(size_t n, double *__restrict__ v, const double *__restrict__ mean) {
  const double m = *mean;
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x)
    v[c] -= m;
}

unsigned int blocks1d(const EcsCtx *ctx, size_t n) {
  size_t want = (n + 255) / 256;
  size_t cap = (size_t)ctx->nsm * 8;
  if (want > cap) want = cap;
  return (unsigned int)(want ? want : 1);
}

}  // namespace

// ============================================================================
// entry points used by ecs_api.cu
// ============================================================================
int ecs_grid_eext(EcsCtx *ctx) {
  GridG g = make_grid(ctx->p, ctx->p.Nx, ctx->p.Ny, ctx->p.Nz);
  k_eext<<<blocks3(g.nx + 1, g.ny + 1, g.nz + 1), threads3(), 0, ctx->stream>>>(
      g, ctx->phi, ctx->prec == ECS_PREC_FP64 ? ctx->eext64 : nullptr,
      ctx->prec == ECS_PREC_MIXED ? ctx->eext32 : nullptr);
  ECS_LAUNCHED(ctx);
  return ECS_OK;
}

int ecs_grid_clear_acc(EcsCtx *ctx) {
  ECS_CUDA(ctx, cudaMemsetAsync(ctx->acc, 0, ctx->ncell * 4 * sizeof(long long), ctx->stream));
  return ECS_OK;
}

int ecs_grid_moments(EcsCtx *ctx) {
  const unsigned g = blocks1d(ctx, ctx->ncell);
  if (ecs_acc_interleaved(ctx))
    k_moments<true><<<g, 256, 0, ctx->stream>>>(ctx->ncell, ctx->acc, ctx->mom, ctx->shift_n, ctx->shift_f, ctx->dstat);
  else
    k_moments<false><<<g, 256, 0, ctx->stream>>>(ctx->ncell, ctx->acc, ctx->mom, ctx->shift_n, ctx->shift_f, ctx->dstat);
  ECS_LAUNCHED(ctx);
  ctx->moments_ready = true;
  ctx->mom_quanta = ctx->prec == ECS_PREC_MIXED;
  return ECS_OK;
}

int ecs_grid_rhs(EcsCtx *ctx) {
  int rc = ecs_solver_alloc(ctx);
  if (rc) return rc;
  const EcsParams &p = ctx->p;
  if (p.rhs_type == ECS_RHS_CONSTANT) {
    k_fill<<<blocks1d(ctx, ctx->ncell), 256, 0, ctx->stream>>>(ctx->ncell, p.n0 * p.scale, ctx->rhs);
    ECS_LAUNCHED(ctx);
    return ECS_OK;
  }
  GridG g = make_grid(p, p.Nx, p.Ny, p.Nz);
  dim3 grid = blocks3(g);
  const unsigned plane_blocks = grid.x * grid.y;
  grid.z = std::max(1u, std::min(grid.z, (unsigned)ctx->nred / plane_blocks));
  const int nb = (int)(grid.x * grid.y * grid.z);
  if (p.rhs_type == ECS_RHS_SINUSOIDAL) {
    k_rhs_sin<<<grid, threads3(), 0, ctx->stream>>>(g, p.ndim, p.dx, p.dy, p.dz, p.n0, p.scale, ctx->rhs, ctx->red);
  } else {
    const RhsK r = make_rhs(p, p.dz);
    if (ctx->mom_quanta)
      k_rhs_quanta<<<grid, threads3(), 0, ctx->stream>>>(g, r, ctx->shift_n, ctx->shift_f, ctx->mom, ctx->rhs, ctx->red);
    else
      k_rhs<<<grid, threads3(), 0, ctx->stream>>>(g, r, ctx->mom, ctx->rhs, ctx->red);
  }
  ECS_LAUNCHED(ctx);
  k_sum_final<<<1, 1024, 0, ctx->stream>>>(nb, ctx->red, (double)ctx->ncell, ctx->dots);
  ECS_LAUNCHED(ctx);
  k_sub_value<<<blocks1d(ctx, ctx->ncell), 256, 0, ctx->stream>>>(ctx->ncell, ctx->rhs, ctx->dots);
  ECS_LAUNCHED(ctx);
  return ECS_OK;
}
