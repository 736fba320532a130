// ecs_rhs_noalloc: the right-hand side of the quasineutral potential equation
// (ComputeFullRHS3D src/rhs.c:259-373 / ComputeFullRHS2D src/rhs.c:151-256,
// or the -rhs constant / sinusoidal options src/rhs.c:6-148, each with the
// reference's mean removal) for callers that cannot allocate device memory.
//
// Some callers cannot call cudaMalloc at the point where they need the RHS:
// a host framework that reserves its whole device-memory budget in its own
// pool at start-up and forbids allocations inside its time-step loop, or a
// latency-critical loop that cannot accept the implicit device
// synchronisation an allocation may cause.  They own the input and output
// buffers; this entry point needs only a small reduction scratch, which lives
// in a file-scope __device__ array instead of an allocation.
//
// Scratch: ECS_NOALLOC_RHS_MAX_BLOCKS FP64 block partial sums plus a slot for
// the mean and one for the reduction's completion count (32 KiB + 16 B),
// present on every device that loads the library until the process exits.
// Each thread block reduces at most ECS_NOALLOC_RHS_CELLS_PER_BLOCK cells, so
// grids of at most ECS_NOALLOC_RHS_MAX_CELLS cells (256 x 256 x 128) are
// accepted.
//
// Every call shares the array: each call writes every partial and the mean
// before it reads them, and the block that finishes last puts the completion
// count back to 0, so a call needs nothing of the calls before it.  Two calls
// that overlap on the GPU (different streams without ordering) race on it:
// either may then subtract a mean of mixed partials or an earlier call's mean.
// A call ordered after both is right again (k_sub_mean_noalloc clears the
// count).
//
// The array's device address is looked up once per device, the first time a
// call runs with that device current, and cached for the life of the
// process.  The cache does not survive cudaDeviceReset (or anything else that
// replaces the device's primary context): a process that resets a device
// must not call this entry point on it afterwards.
#include <math.h>

#include <algorithm>
#include <mutex>

#include "ecs_stencil.cuh"

#define ECS_NOALLOC_RHS_MAX_BLOCKS 4096
#define ECS_NOALLOC_RHS_CELLS_PER_BLOCK 2048
#define ECS_NOALLOC_RHS_MAX_CELLS (ECS_NOALLOC_RHS_MAX_BLOCKS * ECS_NOALLOC_RHS_CELLS_PER_BLOCK)
#define ECS_NOALLOC_MAX_DEVICES 64

// [0, MAX_BLOCKS): block partial sums of b; [MAX_BLOCKS]: the mean of b;
// [MAX_BLOCKS + 1]: blocks done (0 between calls).
static __device__ __align__(256) double g_rhs_scratch[ECS_NOALLOC_RHS_MAX_BLOCKS + 2];

namespace {

constexpr int kThreads = 256;

struct RhsNoAllocK {
  int nx, ny, nz;
  int bc[3];
  int ndim;
  size_t n;
  RhsK r;
  double scale, dx, dy, dz, n0;  // -rhs sinusoidal
};

// b of the full RHS (src/rhs.c:321-354) at node (k, j, i) from
// FluidNode{n,Gx,Gy,Gz} storage, with the reference's ghost semantics
// (periodic wrap, zero outside ghosted axes).  A 2-D grid is one node deep
// with a unit, periodic z cell, so every z term is exactly 0.
__device__ __forceinline__ double full_rhs(const double *__restrict__ mom, const RhsNoAllocK &g, int k, int j,
                                           int i) {
  GridG gg;
  gg.nx = g.nx; gg.ny = g.ny; gg.nz = g.nz;
  for (int d = 0; d < 3; d++) gg.bc[d] = g.bc[d];
  const Nbr q = nbr_of(gg, i, j, k);
  auto at = [&](int off, bool valid, int c) {
    return rd{valid ? mom[(size_t)(unsigned)((int)q.c + off) * 4 + c] : 0.0};
  };
  return rhs_value(g.r, at(0, true, 0), at(q.xp, q.vxp, 0), at(q.xm, q.vxm, 0), at(q.yp, q.vyp, 0),
                   at(q.ym, q.vym, 0), at(q.zp, q.vzp, 0), at(q.zm, q.vzm, 0), at(q.xp, q.vxp, 1),
                   at(q.xm, q.vxm, 1), at(q.yp, q.vyp, 2), at(q.ym, q.vym, 2), at(q.zp, q.vzp, 3),
                   at(q.zm, q.vzm, 3));
}

// b of -rhs sinusoidal (src/rhs.c:82-148; 2-D src/rhs.c:26-79): n0 cos(2 pi
// x) cos(2 pi y) [cos(2 pi z)] scale at the cell centres in grid units.
__device__ __forceinline__ double sin_rhs(const RhsNoAllocK &g, int k, int j, int i) {
  const double twopi = 2 * M_PI;
  const double cx = cos(__dmul_rn(twopi, __dmul_rn(__dadd_rn((double)i, 0.5), g.dx)));
  const double cy = cos(__dmul_rn(twopi, __dmul_rn(__dadd_rn((double)j, 0.5), g.dy)));
  const double cxy = __dmul_rn(cx, cy);
  const double val =
      g.ndim == 2 ? cxy : __dmul_rn(cxy, cos(__dmul_rn(twopi, __dmul_rn(__dadd_rn((double)k, 0.5), g.dz))));
  return __dmul_rn(__dmul_rn(g.n0, val), g.scale);
}

// One block per `cells` consecutive cells (256 on small grids, so that the
// FP64 work spreads over the SMs: with 2048 always, a 32^3 grid ran on 16 of
// them); each block writes its partial sum of b into partials[blockIdx.x], and
// the one that finishes last forms the mean from the partials in a fixed order
// (strided per thread, warp tree, then the warps in order).  No block waits on
// another.
template <bool kSinusoidal>
__global__ void __launch_bounds__(kThreads) k_rhs_noalloc(RhsNoAllocK g, int cells, const double *__restrict__ mom,
                                                          double *__restrict__ b, double *__restrict__ partials) {
  __shared__ double sh[kThreads / 32];
  __shared__ int last;
  double local = 0.0;
  const unsigned c0 = blockIdx.x * (unsigned)cells, n = (unsigned)g.n;
  for (unsigned c = c0 + threadIdx.x; c < n && c < c0 + (unsigned)cells; c += kThreads) {
    const unsigned r = c / (unsigned)g.nx;
    const int i = (int)(c - r * (unsigned)g.nx), j = (int)(r % (unsigned)g.ny), k = (int)(r / (unsigned)g.ny);
    const double v = kSinusoidal ? sin_rhs(g, k, j, i) : full_rhs(mom, g, k, j, i);
    b[c] = v;
    local += v;
  }
  auto block_sum = [&](double t) {
    for (int s = 16; s >= 1; s >>= 1) t += __shfl_xor_sync(ECS_FULL_MASK, t, s);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = t;
    __syncthreads();
    double u = 0.0;
    if (threadIdx.x == 0)
      for (int w = 0; w < kThreads / 32; w++) u += sh[w];
    return u;
  };
  const double mine = block_sum(local);
  unsigned int *done = reinterpret_cast<unsigned int *>(partials + ECS_NOALLOC_RHS_MAX_BLOCKS + 1);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = mine;
    __threadfence();
    last = atomicAdd(done, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  double t = 0.0;
  for (unsigned q = threadIdx.x; q < gridDim.x; q += kThreads) t += __ldcg(partials + q);
  const double u = block_sum(t);
  if (threadIdx.x == 0) {
    partials[ECS_NOALLOC_RHS_MAX_BLOCKS] = u / (double)g.n;
    *done = 0u;  // here, not in the next kernel alone: that launch can fail
  }
}

// b -= mean.  Also clears the completion count, whatever calls that overlapped
// this one have left there, so that the next call starts clean.
__global__ void __launch_bounds__(kThreads) k_sub_mean_noalloc(size_t n, double *__restrict__ b, double *partials) {
  if (blockIdx.x == 0 && threadIdx.x == 0)
    *reinterpret_cast<unsigned int *>(partials + ECS_NOALLOC_RHS_MAX_BLOCKS + 1) = 0u;
  const double mean = partials[ECS_NOALLOC_RHS_MAX_BLOCKS];
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x)
    b[c] -= mean;
}

// -rhs constant (src/rhs.c:6-23): b = n0 scale everywhere, no projection.
__global__ void __launch_bounds__(kThreads) k_fill_noalloc(size_t n, double v, double *__restrict__ b) {
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x)
    b[c] = v;
}

// Device address of the scratch array, looked up once per device.
std::mutex g_setup_mutex;
double *g_scratch_addr[ECS_NOALLOC_MAX_DEVICES] = {nullptr};

cudaError_t scratch_for_current_device(double **out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= ECS_NOALLOC_MAX_DEVICES) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  if (!g_scratch_addr[dev]) {
    double *ptr = nullptr;
    e = cudaGetSymbolAddress((void **)&ptr, g_rhs_scratch);
    if (e != cudaSuccess) return e;
    g_scratch_addr[dev] = ptr;
  }
  *out = g_scratch_addr[dev];
  return cudaSuccess;
}

int launched(const char *what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return ecs_fail(nullptr, ECS_ERR_CUDA, "ecs_rhs_noalloc: %s launch: %s", what, cudaGetErrorString(e));
  return ECS_OK;
}

}  // namespace

extern "C" int ecs_rhs_noalloc(const EcsParams *params, const double *d_moments, double *d_rhs, void *stream) {
  if (!params || !d_rhs) return ecs_fail(nullptr, ECS_ERR_INVALID, "ecs_rhs_noalloc: NULL argument");
  int rc = ecs_validate_params(params);  // the checks of ecs_ctx_create
  if (rc) return rc;
  if (params->rhs_type == ECS_RHS_FULL && !d_moments)
    return ecs_fail(nullptr, ECS_ERR_INVALID, "ecs_rhs_noalloc: NULL moments for -rhs full");
  // 2-D runs on a one-node-deep grid with a unit, periodic z cell, as a
  // context does (the reference's 2-D parameters have dz = 0)
  EcsParams p = *params;
  if (p.ndim == 2) {
    p.dz = 1.0;
    p.bc[2] = ECS_BC_PERIODIC;
  }
  const size_t n = (size_t)p.Nx * p.Ny * p.Nz;
  if (n > (size_t)ECS_NOALLOC_RHS_MAX_CELLS)
    return ecs_fail(nullptr, ECS_ERR_INVALID,
                    "ecs_rhs_noalloc: %zu grid nodes exceed the fixed scratch limit of %d nodes "
                    "(256x256x128); use ecs_rhs on a context for larger grids",
                    n, ECS_NOALLOC_RHS_MAX_CELLS);
  double *scratch = nullptr;
  cudaError_t e = scratch_for_current_device(&scratch);
  if (e != cudaSuccess)
    return ecs_fail(nullptr, ECS_ERR_CUDA, "ecs_rhs_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
  cudaStream_t s = (cudaStream_t)stream;
  const int nb_elem = (int)std::min<size_t>((n + kThreads - 1) / kThreads, 4096);
  if (p.rhs_type == ECS_RHS_CONSTANT) {
    k_fill_noalloc<<<nb_elem, kThreads, 0, s>>>(n, p.n0 * p.scale, d_rhs);
    return launched("fill");
  }
  RhsNoAllocK g;
  g.nx = p.Nx; g.ny = p.Ny; g.nz = p.Nz;
  for (int d = 0; d < 3; d++) g.bc[d] = p.bc[d] == ECS_BC_PERIODIC ? 0 : 1;
  g.ndim = p.ndim;
  g.n = n;
  g.r = make_rhs(p, p.dz);
  g.scale = p.scale;
  g.dx = p.dx; g.dy = p.dy; g.dz = p.dz; g.n0 = p.n0;
  const int cells = (int)std::max<size_t>(kThreads, ((n + ECS_NOALLOC_RHS_MAX_BLOCKS - 1) / ECS_NOALLOC_RHS_MAX_BLOCKS +
                                                     kThreads - 1) / kThreads * kThreads);
  const int nb = (int)((n + cells - 1) / cells);
  if (p.rhs_type == ECS_RHS_SINUSOIDAL)
    k_rhs_noalloc<true><<<nb, kThreads, 0, s>>>(g, cells, d_moments, d_rhs, scratch);
  else
    k_rhs_noalloc<false><<<nb, kThreads, 0, s>>>(g, cells, d_moments, d_rhs, scratch);
  if ((rc = launched("rhs"))) return rc;
  k_sub_mean_noalloc<<<nb_elem, kThreads, 0, s>>>(n, d_rhs, scratch);
  return launched("mean removal");
}
