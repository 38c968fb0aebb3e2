// jacobi_cluster.cu -- FP64 Jacobi sweeps (CalcEpotential.f90:74-96) of a grid
// that fits the shared memory of one thread-block cluster.
//
// A sweep of 32^3 nodes is a third of a microsecond of FP64 work, but 4 us as a
// launch of its own that reads the iterate from L2.  Here one cluster of up to
// 16 CTAs runs a whole batch of sweeps: each CTA keeps a slab of z planes of the
// iterate in shared memory (two buffers, read and written by turns), each thread
// keeps b of its nodes in registers, and after a sweep a CTA stores its first and
// last plane into its neighbours' halo planes (distributed shared memory) and
// meets the others at the cluster barrier, which all of them reach once per sweep.
// A launch reads one iterate and writes another, so the one it started from stays
// as the anchor for a replay.
//
// The update is the expression of sweep_f64_kernel; the residual takes the
// reciprocals of the squared spacings instead of dividing by them.  Its squares
// are summed per warp in a fixed order, one partial per warp and sweep.
//
// What bounds it: FP64 issue on 16 SMs and the barrier.  32^3 (16 CTAs, two nodes
// a thread): 1.33 us per sweep against 4.07 us of kernel time and 3.3 us of host
// time for one launch per sweep.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "grid.cuh"
#include "stencil.cuh"

namespace picard {

namespace {

constexpr int kClThreads = 1024;
constexpr int kClWarps = kClThreads / 32;
constexpr int kClMaxNodes = 8;             // nodes per thread
constexpr size_t kClSmem = 220 * 1024;     // per CTA

struct ClusterArgs {
  int nx, ny, nz, px, py, pz;
  int planes;            // most planes of one CTA
  double ax, ay, az, af, idx2, idy2, idz2;
  const double* Uin;
  double* Uout;
  const double* b;
  double* partial;       // [m][ctas * kClWarps]
  int m;
};

// First plane (1-based) of CTA r of c.
__host__ __device__ inline int first_plane(int nz, int c, int r) { return int((long long)nz * r / c) + 1; }

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t remote_addr(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ void store_remote(uint32_t addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

template <int NPT>
__global__ void __launch_bounds__(kClThreads, 1) sweeps_cluster_kernel(ClusterArgs A) {
  extern __shared__ double cl_smem[];  // [2][planes + 2][ny + 2][nx + 2]
  const int cta = blockIdx.x, ctas = gridDim.x, tid = threadIdx.x;
  const int nxp = A.nx + 2, nyp = A.ny + 2, area = nxp * nyp;
  const int k0 = first_plane(A.nz, ctas, cta), np = first_plane(A.nz, ctas, cta + 1) - k0;
  const int buf = (A.planes + 2) * area;
  // planes k0 - 1 .. k0 + np into both buffers; a periodic axis takes the wrapped
  // interior for its ghosts
  for (int e = tid; e < (np + 2) * area; e += kClThreads) {
    const int p = e / area, r = e - p * area;
    int j = r / nxp, i = r - j * nxp, k = k0 - 1 + p;
    if (A.px) i = i == 0 ? A.nx : i == A.nx + 1 ? 1 : i;
    if (A.py) j = j == 0 ? A.ny : j == A.ny + 1 ? 1 : j;
    if (A.pz) k = k == 0 ? A.nz : k == A.nz + 1 ? 1 : k;
    const double u = A.Uin[(long long)i + (long long)nxp * (j + (long long)nyp * k)];
    cl_smem[e] = u;
    cl_smem[buf + e] = u;
  }
  // this thread's nodes: offset in a buffer (-1: none) and b
  int off[NPT];
  double b[NPT];
  const int interior = A.nx * A.ny;
#pragma unroll
  for (int q = 0; q < NPT; ++q) {
    const int e = tid + q * kClThreads;
    off[q] = -1;
    b[q] = 0.0;
    if (e < np * interior) {
      const int p = e / interior, r = e - p * interior, j = r / A.nx, i = r - j * A.nx;
      off[q] = (p + 1) * area + (j + 1) * nxp + (i + 1);
      b[q] = A.b[(long long)(i + 1) + (long long)nxp * (j + 1 + (long long)nyp * (k0 + p))];
    }
  }
  // the neighbours' halo planes that take this CTA's first and last plane
  const int below = cta > 0 ? cta - 1 : A.pz ? ctas - 1 : -1, above = cta + 1 < ctas ? cta + 1 : A.pz ? 0 : -1;
  const uint32_t base = smem_addr(cl_smem);
  uint32_t to_below = 0, to_above = 0;  // remote address of the halo plane's buffer 0, less this plane's own offset
  if (below >= 0) {
    const int npb = first_plane(A.nz, ctas, below + 1) - first_plane(A.nz, ctas, below);
    to_below = remote_addr(base, below) + uint32_t(8 * (npb + 1 - 1) * area);  // our plane 1 -> its plane npb + 1
  }
  if (above >= 0) to_above = remote_addr(base, above) - uint32_t(8 * np * area);  // our plane np -> its plane 0
  __syncwarp();
  cluster_arrive();  // every CTA's buffers are loaded before the first remote store
  cluster_wait();
  const long long per_sweep = (long long)ctas * kClWarps;
  double* partial = A.partial + cta * kClWarps + (tid >> 5);
  for (int s = 0; s < A.m; ++s) {
    const double* cur = cl_smem + (s & 1) * buf;
    double* nxt = cl_smem + (1 - (s & 1)) * buf;
    const uint32_t nbuf = uint32_t(8 * (1 - (s & 1)) * buf);
    double r2 = 0.0;
#pragma unroll
    for (int q = 0; q < NPT; ++q) {
      const int o = off[q];
      if (o < 0) continue;
      const double u = cur[o];
      const double sx = cur[o + 1] + cur[o - 1], sy = cur[o + nxp] + cur[o - nxp], sz = cur[o + area] + cur[o - area];
      const double res = b[q] - ((sx - 2.0 * u) * A.idx2 + (sy - 2.0 * u) * A.idy2 + (sz - 2.0 * u) * A.idz2);
      r2 += res * res;
      const double v = A.ax * sx + A.ay * sy + A.az * sz - A.af * b[q];
      nxt[o] = v;
      const bool bottom = o < 2 * area, top = o >= np * area;
      if (bottom && below >= 0) store_remote(to_below + nbuf + uint32_t(8 * o), v);
      if (top && above >= 0) store_remote(to_above + nbuf + uint32_t(8 * o), v);
      if (A.px | A.py) {  // the wrapped copies of this node
        const int r = o % area, j = r / nxp, i = r - j * nxp;
        if (A.px && i == 1) nxt[o + A.nx] = v;
        if (A.px && i == A.nx) nxt[o - A.nx] = v;
        if (A.py && j == 1) nxt[o + A.ny * nxp] = v;
        if (A.py && j == A.ny) nxt[o - A.ny * nxp] = v;
      }
    }
    __syncwarp();
    cluster_arrive();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r2 += __shfl_down_sync(0xffffffffu, r2, o);
    if ((tid & 31) == 0) partial[s * per_sweep] = r2;
    __syncwarp();
    cluster_wait();
  }
  const double* last = cl_smem + (A.m & 1) * buf;
#pragma unroll
  for (int q = 0; q < NPT; ++q) {
    const int e = tid + q * kClThreads;
    if (off[q] < 0) continue;
    const int p = e / interior, r = e - p * interior, j = r / A.nx, i = r - j * A.nx;
    A.Uout[(long long)(i + 1) + (long long)nxp * (j + 1 + (long long)nyp * (k0 + p))] = last[off[q]];
  }
}

using ClusterKernel = void (*)(ClusterArgs);
ClusterKernel cluster_kernel(int npt) {
  return npt <= 1 ? sweeps_cluster_kernel<1> : npt <= 2 ? sweeps_cluster_kernel<2>
         : npt <= 4 ? sweeps_cluster_kernel<4> : sweeps_cluster_kernel<kClMaxNodes>;
}

cudaLaunchConfig_t cluster_config(const ClusterPlan& C, cudaLaunchAttribute* at, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C.ctas);
  cfg.blockDim = dim3(kClThreads);
  cfg.dynamicSmemBytes = C.smem;
  cfg.stream = st;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C.ctas;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

}  // namespace

// The largest cluster (16, 8, 4, 2 CTAs) whose slabs fit shared memory and
// registers and that the device can hold at once; ctas == 0 when none does.
// Smaller clusters would be slower than a launch per sweep, and the rows of a
// plane must be worth a CTA, so grids under 2 planes stay with the launches.
ClusterPlan cluster_plan(const KParams& P) {
  ClusterPlan C;
  const long long area = (long long)(P.nx + 2) * (P.ny + 2);
  for (int ctas = 16; ctas >= 2; ctas /= 2) {
    if (ctas > P.nz) continue;
    const int planes = (P.nz + ctas - 1) / ctas;
    const long long nodes = (long long)planes * P.nx * P.ny, smem = 8LL * 2 * (planes + 2) * area;
    if (nodes > (long long)kClMaxNodes * kClThreads || smem > (long long)kClSmem) return C;
    C.ctas = ctas;
    C.planes = planes;
    C.npt = int((nodes + kClThreads - 1) / kClThreads);
    C.smem = (size_t)smem;
    ClusterKernel k = cluster_kernel(C.npt);
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = cluster_config(C, at, nullptr);
    int fit = 0;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClSmem) == cudaSuccess &&
        (ctas <= 8 || cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
        cudaOccupancyMaxActiveClusters(&fit, k, &cfg) == cudaSuccess && fit > 0)
      return C;
    (void)cudaGetLastError();  // a refusal is an answer here
    C = ClusterPlan();
  }
  return C;
}

int cluster_partials(const ClusterPlan& C) { return C.ctas * kClWarps; }

cudaError_t launch_sweeps_cluster(const KParams& P, const ClusterPlan& C, const double* Uin, double* Uout,
                                  const double* b, double* partial, int m, cudaStream_t st) {
  const JacobiCoef J = jacobi_coef(P);
  ClusterArgs A;
  A.nx = P.nx;
  A.ny = P.ny;
  A.nz = P.nz;
  A.px = !P.xflow;
  A.py = !P.yflow;
  A.pz = !P.zflow;
  A.planes = C.planes;
  A.ax = J.ax;
  A.ay = J.ay;
  A.az = J.az;
  A.af = J.af;
  A.idx2 = 1.0 / J.dx2;
  A.idy2 = 1.0 / J.dy2;
  A.idz2 = 1.0 / J.dz2;
  A.Uin = Uin;
  A.Uout = Uout;
  A.b = b;
  A.partial = partial;
  A.m = m;
  cudaLaunchAttribute at[1];
  cudaLaunchConfig_t cfg = cluster_config(C, at, st);
  note_launch();
  return cudaLaunchKernelEx(&cfg, cluster_kernel(C.npt), A);
}

}  // namespace picard
