// jacobi_cluster.cu -- Jacobi sweeps (CalcEpotential.f90:74-96) of a grid that
// fits the shared memory of one thread-block cluster: in FP64, and on the FP32
// increment (sweeps32_cluster_kernel, further down).
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
// What bounds it: the shared-memory pipe of 16 SMs (71 % busy), their issue slots
// (50 %; FP64 23 %) and the fence and wait of the barrier (the first stall).  32^3 (16
// CTAs, two nodes a thread): 1.33 us per sweep against 4.07 us of kernel time and 3.3
// us of host time for one launch per sweep.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "grid.cuh"
#include "pair_tile.cuh"
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

// ------------------------------------------------ FP32 sweeps of the increment
//
// The same residence for the sweeps of the F32_REFINE solver (open boundaries).
// CTA r is tile layer r of the TMA sweep kernels, four planes.  Half a warp takes a
// row of one 32-wide tile, a lane two x-adjacent nodes in packed FP32 pairs and
// their planes in z order, as pair_tile_sweep_body does: every node has the
// operations of jacobi_res_f32 / jacobi_next_f32, and a tile's partial is summed
// the same way (FP32 down each column, the 32-lane tree, the tile's eight rows in
// order), so the bits are those of every other sweep kernel.  A launch starts from
// w = 0, as every round of sweeps after an anchor does.
//
// What bounds it: the chain of shared-memory loads through four planes (that pipe 59 %
// busy) and the barrier (its wait and fence are the first stalls).
// us per sweep of a 24-sweep round, here and with the tile kernel's launches:
// 16^3 1.45 / 2.0, 24^3 1.65 / 1.95, 32^3 1.74 / 1.96 (with the row sums stored ahead
// of the arrival instead 1.54, 1.71 and 1.85).  A second row pair per half
// warp loses (40 x 36 x 30: 2.7 / 1.95, 48 x 40 x 33: 2.6 / 2.05; with every load
// ahead of the first store 3.4), so at most 64 tile rows per layer are taken here;
// among the grids that qualify the launch tuner decides.
constexpr int kCl32Planes = 4;
constexpr int kCl32Tasks = kClThreads / 16;
// A row's sum of sweep s is stored after its thread's arrival at that sweep's
// barrier, in the barrier's shadow, so only the arrival of sweep s + 1 makes it
// visible: in sweep s, after their own arrival, the summing threads take the rows of
// sweep s - kRowLag.  The slot they read is written again in sweep s - kRowLag +
// kRowSlots, by a thread that has passed the barrier of the sweep before, which the
// summing threads reach only when they have read.
constexpr int kRowLag = 2;
constexpr int kRowSlots = 4;
static_assert(kRowLag >= 2 && kRowSlots >= kRowLag + 2, "a barrier between store and read, and between read and store");

struct Cluster32Args {
  Stencil S;
  JacobiCoefF J;
  const float* r;
  float* wout;
  double* partial;  // [m][nblocks]
  int m, gx, gy, nblocks;
};

__device__ __forceinline__ void store_remote(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void store_remote(uint32_t addr, unsigned long long v) {
  asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}

// Row pitch (floats): node i at column i + 1, so that a lane's pair (odd i, i + 1)
// starts on 8 bytes; columns up to nx + 3 are read.
__host__ __device__ inline int cluster32_pitch(int nx) { return (nx + 5) & ~1; }

__global__ void __launch_bounds__(kClThreads, 1) sweeps32_cluster_kernel(Cluster32Args A) {
  constexpr int ZC = kCl32Planes;
  // row sums [kRowSlots][tasks], then w [2][ZC + 2][ny + 2][pitch] in floats
  extern __shared__ double cl32_smem[];
  using pair = unsigned long long;
  const Stencil& S = A.S;
  const int cta = blockIdx.x, ctas = gridDim.x, lane = threadIdx.x & 31;
  const int pitch = cluster32_pitch(S.nx), area = pitch * (S.ny + 2), tasks = A.gx * S.ny;
  const int z0 = cta * ZC, kend = min(ZC, S.nz - z0);
  double* rows = cl32_smem;
  float* w0 = reinterpret_cast<float*>(cl32_smem + kRowSlots * tasks);
  const int buf = (ZC + 2) * area;
  for (int e = threadIdx.x; e < 2 * buf; e += kClThreads) w0[e] = 0.0f;  // ghosts and the increment itself
  // this lane's pair: which of its two nodes exist, and r
  const int task = threadIdx.x >> 4, j = task / A.gx + 1, i0 = (task % A.gx) * 32 + 2 * (lane & 15) + 1;
  const bool a0 = task < tasks && i0 <= S.nx, both = a0 && i0 < S.nx;
  const int off = j * pitch + i0 + 1;
  pair r[ZC];
#pragma unroll
  for (int kk = 0; kk < ZC; ++kk) {
    const float* p = A.r + fidx(S, i0, j, z0 + 1 + kk);
    r[kk] = pk2(a0 && kk < kend ? p[0] : 0.0f, both && kk < kend ? p[1] : 0.0f);
  }
  const uint32_t base = smem_addr(w0);
  uint32_t to_below = 0, to_above = 0;  // our plane 1 -> the halo above its ZC planes; our plane ZC -> plane 0
  if (cta > 0) to_below = remote_addr(base, cta - 1) + uint32_t(4 * (off + (ZC + 1) * area));
  if (cta + 1 < ctas) to_above = remote_addr(base, cta + 1) + uint32_t(4 * off);
  const pair m2 = pk2(-2.0f, -2.0f), ix2 = pk2(A.J.idx2, A.J.idx2), iy2 = pk2(A.J.idy2, A.J.idy2),
             iz2 = pk2(A.J.idz2, A.J.idz2), naf = pk2(-A.J.af, -A.J.af);
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  // a tile's partial of sweep s from its rows, by the last warps (they have the fewest rows)
  auto flush = [&](int s) {
    const int tiles = A.gx * A.gy;
    for (int t = kClThreads - 1 - threadIdx.x; t < tiles; t += kClThreads) {
      const int bx = t % A.gx, by = t / A.gx;
      double v = 0.0;
      for (int w = 0; w < 8; ++w) {
        const int row = by * 8 + w;
        v += row < S.ny ? rows[(s % kRowSlots) * tasks + row * A.gx + bx] : 0.0;
      }
      A.partial[(long long)s * A.nblocks + bx + A.gx * (by + A.gy * cta)] = v;
    }
  };
  for (int s = 0; s < A.m; ++s) {
    const float* c = w0 + (s & 1) * buf + off;
    float* n = w0 + (1 - (s & 1)) * buf + off;
    const uint32_t nbuf = uint32_t(4 * (1 - (s & 1)) * buf);
    pair r2 = 0ull;  // (+0.0f, +0.0f)
    if (a0) {
      pair wm = *reinterpret_cast<const pair*>(c), wc = *reinterpret_cast<const pair*>(c + area);
#pragma unroll
      for (int kk = 0; kk < ZC; ++kk) {
        if (kk < kend) {
          c += area;
          n += area;
          const pair wp = *reinterpret_cast<const pair*>(c + area);
          pair res = r[kk];
          if (s > 0) {
            const pair ym = *reinterpret_cast<const pair*>(c - pitch), yp = *reinterpret_cast<const pair*>(c + pitch);
            const float2 f = up2(wc);
            const pair sx = add2(pk2(f.y, c[2]), pk2(c[-1], f.x)), sy = add2(yp, ym), sz = add2(wp, wm);
            pair lap = mul2(fma2(m2, wc, sx), ix2);
            lap = fma2(fma2(m2, wc, sy), iy2, lap);
            lap = fma2(fma2(m2, wc, sz), iz2, lap);
            res = sub2(res, lap);
          }
          const pair v = fma2(naf, res, wc);
          if (both) {
            *reinterpret_cast<pair*>(n) = v;
            if (kk == 0 && to_below) store_remote(to_below + nbuf, v);
            if (kk == ZC - 1 && to_above) store_remote(to_above + nbuf, v);
          } else {  // the last column of an odd row: its neighbour is a ghost
            const float x = up2(v).x;
            res = pk2(up2(res).x, 0.0f);
            *n = x;
            if (kk == 0 && to_below) store_remote(to_below + nbuf, x);
            if (kk == ZC - 1 && to_above) store_remote(to_above + nbuf, x);
          }
          r2 = fma2(res, res, r2);
          wm = wc;
          wc = wp;
        }
      }
    }
    __syncwarp();
    cluster_arrive();
    if (s >= kRowLag) flush(s - kRowLag);
    // block_sum_store's 32-lane tree on 16 lanes of pairs
    const float2 f = up2(r2);
    double v0 = (double)f.x, v1 = (double)f.y;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      v0 += __shfl_down_sync(0xffffffffu, v0, o);
      v1 += __shfl_down_sync(0xffffffffu, v1, o);
    }
    if ((lane & 15) == 0 && task < tasks) rows[(s % kRowSlots) * tasks + task] = v0 + v1;
    __syncwarp();
    cluster_wait();
  }
  __syncthreads();
  for (int s = max(0, A.m - kRowLag); s < A.m; ++s) flush(s);
  if (!a0) return;
  const float* last = w0 + (A.m & 1) * buf + off;
  for (int kk = 0; kk < kend; ++kk) {
    float* out = A.wout + fidx(S, i0, j, z0 + 1 + kk);
    const float* v = last + (kk + 1) * area;
    out[0] = v[0];
    if (both) out[1] = v[1];
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

// The FP32 sweeps: one CTA per tile layer (2 .. 16 of four planes), a half warp
// per tile row of it.
ClusterPlan cluster32_plan(const KParams& P, const JacobiGeom& G) {
  ClusterPlan C;
  const int ctas = (int)G.grid.z, tasks = (int)G.grid.x * P.ny;
  if (!G.tma || G.zc != kCl32Planes || ctas < 2 || ctas > 16 || tasks > kCl32Tasks) return C;
  C.ctas = ctas;
  C.planes = kCl32Planes;
  C.smem = sizeof(double) * kRowSlots * (size_t)tasks + 8 * (size_t)(kCl32Planes + 2) * cluster32_pitch(P.nx) * (P.ny + 2);
  static_assert(8 * kRowSlots * kCl32Tasks + 8 * (kCl32Planes + 2) * 68 * (kCl32Tasks + 2) <= kClSmem, "at most 64 x 64 nodes");
  auto k = sweeps32_cluster_kernel;
  cudaLaunchAttribute at[1];
  const cudaLaunchConfig_t cfg = cluster_config(C, at, nullptr);
  int fit = 0;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClSmem) == cudaSuccess &&
      (ctas <= 8 || cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
      cudaOccupancyMaxActiveClusters(&fit, k, &cfg) == cudaSuccess && fit > 0)
    return C;
  (void)cudaGetLastError();
  return ClusterPlan();
}

cudaError_t launch_sweeps32_cluster(const KParams& P, const JacobiGeom& G, const ClusterPlan& C, const float* r,
                                    float* wout, double* partial, int m, cudaStream_t st) {
  Cluster32Args A;
  A.S = make_stencil(P);
  A.J = jacobi_coef_f(P);
  A.r = r;
  A.wout = wout;
  A.partial = partial;
  A.m = m;
  A.gx = (int)G.grid.x;
  A.gy = (int)G.grid.y;
  A.nblocks = G.nblocks;
  cudaLaunchAttribute at[1];
  cudaLaunchConfig_t cfg = cluster_config(C, at, st);
  note_launch();
  return cudaLaunchKernelEx(&cfg, sweeps32_cluster_kernel, A);
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
