// grid.cu -- node-array kernels: deposit finalisation, open-boundary
// potentials, Jacobi sweeps, E-field, field energy.
//
// Jacobi.  CalcEpotential.f90:58-96 runs pure Jacobi from U = 0 (inside) and
// stops at the top of sweep ss when ||b - L U_{ss-1}|| <= maxerr ||b||.  The
// update is U_new = U - af (b - L U)... written as
// U_new = ax(U+x + U-x) + ay(..) + az(..) - af b, so one read of the 7-point
// stencil of U_{s-1} gives both U_s and the residual of U_{s-1}.  Each sweep
// kernel therefore writes U_s and the block partial sums of |res(U_{s-1})|^2;
// a check kernel after every batch of sweeps reduces the partials of each
// sweep in a fixed order (deterministic) and finds the first iterate that
// meets the reference's stopping test.  The batch starts from an anchor
// (a snapshot of the iterate), so the iterate the test selects is rebuilt by
// replaying the sweeps from the anchor.
//
// F32_REFINE keeps the iterate as U = V + sigma * w: V in FP64 (the anchor),
// w in FP32.  The FP32 sweeps advance w with the scaled anchor residual
// r = (b - L V) / sigma, which gives the same Jacobi iterate sequence because
// the update is linear; the anchor pass folds w into V in FP64 and recomputes
// r and its FP64 norm (the exact stopping test of the anchor iterate).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>

#include "chain.cuh"
#include "common.cuh"
#include "grid.cuh"
#include "stencil.cuh"
#include "pair_tile.cuh"
#include "tile32.cuh"

namespace picard {

namespace {

constexpr int kThreads = 256;

inline int grid_for(long long n, int threads = kThreads) {
  long long b = (n + threads - 1) / threads;
  return b < 1 ? 1 : int(b);
}

// --------------------------------------------------------- deposit finish

// Ghost node -> interior node whose deposit it mirrors (-1: open-face ghost,
// which the reference folds and zeroes).
__device__ inline int mirror(int i, int n, int open) {
  if (i >= 1 && i <= n) return i;
  if (open) return -1;
  return i < 1 ? i + n : i - n;
}

// n zero words of 8 bytes (p 16-byte aligned), in the chain: a copy-engine memset
// of a small array costs some 5 us between kernels, this 1.
__global__ void __launch_bounds__(kThreads) zero_kernel(unsigned long long* p, long long n) {
  chain_begin();
  const long long stride = (long long)gridDim.x * blockDim.x, first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  for (long long q = first; q < n >> 1; q += stride) reinterpret_cast<ulonglong2*>(p)[q] = ulonglong2{0ull, 0ull};
  if (first == 0 && (n & 1)) p[n - 1] = 0ull;
}

// N_s = n2p_s * acc * 2^-40 at every node (ParticlesGridify.f90:98-121 with the
// folds of 149-278), C = sum_s q_s N_s (288-293).
__global__ void finish_deposit_kernel(KParams P, const unsigned long long* Nacc, double* N, double* Cout) {
  chain_begin();
  long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= P.nodes) return;
  int i = int(g % P.nxp), j = int((g / P.nxp) % P.nyp), k = int(g / ((long long)P.nxp * P.nyp));
  int mi = mirror(i, P.nx, P.xflow), mj = mirror(j, P.ny, P.yflow), mk = mirror(k, P.nz, P.zflow);
  double c = 0.0;
  for (int s = 0; s < P.species; ++s) {
    double v = 0.0;
    if (mi >= 0 && mj >= 0 && mk >= 0) {
      long long acc = (long long)Nacc[(long long)s * P.nodes + node_index(P, mi, mj, mk)];
      v = P.n2p[s] * ((double)acc * (1.0 / kDepositScale));
    }
    N[(long long)s * P.nodes + g] = v;
    c = c + v * P.charge[s];
  }
  Cout[g] = c;
}

__global__ void finish_flux_kernel(KParams P, const unsigned long long* Facc, double* F) {
  long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= P.nodes) return;
  int i = int(g % P.nxp), j = int((g / P.nxp) % P.nyp), k = int(g / ((long long)P.nxp * P.nyp));
  int mi = mirror(i, P.nx, P.xflow), mj = mirror(j, P.ny, P.yflow), mk = mirror(k, P.nz, P.zflow);
  for (int sc = 0; sc < 3 * P.species; ++sc) {
    int s = sc / 3;
    double v = 0.0;
    if (mi >= 0 && mj >= 0 && mk >= 0) {
      long long acc = (long long)Facc[(long long)sc * P.nodes + node_index(P, mi, mj, mk)];
      v = P.n2p[s] * ((double)acc * (1.0 / kFluxScale));
    }
    F[(long long)sc * P.nodes + g] = v;
  }
}

// ------------------------------------------------------ BCpotentials (a9)

// BCpotentials.f90:51-139 on one rank.  One block computes a 16 x 16 tile of
// face nodes (p1, p2) for both faces of one axis; it walks the interior cells
// plane by plane along the face normal in 16 x 16 in-plane tiles, staging the
// charge tile and the two 31 x 31 windows of the inverse-distance table D in
// shared memory.
constexpr int kBT = 16;

struct FaceGeom {
  int axis;         // normal axis
  int n1, n2, nn;   // in-plane extents (p1 fastest) and normal extent
};

__device__ inline long long dindex(const KParams& P, int a, int b, int c) {
  // 1-based D(a, b, c) of a (2Nx+1, 2Ny+1, 2Nz+1) array
  long long DX = 2LL * P.nx + 1, DY = 2LL * P.ny + 1;
  return (long long)(a - 1) + DX * ((long long)(b - 1) + DY * (long long)(c - 1));
}

// blockIdx.z takes the planes [z per, z per + per): on small faces the planes
// are split over blocks, or a 32 x 32 face would keep 4 of the 148 SMs busy
// (2.7 ms a call at 32^3).  The blocks' sums go to partial[z][face][p2][p1] and
// are added in plane order by bc_direct_sum_kernel.
__global__ void bc_potentials_kernel(KParams P, int axis, int per, const double* __restrict__ C,
                                     const double* __restrict__ D, double* __restrict__ partial) {
  __shared__ double cs[kBT][kBT];
  __shared__ double d0[2 * kBT][2 * kBT + 1];
  __shared__ double d1[2 * kBT][2 * kBT + 1];
  const int Nx = P.nx, Ny = P.ny, Nz = P.nz;
  // in-plane axes (a1 fastest), normal axis
  int n1, n2, nn;
  if (axis == 0) n1 = Ny, n2 = Nz, nn = Nx;
  else if (axis == 1) n1 = Nx, n2 = Nz, nn = Ny;
  else n1 = Nx, n2 = Ny, nn = Nz;
  const int tx = threadIdx.x, ty = threadIdx.y;  // tx along p1, ty along p2
  const int p1 = blockIdx.x * kBT + tx + 1, p2 = blockIdx.y * kBT + ty + 1;  // 1-based face node
  double acc0 = 0.0, acc1 = 0.0;
  const int N1 = n1, N2 = n2;
  const int q_lo = blockIdx.z * per + 1, q_hi = min(nn, q_lo + per - 1);
  for (int q = q_lo; q <= q_hi; ++q) {
    for (int t2 = 0; t2 < (N2 + kBT - 1) / kBT; ++t2)
      for (int t1 = 0; t1 < (N1 + kBT - 1) / kBT; ++t1) {
        // charge tile: cells (q1, q2) = (t1*16 + tx + 1, t2*16 + ty + 1)
        int q1 = t1 * kBT + tx + 1, q2 = t2 * kBT + ty + 1;
        double cv = 0.0;
        if (q1 <= N1 && q2 <= N2) {
          int ci, cj, ck;
          if (axis == 0) ci = q, cj = q1, ck = q2;
          else if (axis == 1) ci = q1, cj = q, ck = q2;
          else ci = q1, cj = q2, ck = q;
          cv = C[node_index(P, ci, cj, ck)];
        }
        cs[ty][tx] = cv;
        // D windows: offsets o1 = q1 - p1 in [t1*16 - b1*16 - 15, ... + 15]
        int base1 = t1 * kBT - blockIdx.x * kBT - (kBT - 1);
        int base2 = t2 * kBT - blockIdx.y * kBT - (kBT - 1);
        // normal offsets of the two faces: face 0 at node 1 -> offset q;
        // face 1 at node N+2 -> offset q - (N + 1)
        int on0 = q, on1 = q - (nn + 1);
        for (int e = ty * kBT + tx; e < (2 * kBT) * (2 * kBT); e += kBT * kBT) {
          int w1 = e % (2 * kBT), w2 = e / (2 * kBT);
          int o1 = base1 + w1, o2 = base2 + w2;
          double v0 = 0.0, v1 = 0.0;
          if (o1 >= -(N1 - 1) && o1 <= N1 - 1 && o2 >= -(N2 - 1) && o2 <= N2 - 1) {
            int a0, b0, c0, a1, b1, c1;
            if (axis == 0) {
              a0 = Nx + 1 + on0; b0 = Ny + 1 + o1; c0 = Nz + 1 + o2;
              a1 = Nx + 1 + on1; b1 = b0; c1 = c0;
            } else if (axis == 1) {
              a0 = Nx + 1 + o1; b0 = Ny + 1 + on0; c0 = Nz + 1 + o2;
              a1 = a0; b1 = Ny + 1 + on1; c1 = c0;
            } else {
              a0 = Nx + 1 + o1; b0 = Ny + 1 + o2; c0 = Nz + 1 + on0;
              a1 = a0; b1 = b0; c1 = Nz + 1 + on1;
            }
            v0 = D[dindex(P, a0, b0, c0)];
            v1 = D[dindex(P, a1, b1, c1)];
          }
          d0[w2][w1] = v0;
          d1[w2][w1] = v1;
        }
        __syncthreads();
        // thread (tx, ty) owns face node (p1, p2): offset of cell (u1, u2) of
        // the tile is (t1*16 + u1 + 1 - p1, ...) -> window index u1 - tx + 15
#pragma unroll 4
        for (int u2 = 0; u2 < kBT; ++u2)
#pragma unroll
          for (int u1 = 0; u1 < kBT; ++u1) {
            double c = cs[u2][u1];
            acc0 += c * d0[u2 - ty + kBT - 1][u1 - tx + kBT - 1];
            acc1 += c * d1[u2 - ty + kBT - 1][u1 - tx + kBT - 1];
          }
        __syncthreads();
      }
  }
  if (p1 <= N1 && p2 <= N2) {
    const long long face = (long long)N1 * N2, at = (long long)(p2 - 1) * N1 + (p1 - 1);
    partial[(2LL * blockIdx.z) * face + at] = acc0;
    partial[(2LL * blockIdx.z + 1) * face + at] = acc1;
  }
}

// U on the two faces normal to `axis`: the partial sums in plane order.
__global__ void bc_direct_sum_kernel(KParams P, int axis, int groups, const double* __restrict__ partial, double* U) {
  const int Nx = P.nx, Ny = P.ny, Nz = P.nz;
  const int N1 = axis == 0 ? Ny : Nx, N2 = axis == 2 ? Ny : Nz;
  const long long face = (long long)N1 * N2, t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= face) return;
  const int p1 = int(t % N1) + 1, p2 = int(t / N1) + 1;
  double a0 = 0.0, a1 = 0.0;
#pragma unroll 8
  for (int g = 0; g < groups; ++g) {
    a0 += partial[2LL * g * face + t];
    a1 += partial[(2LL * g + 1) * face + t];
  }
  const double scale = 1.0 / (2.0 * kTau * kEps0);
  long long g0, g1;
  if (axis == 0) {
    g0 = node_index(P, 0, p1, p2);
    g1 = node_index(P, Nx + 1, p1, p2);
  } else if (axis == 1) {
    g0 = node_index(P, p1, 0, p2);
    g1 = node_index(P, p1, Ny + 1, p2);
  } else {
    g0 = node_index(P, p1, p2, 0);
    g1 = node_index(P, p1, p2, Nz + 1);
  }
  U[g0] = a0 * scale;
  U[g1] = a1 * scale;
}

// Plane groups of one axis: about four blocks of 256 threads per SM, and no more
// than `room` doubles of partial sums hold (one group always fits a node array).
struct DirectSplit {
  int n1, n2, nn, bx, by, per, groups;
};
inline DirectSplit direct_split(const KParams& P, int axis, long long room) {
  DirectSplit S;
  S.n1 = axis == 0 ? P.ny : P.nx;
  S.n2 = axis == 2 ? P.ny : P.nz;
  S.nn = axis == 0 ? P.nx : axis == 1 ? P.ny : P.nz;
  S.bx = (S.n1 + kBT - 1) / kBT;
  S.by = (S.n2 + kBT - 1) / kBT;
  const long long want =
      std::max<long long>(1, std::min({148LL * 4 / ((long long)S.bx * S.by), (long long)S.nn, room / (2LL * S.n1 * S.n2)}));
  S.per = int((S.nn + want - 1) / want);
  S.groups = (S.nn + S.per - 1) / S.per;
  return S;
}

// ------------------------------------------------------------- Jacobi

__device__ inline void neighbours(const Stencil& S, int i, int j, int k, long long& xm, long long& xp, long long& ym,
                                  long long& yp, long long& zm, long long& zp) {
  int im = (S.px && i == 1) ? S.nx : i - 1, ip = (S.px && i == S.nx) ? 1 : i + 1;
  int jm = (S.py && j == 1) ? S.ny : j - 1, jp = (S.py && j == S.ny) ? 1 : j + 1;
  int km = (S.pz && k == 1) ? S.nz : k - 1, kp = (S.pz && k == S.nz) ? 1 : k + 1;
  long long row = (long long)S.nxp * ((long long)j + (long long)S.nyp * k);
  xm = row + im;
  xp = row + ip;
  ym = (long long)i + (long long)S.nxp * ((long long)jm + (long long)S.nyp * k);
  yp = (long long)i + (long long)S.nxp * ((long long)jp + (long long)S.nyp * k);
  zm = (long long)i + (long long)S.nxp * ((long long)j + (long long)S.nyp * km);
  zp = (long long)i + (long long)S.nxp * ((long long)j + (long long)S.nyp * kp);
}

// b = -C / (dV eps0) everywhere; block partials of b^2 over the interior.
__global__ void rhs_kernel(KParams P, const double* C, double* b, double* partial) {
  long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double v2 = 0.0;
  if (g < P.nodes) {
    double binv = 1.0 / (P.dV * kEps0);
    double v = -C[g] * binv;
    b[g] = v;
    int i = int(g % P.nxp), j = int((g / P.nxp) % P.nyp), k = int(g / ((long long)P.nxp * P.nyp));
    if (i >= 1 && i <= P.nx && j >= 1 && j <= P.ny && k >= 1 && k <= P.nz) v2 = v * v;
  }
  __shared__ double sh[32];
  for (int o = 16; o > 0; o >>= 1) v2 += __shfl_down_sync(0xffffffffu, v2, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v2;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < int(blockDim.x >> 5); ++w) s += sh[w];
    partial[blockIdx.x] = s;
  }
}

// FP64 sweep: Uout = Jacobi(Uin); partial = sum |b - L Uin|^2 of this block.
__global__ void __launch_bounds__(256) sweep_f64_kernel(Stencil S, JacobiCoef J, const double* __restrict__ Uin,
                                                        double* __restrict__ Uout, const double* __restrict__ b,
                                                        double* partial, int zc) {
  int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  int k0 = blockIdx.z * zc + 1;
  double r2 = 0.0;
  if (i <= S.nx && j <= S.ny) {
    int k1 = min(k0 + zc - 1, S.nz);
    for (int k = k0; k <= k1; ++k) {
      long long c = (long long)i + (long long)S.nxp * ((long long)j + (long long)S.nyp * k);
      long long xm, xp, ym, yp, zm, zp;
      neighbours(S, i, j, k, xm, xp, ym, yp, zm, zp);
      double u = Uin[c];
      double sx = Uin[xp] + Uin[xm], sy = Uin[yp] + Uin[ym], sz = Uin[zp] + Uin[zm];
      double bc = b[c];
      double res = bc - ((sx - 2.0 * u) / J.dx2 + (sy - 2.0 * u) / J.dy2 + (sz - 2.0 * u) / J.dz2);
      r2 += res * res;
      Uout[c] = J.ax * sx + J.ay * sy + J.az * sz - J.af * bc;
    }
  }
  block_sum_store(r2, partial + (blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)));
}

// FP32 sweep of the increment: res = r - L w, w_out = w - af res.
// w_zero: the input increment is zero (first sweep after an anchor).
__global__ void __launch_bounds__(256) sweep_f32_kernel(Stencil S, JacobiCoefF J, const float* __restrict__ win,
                                                        float* __restrict__ wout, const float* __restrict__ r,
                                                        double* partial, int zc, int w_zero) {
  int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  int k0 = blockIdx.z * zc + 1;
  float r2 = 0.0f;
  if (i <= S.nx && j <= S.ny) {
    int k1 = min(k0 + zc - 1, S.nz);
    long long plane = (long long)S.fpitch * S.nyp;
    long long c = fidx(S, i, j, k0);
    if (w_zero) {
      for (int k = k0; k <= k1; ++k, c += plane) {
        float res = __ldg(r + c);
        r2 = acc_r2_f32(r2, res);
        wout[c] = jacobi_next_f32(J, 0.0f, res);
      }
    } else {
      int im = (S.px && i == 1) ? S.nx : i - 1, ip = (S.px && i == S.nx) ? 1 : i + 1;
      int jm = (S.py && j == 1) ? S.ny : j - 1, jp = (S.py && j == S.ny) ? 1 : j + 1;
      long long dxm = im - i, dxp = ip - i;
      long long dym = (long long)(jm - j) * S.fpitch, dyp = (long long)(jp - j) * S.fpitch;
      // z pipeline in registers
      long long cm = (S.pz && k0 == 1) ? c + (long long)(S.nz - 1) * plane : c - plane;
      float wm = __ldg(win + cm);
      float wc = __ldg(win + c);
      for (int k = k0; k <= k1; ++k, c += plane) {
        long long cp = (S.pz && k == S.nz) ? c - (long long)(S.nz - 1) * plane : c + plane;
        float wp = __ldg(win + cp);
        float res = jacobi_res_f32(J, wc, __ldg(win + c + dxm), __ldg(win + c + dxp), __ldg(win + c + dym),
                                   __ldg(win + c + dyp), wm, wp, __ldg(r + c));
        r2 = acc_r2_f32(r2, res);
        wout[c] = jacobi_next_f32(J, wc, res);
        wm = wc;
        wc = wp;
      }
    }
  }
  block_sum_store((double)r2, partial + (blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)));
}

// Anchor of F32_REFINE: Vout = Vin + sigma w (interior), r = (b - L Vout)/sigma
// as FP32, partial = sum (b - L Vout)^2 in FP64.
__global__ void __launch_bounds__(256) anchor_kernel(Stencil S, JacobiCoef J, const double* __restrict__ Vin,
                                                     double* __restrict__ Vout, const float* __restrict__ w,
                                                     const double* __restrict__ b, float* __restrict__ r,
                                                     double sigma, double* partial, int zc, int w_zero) {
  int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  int k0 = blockIdx.z * zc + 1;
  double r2 = 0.0;
  if (i <= S.nx && j <= S.ny) {
    int k1 = min(k0 + zc - 1, S.nz);
    const int im = (S.px && i == 1) ? S.nx : i - 1, ip = (S.px && i == S.nx) ? 1 : i + 1;
    const int jm = (S.py && j == 1) ? S.ny : j - 1, jp = (S.py && j == S.ny) ? 1 : j + 1;
    for (int k = k0; k <= k1; ++k) {
      const int km = (S.pz && k == 1) ? S.nz : k - 1, kp = (S.pz && k == S.nz) ? 1 : k + 1;
      // U = V + sigma w at node (ii, jj, kk): the FP64 array is (nxp, nyp, ..), the
      // FP32 one has rows of fpitch with node ii at column ii + 3
      auto val = [&](int ii, int jj, int kk) {
        const long long rest = (long long)jj + (long long)S.nyp * kk;
        const long long g = (long long)ii + (long long)S.nxp * rest;
        return w_zero ? Vin[g] : Vin[g] + sigma * (double)w[(long long)(ii + 3) + (long long)S.fpitch * rest];
      };
      const long long c = (long long)i + (long long)S.nxp * ((long long)j + (long long)S.nyp * k);
      double u = val(i, j, k);
      double sx = val(ip, j, k) + val(im, j, k), sy = val(i, jp, k) + val(i, jm, k),
             sz = val(i, j, kp) + val(i, j, km);
      double bc = b[c];
      double res = bc - ((sx - 2.0 * u) / J.dx2 + (sy - 2.0 * u) / J.dy2 + (sz - 2.0 * u) / J.dz2);
      r2 += res * res;
      Vout[c] = u;
      r[fidx(S, i, j, k)] = (float)(res / sigma);
    }
  }
  block_sum_store(r2, partial + (blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)));
}

// U = V + sigma w on the interior.
__global__ void finalize_kernel(Stencil S, const double* V, const float* w, double sigma, double* U, int w_zero) {
  long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= S.nodes) return;
  int i = int(g % S.nxp), j = int((g / S.nxp) % S.nyp), k = int(g / ((long long)S.nxp * S.nyp));
  bool interior = i >= 1 && i <= S.nx && j >= 1 && j <= S.ny && k >= 1 && k <= S.nz;
  U[g] = (interior && !w_zero) ? V[g] + sigma * (double)w[fidx(S, i, j, k)] : V[g];
}

// ------------------------------------------------- TMA-staged FP32 sweep

// The interior is cut into 32 x 8 x ZC columns of nodes ("tiles", x fastest).
// A CTA walks the tiles t = blockIdx.x, + gridDim.x, ... through a two-stage
// shared-memory pipeline: while it sweeps tile t from one stage, the TMA
// engine fills the other stage with tile t + gridDim.x.  Per tile one elected
// thread issues two TMA tile loads completing on the stage's mbarrier -- the
// increment w with a one-node halo (box 40 x 10 x (ZC+2) from the 16-byte
// aligned column 32 bx) and the scaled residual r (box 32 x 8 x ZC from the
// tile's first interior column, 32 bx + 4, also 16-byte aligned) -- and
// the block then sweeps the column plane by plane from shared memory and
// writes w' with coalesced stores.  Open axes only: the ghost layer of w is
// zero, which the box supplies (and TMA zero-fills outside the array).
//
// The grid size (a multiple of the SM count, or one CTA per tile) and the
// number of stages (1: the next tile is loaded after the current one is
// consumed) are tuning knobs: each node's update and each tile's partial sum
// of squared residuals are computed the same way whatever they are, so results
// do not depend on them.
//
// Launched with programmatic dependent launch: the CTAs of sweep s+1 are
// scheduled while sweep s drains and block in griddepcontrol.wait -- which
// returns once sweep s has completed and its stores are visible -- before
// their first load.
//
// Waits are bounded: when a stage's copies do not land within the limit the
// block (deciding together, so that no thread is left at a barrier) records
// kDevTimeout in *err, waits (bounded) for the copies it has in flight and
// returns.
constexpr int kTmaTx = 32, kTmaTy = 8, kTmaBoxX = 40;
constexpr long long kMbarSpin = 1LL << 24;

__device__ inline bool mbar_wait(uint32_t mbar, uint32_t phase, long long limit) {
  for (long long it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(mbar), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}

template <int ZC>
struct TmaStage {
  static constexpr int kW = (ZC + 2) * (kTmaTy + 2) * kTmaBoxX;  // floats of the w box
  static constexpr int kR = ZC * kTmaTy * kTmaTx;                // floats of the r box
  static constexpr int kFloats = kW + kR;
  static constexpr size_t kBytes = sizeof(float) * kFloats;
  static_assert(kBytes % 128 == 0, "stage buffers stay 128-byte aligned");
};

template <int ZC>
__device__ inline void tma_issue_tile(const CUtensorMap* tw, const CUtensorMap* tr, float* stage, uint32_t mb, int t,
                                      int gx, int gy, int w_zero) {
  const int bx = t % gx, by = (t / gx) % gy, bz = t / (gx * gy);
  const int x0 = bx * kTmaTx, y0 = by * kTmaTy, z0 = bz * ZC;
  float* sw = stage;
  float* sr = stage + TmaStage<ZC>::kW;
  uint32_t bytes = (uint32_t)(TmaStage<ZC>::kR * sizeof(float));
  if (!w_zero) bytes += (uint32_t)(TmaStage<ZC>::kW * sizeof(float));
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(bytes) : "memory");
  if (!w_zero)
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"((uint32_t)__cvta_generic_to_shared(sw)), "l"((unsigned long long)tw), "r"(x0), "r"(y0), "r"(z0), "r"(mb)
        : "memory");
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"((uint32_t)__cvta_generic_to_shared(sr)), "l"((unsigned long long)tr), "r"(x0 + 4), "r"(y0 + 1), "r"(z0 + 1),
      "r"(mb)
      : "memory");
}

template <int ZC, int STAGES>
__global__ void __launch_bounds__(256) sweep_tma_kernel(const __grid_constant__ CUtensorMap tw,
                                                        const __grid_constant__ CUtensorMap tr, Stencil S,
                                                        JacobiCoefF J, float* __restrict__ wout, double* partial,
                                                        int w_zero, int gx, int gy, int ntiles, int* err) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float* stages = reinterpret_cast<float*>(smem_raw);  // [STAGES][TmaStage<ZC>::kFloats]
  __shared__ __align__(8) unsigned long long mbar[2];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int tid = tx + kTmaTx * ty;
  const uint32_t mb0 = (uint32_t)__cvta_generic_to_shared(&mbar[0]);
  const uint32_t mb1 = (uint32_t)__cvta_generic_to_shared(&mbar[1]);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb0) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&tw) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&tr) : "memory");
  }
  __syncthreads();
  // the previous sweep wrote the w this one reads: wait for it, then let the
  // next sweep's CTAs be scheduled as this grid's CTAs retire
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  int t = blockIdx.x;
  if (t >= ntiles) return;
  if (tid == 0) tma_issue_tile<ZC>(&tw, &tr, stages, mb0, t, gx, gy, w_zero);
  for (int it = 0; t < ntiles; t += gridDim.x, ++it) {
    const int st = STAGES == 2 ? (it & 1) : 0;
    const uint32_t phase = (uint32_t)(STAGES == 2 ? ((it >> 1) & 1) : (it & 1));
    const uint32_t mb = st ? mb1 : mb0;
    const int tn = t + gridDim.x;
    // two stages: prefetch the next tile into the other stage, which was last
    // read in iteration it-1 (ended at a barrier)
    if (STAGES == 2 && tid == 0 && tn < ntiles)
      tma_issue_tile<ZC>(&tw, &tr, stages + (st ^ 1) * TmaStage<ZC>::kFloats, st ? mb0 : mb1, tn, gx, gy, w_zero);
    // tile coordinates before the wait: the divisions overlap the copies
    const int bx = t % gx, by = (t / gx) % gy, bz = t / (gx * gy);
    const bool ok = __syncthreads_and(mbar_wait(mb, phase, kMbarSpin) ? 1 : 0);
    if (!ok) {
      if (tid == 0) atomicCAS(err, 0, int(kDevTimeout));
      // let the copies in flight land before the block exits
      mbar_wait(mb, phase, kMbarSpin);
      if (STAGES == 2 && tn < ntiles) mbar_wait(st ? mb0 : mb1, (uint32_t)(((it + 1) >> 1) & 1), kMbarSpin);
      return;
    }
    const float* sw = stages + st * TmaStage<ZC>::kFloats;
    tile32_sweep<ZC>(sw, sw + TmaStage<ZC>::kW, S, J, wout, partial + t, w_zero, bx, by, bz);
    // every thread is done with this stage (and thread 0 with the reduction
    // scratch) before the stage is refilled
    __syncthreads();
    if (STAGES == 1 && tid == 0 && tn < ntiles) tma_issue_tile<ZC>(&tw, &tr, stages, mb0, tn, gx, gy, w_zero);
  }
}

// ------------------------------------------- TMA-staged FP32 sweep, x pairs
//
// The same sweep over tiles twice as wide: 64 (x) x 8 (y) x ZC (z) nodes per
// tile, 32 x 8 threads, each thread updating the two x-adjacent nodes 2 tx and
// 2 tx + 1 of its row with packed FP32 pair arithmetic (add/sub/mul/fma
// .rn.f32x2, each lane rounded like the scalar __fadd_rn/.../__fmaf_rn of
// jacobi_res_f32) and 8-byte shared-memory loads and global stores, the z
// loop fully unrolled.  The x neighbours outside the pair come from the
// adjacent lanes by shuffle (the tile's outer columns from shared memory).
// Boxes: w 72 x 10 x (ZC+2) from the aligned column 64 bx, r 64 x 8 x ZC from
// the tile's first interior column 64 bx + 4.
//
// Each 64-wide tile is two of the 32 x 8 x ZC tiles the residual partials
// are defined on (lanes 0-15 and 16-31).  Their per-column FP32 sums over z
// are formed node by node as in sweep_tma_kernel, and the 32-lane shuffle
// tree of block_sum_store is reproduced exactly: its steps 16, 8, 4, 2 are
// shuffles by 8, 4, 2, 1 of both pair components, its step 1 the in-lane sum
// of the pair.  So the two kernels write the same partials bit for bit.
constexpr int kTma2BoxX = 72, kTma2Tile = 64;

template <int ZC>
struct Tma2Stage {
  static constexpr int kW = (ZC + 2) * (kTmaTy + 2) * kTma2BoxX;
  static constexpr int kR = ZC * kTmaTy * kTma2Tile;
  static constexpr int kFloats = kW + kR;
  static constexpr size_t kBytes = sizeof(float) * kFloats;
  static_assert(kBytes % 128 == 0, "stage buffers stay 128-byte aligned");
};

template <int ZC>
__device__ inline void tma2_issue_tile(const CUtensorMap* tw, const CUtensorMap* tr, float* stage, uint32_t mb, int t,
                                       int gx2, int gy, int w_zero) {
  const int bx = t % gx2, by = (t / gx2) % gy, bz = t / (gx2 * gy);
  const int x0 = bx * kTma2Tile, y0 = by * kTmaTy, z0 = bz * ZC;
  float* sw = stage;
  float* sr = stage + Tma2Stage<ZC>::kW;
  uint32_t bytes = (uint32_t)(Tma2Stage<ZC>::kR * sizeof(float));
  if (!w_zero) bytes += (uint32_t)(Tma2Stage<ZC>::kW * sizeof(float));
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(bytes) : "memory");
  if (!w_zero)
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"((uint32_t)__cvta_generic_to_shared(sw)), "l"((unsigned long long)tw), "r"(x0), "r"(y0), "r"(z0), "r"(mb)
        : "memory");
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"((uint32_t)__cvta_generic_to_shared(sr)), "l"((unsigned long long)tr), "r"(x0 + 4), "r"(y0 + 1),
      "r"(z0 + 1), "r"(mb)
      : "memory");
}

// W_ZERO: the first sweep after an anchor (zero iterate, no w box), a
// separate instantiation so that the common sweep carries no run-time flag.
// LOOP = false: one CTA per tile (the grid covers every tile), without the
// persistent loop: 42 instead of 54 registers, so shared memory, not
// registers, sets the CTAs per SM (7.6 instead of 8.0 us per sweep at
// 256 x 128 x 128).
template <int ZC, int STAGES, bool W_ZERO, bool LOOP>
__global__ void __launch_bounds__(256) sweep_tma2_kernel(const __grid_constant__ CUtensorMap tw,
                                                         const __grid_constant__ CUtensorMap tr, Stencil S,
                                                         JacobiCoefF J, float* __restrict__ wout, double* partial,
                                                         int gx2, int gx, int gy, int ntiles, int* err) {
  constexpr int w_zero = W_ZERO ? 1 : 0;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float* stages = reinterpret_cast<float*>(smem_raw);  // [STAGES][Tma2Stage<ZC>::kFloats]
  __shared__ __align__(8) unsigned long long mbar[2];
  __shared__ double rows[2][kTmaTy];  // row sums of the two 32-wide partial tiles
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int tid = tx + kTmaTx * ty;
  const uint32_t mb0 = (uint32_t)__cvta_generic_to_shared(&mbar[0]);
  const uint32_t mb1 = (uint32_t)__cvta_generic_to_shared(&mbar[1]);
  if (!LOOP) {
    if (tid == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb0) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int t = blockIdx.x;
    if (t >= ntiles) return;
    const int bx2 = t % gx2, by = (t / gx2) % gy, bz = t / (gx2 * gy);
    if (tid == 0) tma2_issue_tile<ZC>(&tw, &tr, stages, mb0, t, gx2, gy, w_zero);
    if (!__syncthreads_and(mbar_wait(mb0, 0, kMbarSpin) ? 1 : 0)) {
      if (tid == 0) atomicCAS(err, 0, int(kDevTimeout));
      mbar_wait(mb0, 0, kMbarSpin);
      return;
    }
    pair_tile_sweep_wz<ZC, W_ZERO>(stages, stages + Tma2Stage<ZC>::kW, S, J, wout, partial, bx2, by, bz, gx, gy,
                                   rows);
    return;
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb0) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&tw) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&tr) : "memory");
  }
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  int t = blockIdx.x;
  if (t >= ntiles) return;
  if (tid == 0) tma2_issue_tile<ZC>(&tw, &tr, stages, mb0, t, gx2, gy, w_zero);
  for (int it = 0; t < ntiles; t += gridDim.x, ++it) {
    const int st = STAGES == 2 ? (it & 1) : 0;
    const uint32_t phase = (uint32_t)(STAGES == 2 ? ((it >> 1) & 1) : (it & 1));
    const uint32_t mb = st ? mb1 : mb0;
    const int tn = t + gridDim.x;
    if (STAGES == 2 && tid == 0 && tn < ntiles)
      tma2_issue_tile<ZC>(&tw, &tr, stages + (st ^ 1) * Tma2Stage<ZC>::kFloats, st ? mb0 : mb1, tn, gx2, gy, w_zero);
    // tile coordinates before the wait: computed after it, the three divisions
    // sat between the copies landing and the sweep and cost ~1.5 us per sweep
    // at 256 x 128 x 128 (9.1 instead of 7.6 us)
    const int bx2 = t % gx2, by = (t / gx2) % gy, bz = t / (gx2 * gy);
    const bool ok = __syncthreads_and(mbar_wait(mb, phase, kMbarSpin) ? 1 : 0);
    if (!ok) {
      if (tid == 0) atomicCAS(err, 0, int(kDevTimeout));
      mbar_wait(mb, phase, kMbarSpin);
      if (STAGES == 2 && tn < ntiles) mbar_wait(st ? mb0 : mb1, (uint32_t)(((it + 1) >> 1) & 1), kMbarSpin);
      return;
    }
    const float* sw = stages + st * Tma2Stage<ZC>::kFloats;
    pair_tile_sweep_wz<ZC, W_ZERO>(sw, sw + Tma2Stage<ZC>::kW, S, J, wout, partial, bx2, by, bz, gx, gy, rows);
    __syncthreads();
    if (STAGES == 1 && tid == 0 && tn < ntiles) tma2_issue_tile<ZC>(&tw, &tr, stages, mb0, tn, gx2, gy, w_zero);
  }
}

// The x-pair sweep with r read from global memory: only the w box goes
// through shared memory (28.8 KB at zc = 8 instead of 45 KB), so more tiles
// are in flight per SM: with 32 registers (the launch bound asks for 7 CTAs
// of 256 threads per SM) 7 tiles fit, so the 1,024 tiles of a 256 x 128 x 128
// sweep run in one wave on 148 SMs.  One CTA per tile, one stage; every node
// and every partial is computed by the same pair_tile body, so the results
// are bit-identical to sweep_tma2_kernel's.
template <int ZC, bool W_ZERO>
__global__ void __launch_bounds__(256, 7) sweep_tma2r_kernel(const __grid_constant__ CUtensorMap tw,
                                                          const float* __restrict__ r, Stencil S, JacobiCoefF J,
                                                          float* __restrict__ wout, double* partial, int gx2, int gx,
                                                          int gy, int ntiles, int* err) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float* sw = reinterpret_cast<float*>(smem_raw);  // [ZC+2][10][72]
  __shared__ __align__(8) unsigned long long mbar[1];
  __shared__ double rows[2][kTmaTy];
  const int tid = threadIdx.x + kTmaTx * threadIdx.y;
  const uint32_t mb0 = (uint32_t)__cvta_generic_to_shared(&mbar[0]);
  if (!W_ZERO && tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb0) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int t = blockIdx.x;
  if (t >= ntiles) return;
  const int bx2 = t % gx2, by = (t / gx2) % gy, bz = t / (gx2 * gy);
  if (!W_ZERO) {
    if (tid == 0) {
      const uint32_t bytes = (uint32_t)(Tma2Stage<ZC>::kW * sizeof(float));
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb0), "r"(bytes) : "memory");
      asm volatile(
          "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
          ::"r"((uint32_t)__cvta_generic_to_shared(sw)), "l"((unsigned long long)&tw), "r"(bx2 * kTma2Tile),
          "r"(by * kTmaTy), "r"(bz * ZC), "r"(mb0)
          : "memory");
    }
    if (!__syncthreads_and(mbar_wait(mb0, 0, kMbarSpin) ? 1 : 0)) {
      if (tid == 0) atomicCAS(err, 0, int(kDevTimeout));
      mbar_wait(mb0, 0, kMbarSpin);
      return;
    }
  }
  pair_tile_sweep_wz<ZC, W_ZERO, true>(sw, nullptr, S, J, wout, partial, bx2, by, bz, gx, gy, rows, r);
}

// ---------------------------------- two sweeps per launch (temporal blocking)
//
// Sweeps s and s+1 of the x-pair kernel in one launch.  Per 64 x 8 x ZC tile
// the CTA loads w_{s-1} with a two-node halo (box 72 x 12 x (ZC+4)) and r with
// a one-node halo (box 72 x 10 x (ZC+2)), computes w_s on the tile and its
// one-node halo (x pairs from tile column -2 to 65, rows -1..8, planes
// -1..ZC) into shared memory -- zero outside the interior, the ghost value --
// and then w_{s+1} on the tile from there.  Every node of either sweep is the
// same jacobi_res_f32 / jacobi_next_f32 arithmetic on the same inputs as in a
// single-sweep launch (halo nodes are recomputed by each neighbouring tile,
// identically), and both sweeps' per-tile partials are formed exactly as in
// sweep_tma2_kernel (per-column FP32 sums in z order, the 32-lane tree, rows
// in order), so results are bit-identical to two single sweeps.  L2 traffic
// per sweep drops from ~15 to ~10.6 bytes per node and launches halve.
//
// RG: r is read from global memory (8-byte pair loads, only where a pair has
// a node inside the domain; the value elsewhere is never used), so only the w
// box is staged: 70.7 KB of shared memory at ZC = 8 instead of 99.5, three
// CTAs per SM instead of two.  The CTA then has 12 rows of 32 threads, so the
// 340 x-pair columns of the first sweep's tile-plus-halo take one pass; the
// second sweep runs on the first 8 rows.  The same arithmetic on the same
// values: the same bits.
template <int ZC, bool RG = false>
struct Sweep2Smem {
  static constexpr int kW0 = (ZC + 4) * 12 * kTma2BoxX;  // w_{s-1}: [ZC+4][12][72]
  static constexpr int kR = RG ? 0 : (ZC + 2) * 10 * kTma2BoxX;  // r: [ZC+2][10][72]
  static constexpr int kW1X = 68;
  static constexpr int kW1 = (ZC + 2) * 10 * kW1X;       // w_s:     [ZC+2][10][68]
  static constexpr int kCS = kTmaTy * kTma2Tile;         // sweep-s column sums [8][64]
  static constexpr size_t kBytes = sizeof(float) * (size_t)(kW0 + kR + kW1 + kCS);
  static_assert((kW0 * 4) % 128 == 0 && ((kW0 + kR) * 4) % 128 == 0, "TMA destinations 128-byte aligned");
};

// 32-lane partial tree of block_sum_store on x-pair column sums (lane l holds
// columns 2l and 2l+1 of a 64-wide row); lanes 0 and 16 return the two
// 32-wide tiles' row sums.
__device__ __forceinline__ double pair_row_tree(float c0, float c1) {
  double v0 = (double)c0, v1 = (double)c1;
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    v0 += __shfl_down_sync(0xffffffffu, v0, o);
    v1 += __shfl_down_sync(0xffffffffu, v1, o);
  }
  return v0 + v1;
}

template <int ZC, bool RG>
__global__ void __launch_bounds__(RG ? 384 : 256, RG ? 3 : 1)
    sweep2_tma_kernel(const __grid_constant__ CUtensorMap tw, const __grid_constant__ CUtensorMap tr,
                      const float* __restrict__ rg, Stencil S, JacobiCoefF J, float* __restrict__ wout,
                      double* partialA, double* partialB, int w_zero, int gx2, int gx, int gy, int ntiles, int* err) {
  using L = Sweep2Smem<ZC, RG>;
  constexpr int kThreads2 = RG ? 384 : 256;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float* W0 = reinterpret_cast<float*>(smem_raw);
  float* R = W0 + L::kW0;
  float* W1 = R + L::kR;
  float* CS = W1 + L::kW1;
  __shared__ __align__(8) unsigned long long mbar;
  __shared__ double rows[2][2][kTmaTy];  // [sweep][32-wide tile][row]
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int tid = tx + kTmaTx * ty;
  const uint32_t mb = (uint32_t)__cvta_generic_to_shared(&mbar);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&tw) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&tr) : "memory");
  }
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int t = blockIdx.x;
  if (t >= ntiles) return;
  const int bx2 = t % gx2, by = (t / gx2) % gy, bz = t / (gx2 * gy);
  const int x0 = bx2 * kTma2Tile, y0 = by * kTmaTy, z0 = bz * ZC;
  // RG with a zero entering iterate: nothing to stage
  const bool staged = !RG || !w_zero;
  if (tid == 0 && staged) {
    uint32_t bytes = (uint32_t)(L::kR * sizeof(float));
    if (!w_zero) bytes += (uint32_t)(L::kW0 * sizeof(float));
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(bytes) : "memory");
    if (!w_zero)
      asm volatile(
          "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
          ::"r"((uint32_t)__cvta_generic_to_shared(W0)), "l"((unsigned long long)&tw), "r"(x0), "r"(y0 - 1),
          "r"(z0 - 1), "r"(mb)
          : "memory");
    if (!RG)
      asm volatile(
          "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
          ::"r"((uint32_t)__cvta_generic_to_shared(R)), "l"((unsigned long long)&tr), "r"(x0), "r"(y0), "r"(z0),
          "r"(mb)
          : "memory");
  }
  if (staged) {
    const bool ok = __syncthreads_and(mbar_wait(mb, 0, kMbarSpin) ? 1 : 0);
    if (!ok) {
      if (tid == 0) atomicCAS(err, 0, int(kDevTimeout));
      mbar_wait(mb, 0, kMbarSpin);
      return;
    }
  }
  const unsigned long long m2 = pk2(-2.0f, -2.0f), ix2 = pk2(J.idx2, J.idx2), iy2 = pk2(J.idy2, J.idy2),
                           iz2 = pk2(J.idz2, J.idz2), naf = pk2(-J.af, -J.af);
  auto node_res = [&](unsigned long long wc, float xl, float xr, unsigned long long ym, unsigned long long yp,
                      unsigned long long wm, unsigned long long wp, unsigned long long rr) {
    const float2 c = up2(wc);
    const unsigned long long xm = pk2(xl, c.x), xp = pk2(c.y, xr);
    const unsigned long long sx = add2(xp, xm), sy = add2(yp, ym), sz = add2(wp, wm);
    unsigned long long lap = mul2(fma2(m2, wc, sx), ix2);
    lap = fma2(fma2(m2, wc, sy), iy2, lap);
    lap = fma2(fma2(m2, wc, sz), iz2, lap);
    return sub2(rr, lap);
  };
  auto u64at = [](const float* base, int idx) { return *reinterpret_cast<const unsigned long long*>(base + idx); };

  // ---- sweep s on the tile and its one-node halo: 34 x-pairs x 10 rows, z marching
  for (int item = tid; item < 34 * 10; item += kThreads2) {
    const int p = item % 34, ry = item / 34;
    const int xr = 2 * p - 2, yr = ry - 1;  // first node of the pair, tile-relative
    const int i0 = x0 + 1 + xr, j = y0 + 1 + yr;
    const bool rowin = j >= 1 && j <= S.ny;
    const bool in0 = rowin && i0 >= 1 && i0 <= S.nx, in1 = rowin && i0 + 1 >= 1 && i0 + 1 <= S.nx;
    const bool tilecol = p >= 1 && p <= 32 && ry >= 1 && ry <= kTmaTy;
    // W0[kz][ky][kx]: kz = zr + 2, ky = yr + 2, kx = xr + 4
    auto w0 = [&](int zr, int dy) { return u64at(W0, ((zr + 2) * 12 + (yr + 2 + dy)) * kTma2BoxX + xr + 4); };
    auto w0s = [&](int zr, int dx) { return W0[((zr + 2) * 12 + (yr + 2)) * kTma2BoxX + xr + 4 + dx]; };
    unsigned long long wm = w_zero ? 0ull : w0(-2, 0);
    unsigned long long wc = w_zero ? 0ull : w0(-1, 0);
    unsigned long long r2 = 0ull;
#pragma unroll
    for (int zr = -1; zr <= ZC; ++zr) {
      const int k = z0 + 1 + zr;
      unsigned long long wp = 0ull, ym = 0ull, yp = 0ull;
      float xl = 0.0f, xrr = 0.0f;
      if (!w_zero) {
        wp = w0(zr + 1, 0);
        ym = w0(zr, -1);
        yp = w0(zr, 1);
        xl = w0s(zr, -1);
        xrr = w0s(zr, 2);
      }
      const bool kin = k >= 1 && k <= S.nz;
      unsigned long long rr;
      if (RG)
        rr = ((in0 || in1) && kin) ? __ldg(reinterpret_cast<const unsigned long long*>(rg + fidx(S, i0, j, k))) : 0ull;
      else
        rr = u64at(R, ((zr + 1) * 10 + (yr + 1)) * kTma2BoxX + xr + 4);
      const unsigned long long res = node_res(wc, xl, xrr, ym, yp, wm, wp, rr);
      const float2 rf = up2(res);
      const float2 wn = up2(fma2(naf, res, wc));
      const bool a0 = in0 && kin, a1 = in1 && kin;
      *reinterpret_cast<float2*>(W1 + ((zr + 1) * 10 + ry) * L::kW1X + xr + 2) =
          make_float2(a0 ? wn.x : 0.0f, a1 ? wn.y : 0.0f);
      if (tilecol && zr >= 0 && zr < ZC) {
        const unsigned long long resm = pk2(a0 ? rf.x : 0.0f, a1 ? rf.y : 0.0f);
        r2 = fma2(resm, resm, r2);
      }
      wm = wc;
      wc = wp;
    }
    if (tilecol) *reinterpret_cast<float2*>(CS + (ry - 1) * kTma2Tile + xr) = up2(r2);
  }
  __syncthreads();

  // ---- sweep s+1 on the tile from w_s in shared memory (rows ty < 8; whole
  // warps, so the shuffles below see full warps)
  if (!RG || ty < kTmaTy) {
  const int i0 = x0 + 2 * tx + 1, j = y0 + ty + 1;
  const bool act0 = i0 <= S.nx && j <= S.ny, act1 = i0 + 1 <= S.nx && j <= S.ny;
  const int kend = min(ZC, S.nz - z0);
  // W1[kz][ky][kx]: kz = zr + 1, ky = yr + 1, kx = xr + 2
  auto w1 = [&](int zr, int dy) { return u64at(W1, ((zr + 1) * 10 + (ty + 1 + dy)) * L::kW1X + 2 * tx + 2); };
  auto w1s = [&](int zr, int dx) { return W1[((zr + 1) * 10 + (ty + 1)) * L::kW1X + 2 * tx + 2 + dx]; };
  unsigned long long wm = w1(-1, 0), wc = w1(0, 0), r2 = 0ull;
  float* out = wout + fidx(S, i0, j, z0 + 1);
  const long long plane = (long long)S.fpitch * S.nyp;
#pragma unroll
  for (int zr = 0; zr < ZC; ++zr) {
    if (zr < kend) {
      const unsigned long long wp = w1(zr + 1, 0);
      unsigned long long rr;
      if (RG)
        rr = (act0 || act1) ? __ldg(reinterpret_cast<const unsigned long long*>(rg + fidx(S, i0, j, z0 + 1 + zr)))
                            : 0ull;
      else
        rr = u64at(R, ((zr + 1) * 10 + (ty + 1)) * kTma2BoxX + 2 * tx + 4);
      const unsigned long long res = node_res(wc, w1s(zr, -1), w1s(zr, 2), w1(zr, -1), w1(zr, 1), wm, wp, rr);
      const float2 rf = up2(res);
      const unsigned long long resm = pk2(act0 ? rf.x : 0.0f, act1 ? rf.y : 0.0f);
      r2 = fma2(resm, resm, r2);
      const float2 wn = up2(fma2(naf, res, wc));
      if (act1) {
        *reinterpret_cast<float2*>(out) = wn;
      } else if (act0) {
        out[0] = wn.x;
      }
      out += plane;
      wm = wc;
      wc = wp;
    }
  }
  // ---- partials of both sweeps for the two 32-wide tiles
  const float2 ca = *reinterpret_cast<const float2*>(CS + ty * kTma2Tile + 2 * tx);
  const double rowA = pair_row_tree(ca.x, ca.y);
  const float2 cb = up2(r2);
  const double rowB = pair_row_tree(cb.x, cb.y);
  if ((tx & 15) == 0) {
    rows[0][tx >> 4][ty] = rowA;
    rows[1][tx >> 4][ty] = rowB;
  }
  }
  __syncthreads();
  if (tid < 4) {
    const int sw = tid >> 1, half = tid & 1;
    const int bx = 2 * bx2 + half;
    if (bx < gx) {
      double sum = 0.0;
      for (int q = 0; q < kTmaTy; ++q) sum += rows[sw][half][q];
      (sw ? partialB : partialA)[bx + (long long)gx * (by + (long long)gy * bz)] = sum;
    }
  }
}

// Periodic ghost refresh of U (CalcEpotential.f90:100-239 on one rank), in
// z, y, x order over whole planes.
__global__ void refresh_periodic_kernel(Stencil S, double* U, int axis) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int nzp = S.nz + 2;
  if (axis == 2) {
    long long n = (long long)S.nxp * S.nyp;
    if (t >= n) return;
    U[t] = U[t + (long long)S.nz * n];
    U[t + (long long)(S.nz + 1) * n] = U[t + n];
  } else if (axis == 1) {
    long long n = (long long)S.nxp * nzp;
    if (t >= n) return;
    int i = int(t % S.nxp), k = int(t / S.nxp);
    auto at = [&](int j) { return (long long)i + (long long)S.nxp * ((long long)j + (long long)S.nyp * k); };
    U[at(0)] = U[at(S.ny)];
    U[at(S.ny + 1)] = U[at(1)];
  } else {
    long long n = (long long)S.nyp * nzp;
    if (t >= n) return;
    int j = int(t % S.nyp), k = int(t / S.nyp);
    long long row = (long long)S.nxp * ((long long)j + (long long)S.nyp * k);
    U[row] = U[row + S.nx];
    U[row + S.nx + 1] = U[row + 1];
  }
}

// Reduce the block partials of `m` consecutive sweeps (one block each) in a
// fixed order: r2[t] = sum_b partial[t * nb + b].
__global__ void reduce_sweeps_kernel(const double* partial, int nb, double* r2) {
  __shared__ double sh[256];
  const double* p = partial + (long long)blockIdx.x * nb;
  double s = 0.0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) s += p[b];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) r2[blockIdx.x] = sh[0];
}

// ------------------------------------------------------ E-field (a11, a12)

// CalcEfield.f90:27-34 + BCfields.f90:31-90 on one rank: interior central
// differences, open-face ghosts zero, periodic ghosts mirrored.  Writes the
// FP64 planes (Ex, Ey, Ez) and the FP32 float4 copy used by the CELL32 gather.
__global__ void efield_kernel(KParams P, const double* U, double* E, float4* E32) {
  chain_begin();
  long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= P.nodes) return;
  int i = int(g % P.nxp), j = int((g / P.nxp) % P.nyp), k = int(g / ((long long)P.nxp * P.nyp));
  int mi = mirror(i, P.nx, P.xflow), mj = mirror(j, P.ny, P.yflow), mk = mirror(k, P.nz, P.zflow);
  double e[3] = {0.0, 0.0, 0.0};
  if (mi >= 0 && mj >= 0 && mk >= 0) {
    // value at the mirrored interior node (equals (i, j, k) when interior)
    auto u = [&](int a, int b, int c) { return U[node_index(P, a, b, c)]; };
    int ii = mi, jj = mj, kk = mk;
    e[2] = -(u(ii, jj, kk + 1) - u(ii, jj, kk - 1)) * 0.5 / P.dz;
    e[1] = -(u(ii, jj + 1, kk) - u(ii, jj - 1, kk)) * 0.5 / P.dy;
    e[0] = -(u(ii + 1, jj, kk) - u(ii - 1, jj, kk)) * 0.5 / P.dx;
  }
  E[g] = e[0];
  E[P.nodes + g] = e[1];
  E[2 * P.nodes + g] = e[2];
  if (E32) E32[g] = make_float4(float(e[0]), float(e[1]), float(e[2]), 0.0f);
}

// BCfields.f90:31-90 on one rank: zero the ghost layer of every open face.
__global__ void bc_fields_kernel(KParams P, double* E, float4* E32) {
  long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= P.nodes) return;
  int i = int(g % P.nxp), j = int((g / P.nxp) % P.nyp), k = int(g / ((long long)P.nxp * P.nyp));
  bool ghost = (P.xflow && (i == 0 || i == P.nx + 1)) || (P.yflow && (j == 0 || j == P.ny + 1)) ||
               (P.zflow && (k == 0 || k == P.nz + 1));
  if (!ghost) return;
  E[g] = 0.0;
  E[P.nodes + g] = 0.0;
  E[2 * P.nodes + g] = 0.0;
  if (E32) E32[g] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

// Block partials of sum |E + E0|^2 over interior nodes (picard.f90:656-658).
__global__ void energy_field_kernel(KParams P, const double* E, double* partial) {
  long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double v = 0.0;
  if (g < P.nodes) {
    int i = int(g % P.nxp), j = int((g / P.nxp) % P.nyp), k = int(g / ((long long)P.nxp * P.nyp));
    if (i >= 1 && i <= P.nx && j >= 1 && j <= P.ny && k >= 1 && k <= P.nz) {
      double a = E[g] + P.E0[0], b = E[P.nodes + g] + P.E0[1], c = E[2 * P.nodes + g] + P.E0[2];
      v = a * a + b * b + c * c;
    }
  }
  __shared__ double sh[32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < int(blockDim.x >> 5); ++w) s += sh[w];
    partial[blockIdx.x] = s;
  }
}

__global__ void sum_partials_kernel(const double* partial, int nb, double scale, double* out) {
  __shared__ double sh[256];
  double s = 0.0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) s += partial[b];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0] * scale;
}

}  // namespace

// ------------------------------------------------------------ wrappers

Stencil make_stencil(const KParams& P) {
  Stencil S;
  S.nx = P.nx;
  S.ny = P.ny;
  S.nz = P.nz;
  S.nxp = P.nxp;
  S.nyp = P.nyp;
  S.px = !P.xflow;
  S.py = !P.yflow;
  S.pz = !P.zflow;
  S.nodes = P.nodes;
  S.fpitch = f32_pitch(P);
  return S;
}

int f32_pitch(const KParams& P) { return ((P.nx + 5 + 7) / 8) * 8; }
long long f32_elems(const KParams& P) { return (long long)f32_pitch(P) * P.nyp * P.nzp; }

JacobiGeom jacobi_geom(const KParams& P) {
  JacobiGeom G;
  G.block = dim3(32, 8, 1);
  int bx = (P.nx + 31) / 32, by = (P.ny + 7) / 8;
  // enough z-blocks for ~4 blocks per SM, at least 4 nodes per thread
  int want = (4 * 148 + bx * by - 1) / (bx * by);
  int zc = (P.nz + want - 1) / want;
  if (zc < 4) zc = 4;
  if (zc > P.nz) zc = P.nz;
  G.tma = P.xflow && P.yflow && P.zflow;
  if (G.tma) {
    // TMA column depth: 8 planes (26 KB of shared memory, 8 blocks per SM),
    // 4 for shallow grids
    zc = P.nz >= 64 ? 8 : 4;
  }
  G.zc = zc;
  G.grid = dim3(bx, by, (P.nz + zc - 1) / zc);
  G.nblocks = bx * by * G.grid.z;
  return G;
}

JacobiCoef jacobi_coef(const KParams& P) {
  JacobiCoef J;
  double dx = P.dx, dy = P.dy, dz = P.dz;
  double S = (dx * dy) * (dx * dy) + (dx * dz) * (dx * dz) + (dy * dz) * (dy * dz);
  J.ax = 0.5 * (1.0 / S) * ((dy * dz) * (dy * dz));
  J.ay = 0.5 * (1.0 / S) * ((dx * dz) * (dx * dz));
  J.az = 0.5 * (1.0 / S) * ((dx * dy) * (dx * dy));
  J.af = 0.5 * (1.0 / S) * ((dx * dy * dz) * (dx * dy * dz));
  J.dx2 = dx * dx;
  J.dy2 = dy * dy;
  J.dz2 = dz * dz;
  return J;
}

JacobiCoefF jacobi_coef_f(const KParams& P) {
  JacobiCoef J = jacobi_coef(P);
  JacobiCoefF F;
  F.af = float(J.af);
  F.idx2 = float(1.0 / J.dx2);
  F.idy2 = float(1.0 / J.dy2);
  F.idz2 = float(1.0 / J.dz2);
  return F;
}

cudaError_t launch_finish_deposit(const KParams& P, const unsigned long long* Nacc, double* N, double* C,
                                  cudaStream_t st) {
  return launch_chained(finish_deposit_kernel, grid_for(P.nodes), kThreads, 0, st, P, Nacc, N, C);
}

cudaError_t launch_finish_flux(const KParams& P, const unsigned long long* Facc, double* F, cudaStream_t st) {
  note_launch();
  finish_flux_kernel<<<grid_for(P.nodes), kThreads, 0, st>>>(P, Facc, F);
  return cudaGetLastError();
}

long long bc_direct_scratch(const KParams& P) {
  long long most = 0;
  for (int axis = 0; axis < 3; ++axis) {
    const DirectSplit S = direct_split(P, axis, LLONG_MAX);
    most = std::max(most, 2LL * S.groups * S.n1 * S.n2);
  }
  return most;
}

cudaError_t launch_bc_potentials(const KParams& P, const double* C, const double* D, double* U, double* scratch,
                                 long long room, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(U, 0, sizeof(double) * P.nodes, st);  // BCpotentials.f90:36
  if (e != cudaSuccess) return e;
  const int flows[3] = {P.xflow, P.yflow, P.zflow};
  for (int axis = 0; axis < 3; ++axis) {
    if (!flows[axis]) continue;
    const DirectSplit S = direct_split(P, axis, room);
    note_launch();
    bc_potentials_kernel<<<dim3(S.bx, S.by, S.groups), dim3(kBT, kBT), 0, st>>>(P, axis, S.per, C, D, scratch);
    if ((e = cudaGetLastError())) return e;
    note_launch();
    bc_direct_sum_kernel<<<grid_for((long long)S.n1 * S.n2), kThreads, 0, st>>>(P, axis, S.groups, scratch, U);
    if ((e = cudaGetLastError())) return e;
  }
  return cudaSuccess;
}

int rhs_blocks(const KParams& P) { return grid_for(P.nodes); }

cudaError_t launch_rhs(const KParams& P, const double* C, double* b, double* partial, double* bnorm2,
                       cudaStream_t st) {
  int nb = grid_for(P.nodes);
  note_launch();
  rhs_kernel<<<nb, kThreads, 0, st>>>(P, C, b, partial);
  note_launch();
  sum_partials_kernel<<<1, 256, 0, st>>>(partial, nb, 1.0, bnorm2);
  return cudaGetLastError();
}

cudaError_t launch_sweep_f64(const KParams& P, const JacobiGeom& G, const double* Uin, double* Uout, const double* b,
                             double* partial, cudaStream_t st) {
  note_launch();
  sweep_f64_kernel<<<G.grid, G.block, 0, st>>>(make_stencil(P), jacobi_coef(P), Uin, Uout, b, partial, G.zc);
  return cudaGetLastError();
}

cudaError_t launch_sweep_f32(const KParams& P, const JacobiGeom& G, const float* win, float* wout, const float* r,
                             double* partial, int w_zero, cudaStream_t st) {
  note_launch();
  sweep_f32_kernel<<<G.grid, G.block, 0, st>>>(make_stencil(P), jacobi_coef_f(P), win, wout, r, partial, G.zc,
                                                w_zero);
  return cudaGetLastError();
}

int make_tensor_map(CUtensorMap* m, float* base, const KParams& P, int box_x, int box_y, int box_z) {
  using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static Encode encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn)
      return (int)CUDA_ERROR_NOT_FOUND;
    encode = reinterpret_cast<Encode>(fn);
  }
  const int pitch = f32_pitch(P);
  cuuint64_t dims[3] = {(cuuint64_t)pitch, (cuuint64_t)P.nyp, (cuuint64_t)P.nzp};
  cuuint64_t strides[2] = {(cuuint64_t)pitch * sizeof(float), (cuuint64_t)pitch * P.nyp * sizeof(float)};
  cuuint32_t box[3] = {(cuuint32_t)box_x, (cuuint32_t)box_y, (cuuint32_t)box_z};
  cuuint32_t estr[3] = {1, 1, 1};
  return (int)encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

template <int ZC, int STAGES>
static cudaError_t launch_tma_zs(const KParams& P, const JacobiGeom& G, const CUtensorMap* tw, const CUtensorMap* tr,
                                 float* wout, double* partial, int w_zero, int* err, cudaStream_t st) {
  const size_t smem = STAGES * TmaStage<ZC>::kBytes;
  static bool attr = false;
  if (!attr) {
    cudaError_t e =
        cudaFuncSetAttribute(sweep_tma_kernel<ZC, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  const int ntiles = G.nblocks;
  const int ctas = G.ctas > 0 ? std::min(G.ctas, ntiles) : ntiles;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kTmaTx, kTmaTy);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = G.pdl ? 1 : 0;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  note_launch();
  return cudaLaunchKernelEx(&cfg, sweep_tma_kernel<ZC, STAGES>, *tw, *tr, make_stencil(P), jacobi_coef_f(P), wout,
                            partial, w_zero, (int)G.grid.x, (int)G.grid.y, ntiles, err);
}

template <int ZC>
static cudaError_t launch_tma_zc(const KParams& P, const JacobiGeom& G, const CUtensorMap* tw, const CUtensorMap* tr,
                                 float* wout, double* partial, int w_zero, int* err, cudaStream_t st) {
  return G.stages == 2 ? launch_tma_zs<ZC, 2>(P, G, tw, tr, wout, partial, w_zero, err, st)
                       : launch_tma_zs<ZC, 1>(P, G, tw, tr, wout, partial, w_zero, err, st);
}

template <int ZC, int STAGES>
static int occupancy_zs() {
  const size_t smem = STAGES * TmaStage<ZC>::kBytes;
  if (cudaFuncSetAttribute(sweep_tma_kernel<ZC, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return 1;
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, sweep_tma_kernel<ZC, STAGES>, kTmaTx * kTmaTy, smem) !=
      cudaSuccess)
    return 1;
  return n > 0 ? n : 1;
}

int sweep_tma_occupancy(const JacobiGeom& G, int stages) {
  switch (G.zc * 4 + (stages == 2 ? 1 : 0)) {
    case 16: return occupancy_zs<4, 1>();
    case 17: return occupancy_zs<4, 2>();
    case 32: return occupancy_zs<8, 1>();
    case 33: return occupancy_zs<8, 2>();
    case 64: return occupancy_zs<16, 1>();
    case 65: return occupancy_zs<16, 2>();
  }
  return 1;
}

template <int ZC, int STAGES>
static cudaError_t launch_tma2_zs(const KParams& P, const JacobiGeom& G, const CUtensorMap* tw, const CUtensorMap* tr,
                                  const float* r, float* wout, double* partial, int w_zero, int* err,
                                  cudaStream_t st) {
  const size_t smem = STAGES * Tma2Stage<ZC>::kBytes;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaSuccess;
    for (auto k : {sweep_tma2_kernel<ZC, STAGES, false, true>, sweep_tma2_kernel<ZC, STAGES, true, true>,
                   sweep_tma2_kernel<ZC, STAGES, false, false>, sweep_tma2_kernel<ZC, STAGES, true, false>})
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  const int gx2 = (P.nx + kTma2Tile - 1) / kTma2Tile;
  const int ntiles = gx2 * (int)G.grid.y * (int)G.grid.z;
  const int ctas = G.ctas > 0 ? std::min(G.ctas, ntiles) : ntiles;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kTmaTx, kTmaTy);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = G.pdl ? 1 : 0;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  note_launch();
  // one CTA per tile with one stage: the loop-free instantiation
  const bool loop = STAGES == 2 || ctas < ntiles;
  if (G.rglobal && !loop && r) {
    // r from global memory: the w box alone in shared memory (below the
    // 48 KB default, no attribute needed)
    cfg.dynamicSmemBytes = Tma2Stage<ZC>::kW * sizeof(float);
    auto kr = w_zero ? sweep_tma2r_kernel<ZC, true> : sweep_tma2r_kernel<ZC, false>;
    return cudaLaunchKernelEx(&cfg, kr, *tw, r, make_stencil(P), jacobi_coef_f(P), wout, partial, gx2,
                              (int)G.grid.x, (int)G.grid.y, ntiles, err);
  }
  auto kern = w_zero ? (loop ? sweep_tma2_kernel<ZC, STAGES, true, true> : sweep_tma2_kernel<ZC, STAGES, true, false>)
                     : (loop ? sweep_tma2_kernel<ZC, STAGES, false, true> : sweep_tma2_kernel<ZC, STAGES, false, false>);
  return cudaLaunchKernelEx(&cfg, kern, *tw, *tr, make_stencil(P), jacobi_coef_f(P), wout, partial, gx2,
                            (int)G.grid.x, (int)G.grid.y, ntiles, err);
}

template <int ZC>
static cudaError_t launch_tma2_zc(const KParams& P, const JacobiGeom& G, const CUtensorMap* tw, const CUtensorMap* tr,
                                  const float* r, float* wout, double* partial, int w_zero, int* err,
                                  cudaStream_t st) {
  return G.stages == 2 ? launch_tma2_zs<ZC, 2>(P, G, tw, tr, r, wout, partial, w_zero, err, st)
                       : launch_tma2_zs<ZC, 1>(P, G, tw, tr, r, wout, partial, w_zero, err, st);
}

template <int ZC, int STAGES>
static int occupancy2_zs() {
  const size_t smem = STAGES * Tma2Stage<ZC>::kBytes;
  if (cudaFuncSetAttribute(sweep_tma2_kernel<ZC, STAGES, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem) != cudaSuccess)
    return 1;
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, sweep_tma2_kernel<ZC, STAGES, false, true>, kTmaTx * kTmaTy,
                                                    smem) !=
      cudaSuccess)
    return 1;
  return n > 0 ? n : 1;
}

int sweep_tma2_occupancy(const JacobiGeom& G, int stages) {
  switch (G.zc * 4 + (stages == 2 ? 1 : 0)) {
    case 16: return occupancy2_zs<4, 1>();
    case 17: return occupancy2_zs<4, 2>();
    case 32: return occupancy2_zs<8, 1>();
    case 33: return occupancy2_zs<8, 2>();
    case 64: return occupancy2_zs<16, 1>();
    case 65: return occupancy2_zs<16, 2>();
  }
  return 1;
}

int sweep_tma2_tiles(const KParams& P, const JacobiGeom& G) {
  return ((P.nx + kTma2Tile - 1) / kTma2Tile) * (int)G.grid.y * (int)G.grid.z;
}

cudaError_t launch_sweep_tma2(const KParams& P, const JacobiGeom& G, const CUtensorMap* tw, const CUtensorMap* tr,
                              const float* r, float* wout, double* partial, int w_zero, int* err, cudaStream_t st) {
  switch (G.zc) {
    case 4: return launch_tma2_zc<4>(P, G, tw, tr, r, wout, partial, w_zero, err, st);
    case 8: return launch_tma2_zc<8>(P, G, tw, tr, r, wout, partial, w_zero, err, st);
    case 16: return launch_tma2_zc<16>(P, G, tw, tr, r, wout, partial, w_zero, err, st);
  }
  return cudaErrorInvalidValue;
}

template <int ZC, bool RG>
static cudaError_t launch_sweep2_zc(const KParams& P, const JacobiGeom& G, const CUtensorMap* tw,
                                    const CUtensorMap* tr, const float* r, float* wout, double* partialA,
                                    double* partialB, int w_zero, int* err, cudaStream_t st) {
  const size_t smem = Sweep2Smem<ZC, RG>::kBytes;
  static bool attr = false;
  if (!attr) {
    cudaError_t e =
        cudaFuncSetAttribute(sweep2_tma_kernel<ZC, RG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  const int gx2 = (P.nx + kTma2Tile - 1) / kTma2Tile;
  const int ntiles = gx2 * (int)G.grid.y * (int)G.grid.z;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ntiles);
  cfg.blockDim = dim3(kTmaTx, RG ? 12 : kTmaTy);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = G.pdl ? 1 : 0;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  note_launch();
  return cudaLaunchKernelEx(&cfg, sweep2_tma_kernel<ZC, RG>, *tw, *tr, r, make_stencil(P), jacobi_coef_f(P), wout,
                            partialA, partialB, w_zero, gx2, (int)G.grid.x, (int)G.grid.y, ntiles, err);
}

cudaError_t launch_sweep2_tma(const KParams& P, const JacobiGeom& G, const CUtensorMap* tw, const CUtensorMap* tr,
                              const float* r, float* wout, double* partialA, double* partialB, int w_zero, int* err,
                              cudaStream_t st) {
  const bool rg = G.rglobal != 0;
  switch (G.zc) {
    case 4:
      return rg ? launch_sweep2_zc<4, true>(P, G, tw, tr, r, wout, partialA, partialB, w_zero, err, st)
                : launch_sweep2_zc<4, false>(P, G, tw, tr, r, wout, partialA, partialB, w_zero, err, st);
    case 8:
      return rg ? launch_sweep2_zc<8, true>(P, G, tw, tr, r, wout, partialA, partialB, w_zero, err, st)
                : launch_sweep2_zc<8, false>(P, G, tw, tr, r, wout, partialA, partialB, w_zero, err, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_sweep_tma(const KParams& P, const JacobiGeom& G, const CUtensorMap* tw, const CUtensorMap* tr,
                             float* wout, double* partial, int w_zero, int* err, cudaStream_t st) {
  switch (G.zc) {
    case 4: return launch_tma_zc<4>(P, G, tw, tr, wout, partial, w_zero, err, st);
    case 8: return launch_tma_zc<8>(P, G, tw, tr, wout, partial, w_zero, err, st);
    case 16: return launch_tma_zc<16>(P, G, tw, tr, wout, partial, w_zero, err, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_anchor(const KParams& P, const JacobiGeom& G, const double* Vin, double* Vout, const float* w,
                          const double* b, float* r, double sigma, double* partial, int w_zero, cudaStream_t st) {
  note_launch();
  anchor_kernel<<<G.grid, G.block, 0, st>>>(make_stencil(P), jacobi_coef(P), Vin, Vout, w, b, r, sigma, partial,
                                             G.zc, w_zero);
  return cudaGetLastError();
}

cudaError_t launch_finalize(const KParams& P, const double* V, const float* w, double sigma, double* U, int w_zero,
                            cudaStream_t st) {
  note_launch();
  finalize_kernel<<<grid_for(P.nodes), kThreads, 0, st>>>(make_stencil(P), V, w, sigma, U, w_zero);
  return cudaGetLastError();
}

cudaError_t launch_refresh_periodic(const KParams& P, double* U, cudaStream_t st) {
  Stencil S = make_stencil(P);
  if (S.pz) {
    note_launch();
    refresh_periodic_kernel<<<grid_for((long long)S.nxp * S.nyp), kThreads, 0, st>>>(S, U, 2);
  }
  if (S.py) {
    note_launch();
    refresh_periodic_kernel<<<grid_for((long long)S.nxp * (S.nz + 2)), kThreads, 0, st>>>(S, U, 1);
  }
  if (S.px) {
    note_launch();
    refresh_periodic_kernel<<<grid_for((long long)S.nyp * (S.nz + 2)), kThreads, 0, st>>>(S, U, 0);
  }
  return cudaGetLastError();
}

cudaError_t launch_reduce_sweeps(const double* partial, int nb, int m, double* r2, cudaStream_t st) {
  if (m <= 0) return cudaSuccess;
  note_launch();
  reduce_sweeps_kernel<<<m, 256, 0, st>>>(partial, nb, r2);
  return cudaGetLastError();
}

cudaError_t launch_zero(void* p, long long n, cudaStream_t st) {
  const long long blocks = (n / 2 + kThreads - 1) / kThreads;
  return launch_chained(zero_kernel, int(blocks < 1 ? 1 : blocks < 148 * 8 ? blocks : 148 * 8), kThreads, 0, st,
                        static_cast<unsigned long long*>(p), n);
}

cudaError_t launch_efield(const KParams& P, const double* U, double* E, float4* E32, cudaStream_t st) {
  return launch_chained(efield_kernel, grid_for(P.nodes), kThreads, 0, st, P, U, E, E32);
}

cudaError_t launch_bc_fields(const KParams& P, double* E, float4* E32, cudaStream_t st) {
  note_launch();
  bc_fields_kernel<<<grid_for(P.nodes), kThreads, 0, st>>>(P, E, E32);
  return cudaGetLastError();
}

cudaError_t launch_energy_field(const KParams& P, const double* E, double* partial, double* out, cudaStream_t st) {
  int nb = grid_for(P.nodes);
  note_launch();
  energy_field_kernel<<<nb, kThreads, 0, st>>>(P, E, partial);
  note_launch();
  sum_partials_kernel<<<1, 256, 0, st>>>(partial, nb, 0.5 * kEps0 * P.dV, out);
  return cudaGetLastError();
}

}  // namespace picard
