// spectral.cu -- CalcEpotential's Jacobi iterate (CalcEpotential.f90:55-96)
// evaluated in closed form in the eigenbasis of the sweep.
//
// One reference sweep is U <- U - af * res with res = b - L U (L the 7-point
// Laplacian over the interior; ghosts held fixed on open faces, wrapped on
// periodic axes; CalcEpotential.f90:74-92, with af/d^2 = a_d).  A sweep
// changes only interior nodes, so the residual of iterate d is
//   r_d = G^d r_0,  G = ax S_x + ay S_y + az S_z,
// S_d the neighbour-sum operator of axis d with zero ghosts (open) or wrap
// (periodic), and
//   U_d = U_0 - af * sum_{j<d} G^j r_0.
// Each S_d is diagonalised by an orthonormal basis Q_d of its axis:
//   open:     Q[m][i] = sqrt(2/(n+1)) sin(pi (m+1)(i+1)/(n+1)), eigenvalue
//             2 cos(pi (m+1)/(n+1))  (the discrete sine transform, DST-I);
//   periodic: the real Fourier basis 1/sqrt(n), sqrt(2/n) cos / sin(2 pi f i/n)
//             and (-1)^i/sqrt(n), eigenvalue 2 cos(2 pi f/n).
// In the product basis Q = Qz Qy Qx the operator G is diagonal with
// g = 1 - omg, omg = sum_d a_d (2 - sigma_d) (2 (ax + ay + az) = 1), so with
// rh = Q r_0:
//   ||r_d||^2 = sum_m g_m^(2d) rh_m^2            (Parseval),
//   U_d = U_0 - af Q^T [ (1 - g^d)/(1 - g) rh ].
// ||r_d|| does not increase with d (|g| <= 1), and the stopping sweep of the
// reference -- the first iterate d >= 1 with d + 1 <= maxit and
// ||r_d|| <= maxerr ||b|| -- is found by a bracketing search: each launch
// evaluates the Parseval sum at up to kSpecPoints sweep counts, and its last
// block narrows the bracket and chooses the next ones (SpecState), so that the
// whole solve is queued without a host round trip.
//
// The transforms are per-axis products, one launch each, on the FP64 tensor
// cores (spec_axis_kernel).  Every axis basis is folded by its even / odd
// symmetry, which halves the flops.  Everything is FP64; the result equals the
// FP64 sweeps' iterate to rounding (the sweeps themselves round each of their
// d updates).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "chain.cuh"
#include "context.cuh"
#include "picard_gpu.h"
#include "solve_f32.cuh"

namespace picard {

namespace {

constexpr int kSpecPoints = 32;     // sweep counts per evaluation launch
constexpr int kSpecThreads = 256;
enum SpecPhase { kSpecDoubling = 0, kSpecUniform = 1, kSpecFinal = 2 };
constexpr int kAxTile = 64, kAxK = 16;  // spec_axis_kernel: 64 x 64 outputs per parity, K chunks of 16

// Element t of a compact nx x ny array of planes -> (i, j, k).  T is 32 bits
// wherever the element count allows: the two divisions by run-time extents are
// most of the integer work of the passes below.
template <class T>
__device__ __forceinline__ void split3(T t, int nx, int ny, int& i, int& j, int& k) {
  const T r = t / T(nx), q = r / T(ny);
  i = int(t - r * T(nx));
  j = int(r - q * T(ny));
  k = int(q);
}
inline bool fits32(long long n) { return n < (1LL << 31); }

// The sum over the block of one value per thread, in thread 0 (fixed order).
__device__ __forceinline__ double block_sum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < int(blockDim.x >> 5); ++w) t += sh[w];
  return t;
}

// A queued solve's times on the device's clock, behind its SpecState: start of the
// set-up, of the search and of the iterate, and the latest end of a block of the
// last pass.  (Events would keep the kernels on either side of them apart.)
__device__ __forceinline__ SpecStamps* stamps_of(SpecState* state) { return reinterpret_cast<SpecStamps*>(state + 1); }
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long v;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(v));
  return v;
}

// b = -C/(dV eps0) and r_0 = b - L U over the interior, compact x-fastest
// (CalcEpotential.f90:50-54, 83-92; periodic axes read the wrapped interior
// instead of the ghost), ||b||^2, and from it, in the last block, the start of
// the stopping-sweep search.  The test at the top of sweep 1 uses ||b|| itself
// (CalcEpotential.f90:55-61).
template <class T>
__global__ void __launch_bounds__(kSpecThreads) spec_begin_kernel(KParams P, double idx2, double idy2, double idz2,
                                                                  double binv, const double* C,
                                                                  const double* U, double* R,
                                                                  double maxerr, int maxit,
                                                                  double* __restrict__ partial, unsigned int* counter,
                                                                  SpecState* state) {
  chain_begin();
  if (blockIdx.x == 0 && threadIdx.x == 0) *stamps_of(state) = SpecStamps{global_ns(), 0, 0, 0};
  const T n = T(P.nx) * T(P.ny) * T(P.nz);
  double b2 = 0.0;
  for (T t = T(blockIdx.x) * blockDim.x + threadIdx.x; t < n; t += T(gridDim.x) * blockDim.x) {
    int i, j, k;
    split3(t, P.nx, P.ny, i, j, k);
    ++i, ++j, ++k;
    const int im = (i == 1 && !P.xflow) ? P.nx : i - 1, ip = (i == P.nx && !P.xflow) ? 1 : i + 1;
    const int jm = (j == 1 && !P.yflow) ? P.ny : j - 1, jp = (j == P.ny && !P.yflow) ? 1 : j + 1;
    const int km = (k == 1 && !P.zflow) ? P.nz : k - 1, kp = (k == P.nz && !P.zflow) ? 1 : k + 1;
    const long long g = node_index(P, i, j, k);
    const double u = U[g];
    const double lap = (U[node_index(P, ip, j, k)] + U[node_index(P, im, j, k)] - 2.0 * u) * idx2 +
                       (U[node_index(P, i, jp, k)] + U[node_index(P, i, jm, k)] - 2.0 * u) * idy2 +
                       (U[node_index(P, i, j, kp)] + U[node_index(P, i, j, km)] - 2.0 * u) * idz2;
    const double b = -C[g] * binv;
    R[t] = b - lap;
    b2 += b * b;
  }
  __shared__ double sh[kSpecThreads / 32];
  __shared__ bool last;
  b2 = block_sum(b2, sh);
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = b2;
    __threadfence();
    last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double v = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) v += __ldcg(partial + b);
  v = block_sum(v, sh);
  if (threadIdx.x != 0) return;
  *counter = 0u;
  SpecState Q;
  Q.bnorm = sqrt(v);
  const double tol = maxerr * Q.bnorm;
  Q.tol2 = tol * tol;
  Q.f1 = Q.r2_hit = 0.0;
  Q.smax = 2LL * maxit + 1;
  Q.dmax = (long long)maxit - 1;
  Q.lo = 0;
  Q.hi = Q.dmax + 1;
  Q.d = 0;
  Q.d0 = 1;
  Q.step = 0;
  Q.g2_skip = -1.0;
  Q.trivial = 1 <= maxit && Q.bnorm <= tol;
  Q.done = Q.trivial;
  Q.converged = 1;
  if (Q.dmax >= 1) {
    Q.phase = kSpecDoubling;
    Q.count = 1;
    while (Q.count < kSpecPoints && (1LL << (Q.count - 1)) < Q.dmax) ++Q.count;
  } else {
    Q.phase = kSpecFinal;
    Q.d0 = Q.smax;
    Q.count = 1;
  }
  *state = Q;
}

// D += A B for one 8 x 4 by 4 x 8 FP64 tile: lane l holds A[l / 4][l % 4],
// B[l % 4][l / 4] and D[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void mma_f64(double& d0, double& d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

// One axis pass of the transform.  An axis of length n has `ne` even and `no`
// odd basis functions about the reflection i -> n - 1 - i + s (s = 0 open, 1
// periodic, indices mod n): element i < ne stands for itself and, when s <= i
// < no + s, for its partner n - 1 - i + s, so
//   forward: out[m] = sum_i Pe[m][i] (x[i] + x[partner]),
//            out[ne + m] = sum_i Po[m][i - s] (x[i] - x[partner]);
//   inverse: out[i] = E[i] + O[i], out[partner] = E[i] - O[i], with
//            E[i] = sum_k Pe[k][i] in[k] and O[i] = sum_k Po[k][i - s] in[ne + k].
// Both halves read the same input, so one block computes the 64 x 64 outputs
// of both: warps 0-3 the even half, warps 4-7 the odd one, 32 x 32 each as 4 x
// 4 tiles of mma.m8n8k4.  The fold is done while the input is staged and the
// unfold while the output is written, so a pass reads and writes the array
// once.
//
// X: the axis is contiguous (rows of n, `rows` of them): A = data, B = matrix
// (Pe, Po given as [k][output]).  Else the axis has stride I and the block
// takes 64 of the I contiguous columns of slab blockIdx.z: A = matrix ([output]
// [k]), B = data.  APPLY (x, inverse): adds the outputs to U's interior instead
// of storing them.
//
// What bounds it: the inverse passes the FP64 tensor pipe (53 % busy, its throttle
// the first stall), the forward ones the latency of the staging loads, which two
// blocks of 128 registers per SM do not hide (35 to 39 % busy, long scoreboard);
// small grids the launch.  4.3 GFLOP of products for both transforms of 256 x 128 x
// 128 are 0.12 ms at 37 TFLOP/s.
// Both transforms of 256 x 128 x 128 with the update of U: 286 us in 6 launches,
// against 498 us in 19 for products with 4 x 4 outputs per thread (as many
// shared-memory as FP64 cycles), in-place butterflies and a pass of its own for
// the update; 24^3: 28 us against 55 us.
template <bool INV, bool X, bool APPLY>
__global__ void __launch_bounds__(256, 2) spec_axis_kernel(const double* in, double* out,
                                                           const double* __restrict__ Pe,
                                                           const double* __restrict__ Po, int n, int ne, int no, int s,
                                                           long long I, int rows, KParams P, double* U,
                                                           SpecState* state) {
  chain_begin();
  if (APPLY && state->trivial) return;  // zero sweeps: U stays
  // row strides 4 mod 16 doubles: the 16 lanes of a half-warp read 16 banks
  __shared__ double sh[2 * kAxTile * (kAxK + 4) + 2 * kAxK * (kAxTile + 4)];
  double(*As)[kAxTile][kAxK + 4] = reinterpret_cast<double(*)[kAxTile][kAxK + 4]>(sh);
  double(*Bs)[kAxK][kAxTile + 4] = reinterpret_cast<double(*)[kAxK][kAxTile + 4]>(sh + 2 * kAxTile * (kAxK + 4));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int par = warp >> 2, wm = (warp >> 1) & 1, wn = warp & 1;
  const int c0 = blockIdx.x * kAxTile, r0 = blockIdx.y * kAxTile;  // first output column and row of the tile
  // outputs run over rows (not X) or columns (X); the other index is the data's
  const int o0 = X ? c0 : r0;
  const long long v0 = X ? r0 : c0, vn = X ? rows : I;
  const long long slab = X ? 0 : (long long)blockIdx.z * n * I;
  in += slab;
  if (!APPLY) out += slab;
  const int K = ne;
  // data element `i` of vector v: even and odd value (i - s: the odd index)
  auto data = [&](long long v, int i, double& e, double& o) {
    e = o = 0.0;
    if (v >= vn || i >= ne) return;
    const double* x = X ? in + v * n : in + v;
    const long long st = X ? 1 : I;
    if (INV) {
      e = x[(long long)i * st];
      if (i < no) o = x[(long long)(ne + i) * st];
    } else {
      const double a = x[(long long)i * st];
      if (i >= s && i < no + s) {
        const double b = x[(long long)(n - 1 - i + s) * st];
        e = a + b;
        o = a - b;
      } else {
        e = a;
      }
    }
  };
  // matrix entry of output q (a mode, or INV an element) and summation index k
  auto matrix = [&](int q, int k, double& e, double& o) {
    const int qo = INV ? q - s : q, ko = INV ? k : k - s;
    e = (q < ne && k < ne) ? (X ? Pe[(long long)k * ne + q] : Pe[(long long)q * ne + k]) : 0.0;
    o = (qo >= 0 && qo < no && ko >= 0 && ko < no) ? (X ? Po[(long long)ko * no + qo] : Po[(long long)qo * no + ko]) : 0.0;
  };
  double acc[4][4][2];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
  // rows of this warp's parity that exist at all (uniform per warp)
  const int lim = INV ? ne : (par ? no : ne);
  const bool live = X ? (c0 + wn * 32 < lim && r0 + wm * 32 < rows) : (r0 + wm * 32 < lim && v0 + wn * 32 < I);
  double ae[4], ao[4], be[4], bo[4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int q = tid + 256 * e;
      if (X) {
        data(v0 + (q >> 4), k0 + (q & 15), ae[e], ao[e]);
        matrix(o0 + (q & 63), k0 + (q >> 6), be[e], bo[e]);
      } else {
        matrix(o0 + (q >> 4), k0 + (q & 15), ae[e], ao[e]);
        data(v0 + (q & 63), k0 + (q >> 6), be[e], bo[e]);
      }
    }
  };
  fetch(0);
  for (int k0 = 0; k0 < K; k0 += kAxK) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int q = tid + 256 * e;
      As[0][q >> 4][q & 15] = ae[e];
      As[1][q >> 4][q & 15] = ao[e];
      Bs[0][q >> 6][q & 63] = be[e];
      Bs[1][q >> 6][q & 63] = bo[e];
    }
    __syncthreads();
    if (k0 + kAxK < K) fetch(k0 + kAxK);
    if (live) {
#pragma unroll
      for (int kk = 0; kk < kAxK; kk += 4) {
        double a[4], b[4];
#pragma unroll
        for (int f = 0; f < 4; ++f) a[f] = As[par][wm * 32 + 8 * f + (lane >> 2)][kk + (lane & 3)];
#pragma unroll
        for (int f = 0; f < 4; ++f) b[f] = Bs[par][kk + (lane & 3)][wn * 32 + 8 * f + (lane >> 2)];
#pragma unroll
        for (int fa = 0; fa < 4; ++fa)
#pragma unroll
          for (int fb = 0; fb < 4; ++fb) mma_f64(acc[fa][fb][0], acc[fa][fb][1], a[fa], b[fb]);
      }
    }
    __syncthreads();
  }
  if constexpr (INV) {  // the odd half goes to the even warps
    double(*Os)[kAxTile + 2] = reinterpret_cast<double(*)[kAxTile + 2]>(sh);
    if (par == 1) {
#pragma unroll
      for (int fa = 0; fa < 4; ++fa)
#pragma unroll
        for (int fb = 0; fb < 4; ++fb)
#pragma unroll
          for (int t = 0; t < 2; ++t)
            Os[wm * 32 + 8 * fa + (lane >> 2)][wn * 32 + 8 * fb + 2 * (lane & 3) + t] = acc[fa][fb][t];
    }
    __syncthreads();
    if (par == 1) return;
#pragma unroll
    for (int fa = 0; fa < 4; ++fa) {
      const int row = wm * 32 + 8 * fa + (lane >> 2);
      double* y = nullptr;  // x: the row's first output
      if constexpr (X) {
        const unsigned v = unsigned(v0) + row, vk = v / unsigned(P.ny);
        if (v >= unsigned(rows)) continue;
        y = APPLY ? U + node_index(P, 1, 1 + int(v - vk * P.ny), 1 + int(vk)) : out + (long long)v * n;
      }
      double u0[4][2], u1[4][2];  // APPLY: all of a row's loads before its first store
      if constexpr (APPLY) {
#pragma unroll
        for (int fb = 0; fb < 4; ++fb)
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const int i = o0 + wn * 32 + 8 * fb + 2 * (lane & 3) + t;
            u0[fb][t] = i < ne ? y[i] : 0.0;
            u1[fb][t] = i < ne && i >= s && i < no + s ? y[n - 1 - i + s] : 0.0;
          }
      }
#pragma unroll
      for (int fb = 0; fb < 4; ++fb)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int col = wn * 32 + 8 * fb + 2 * (lane & 3) + t;
          const int i = o0 + (X ? col : row);
          const double E = acc[fa][fb][t], O = Os[row][col];
          const bool pair = i >= s && i < no + s;
          const int j = n - 1 - i + s;
          if (i >= ne) continue;
          if constexpr (APPLY) {
            y[i] = u0[fb][t] + (pair ? E + O : E);
            if (pair) y[j] = u1[fb][t] + (E - O);
          } else if constexpr (X) {
            y[i] = pair ? E + O : E;
            if (pair) y[j] = E - O;
          } else {
            const long long v = v0 + col;
            if (v >= I) continue;
            out[(long long)i * I + v] = pair ? E + O : E;
            if (pair) out[(long long)j * I + v] = E - O;
          }
        }
    }
    if (APPLY && tid == 0) atomicMax(&stamps_of(state)->end, global_ns());
  } else {
#pragma unroll
    for (int fa = 0; fa < 4; ++fa)
#pragma unroll
      for (int fb = 0; fb < 4; ++fb)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int row = wm * 32 + 8 * fa + (lane >> 2), col = wn * 32 + 8 * fb + 2 * (lane & 3) + t;
          const int m = o0 + (X ? col : row);
          const long long v = v0 + (X ? row : col);
          if (m >= lim || v >= vn) continue;
          const long long q = (par ? ne : 0) + m;
          if (X)
            out[v * n + q] = acc[fa][fb][t];
          else
            out[q * I + v] = acc[fa][fb][t];
        }
  }
}

// x^e for e >= 0 by binary powering.
__device__ inline double ipow(double x, long long e) {
  double r = 1.0;
  while (e > 0) {
    if (e & 1) r *= x;
    x *= x;
    e >>= 1;
  }
  return r;
}

// The stopping-sweep search: the first d in [1, dmax] with f(d) <= tol^2
// (checked at the top of sweep d + 1 <= maxit).  Invariant: f(lo) > tol^2
// (lo = 0: no sweep yet), and f(hi) <= tol^2 when hi <= dmax (hi = dmax + 1:
// no passing d known).  The first evaluation doubles d from 1 up to the first
// power of two >= dmax; later ones take up to 32 candidates of (lo, hi) at
// equal steps, which leaves a bracket of ceil((hi - lo) / 33).  Without a
// passing d the iterate of sweep smax is kept, after f(smax) (its residual).
//
// Modes whose g^2 is at most g2_skip add at most 2^-60 tol^2 to any f(d) that
// an evaluation at equal steps takes (d > lo): sum over those modes of w
// g^(2d) <= g2_max^(d-1) f(1).  None is skipped while lo < 2 or f(1) is unknown.
__device__ void spec_advance(SpecState& Q, const double* f) {
  if (Q.phase == kSpecFinal) {
    Q.d = Q.smax;
    Q.converged = 0;
    Q.r2_hit = f[0];
    Q.done = 1;
    return;
  }
  const bool doubling = Q.phase == kSpecDoubling;
  if (doubling) Q.f1 = f[0];
  for (int t = 0; t < Q.count; ++t) {
    const long long d = doubling ? 1LL << t : Q.d0 + Q.step * t;
    if (d > Q.dmax) break;
    if (f[t] <= Q.tol2) {
      Q.hi = d;
      Q.r2_hit = f[t];
      break;
    }
    Q.lo = d;
  }
  if (Q.hi - Q.lo > 1) {
    Q.phase = kSpecUniform;
    Q.step = (Q.hi - Q.lo + kSpecPoints) / (kSpecPoints + 1);
    const long long cnt = (Q.hi - Q.lo - 1) / Q.step;
    Q.count = int(cnt < kSpecPoints ? cnt : kSpecPoints);
    Q.d0 = Q.lo + Q.step;
    Q.g2_skip = -1.0;
    if (Q.lo >= 2 && Q.f1 > 0.0 && Q.tol2 > 0.0) {
      const double ratio = Q.tol2 * 0x1p-60 / Q.f1;
      if (ratio < 1.0) Q.g2_skip = exp(log(ratio) / double(Q.lo - 1));
    }
  } else if (Q.hi <= Q.dmax) {
    Q.d = Q.hi;
    Q.done = 1;
  } else {
    Q.phase = kSpecFinal;
    Q.d0 = Q.smax;
    Q.step = 1;
    Q.count = 1;
    Q.g2_skip = -1.0;
  }
}

// What bounds it: the FP64 powers at large sizes, the final sum at small ones.
// 256 x 128 x 128 37 us (76 with 64-bit element indices, 160 shuffles a warp
// and a last block that read the partials one point at a time), 77^3 14 us (42).
//
// One step of the search: the Parseval sums f(d_t) = sum_m g_m^(2 d_t) rh_m^2
// at the sweep counts d_t = d0 2^t (the first evaluation) or d0 + t step, t <
// count.  Modes with g^2 <= g2_skip add nothing (spec_advance bounds what they
// could add far below the stop test's resolution).  Per-block partials in a
// fixed order; the last block to finish sums them, re-arms the counter and
// moves the search on.  A finished search returns at once.
template <class T>
__global__ void __launch_bounds__(kSpecThreads) spec_norms_kernel(const double* Rh, int nx, int ny,
                                                                  int nz, const double* __restrict__ omx,
                                                                  const double* __restrict__ omy,
                                                                  const double* __restrict__ omz,
                                                                  double* __restrict__ partial, unsigned int* counter,
                                                                  SpecState* state) {
  chain_begin();
  if (state->done) return;
  if (blockIdx.x == 0 && threadIdx.x == 0 && stamps_of(state)->search == 0) stamps_of(state)->search = global_ns();
  const long long d0 = state->d0, step = state->step;
  const int count = state->count, doubling = state->phase == kSpecDoubling;
  const double g2_skip = state->g2_skip;
  double acc[kSpecPoints];
#pragma unroll
  for (int t = 0; t < kSpecPoints; ++t) acc[t] = 0.0;
  const T n = T(nx) * T(ny) * T(nz);
  for (T q = T(blockIdx.x) * blockDim.x + threadIdx.x; q < n; q += T(gridDim.x) * blockDim.x) {
    int mx, my, mz;
    split3(q, nx, ny, mx, my, mz);
    const double g = 1.0 - (omx[mx] + omy[my] + omz[mz]);
    const double g2 = g * g;
    if (g2 <= g2_skip) continue;
    const double r = Rh[q];
    const double w = r * r;
    const double x = ipow(g2, d0);
    if (doubling) {
      double y = x;  // d0 * 2^t: a chain of squarings
#pragma unroll
      for (int t = 0; t < kSpecPoints; ++t) {
        if (t < count) acc[t] = fma(w, y, acc[t]);
        y *= y;
      }
    } else {
      // x h^t with h^t from the binary digits of t: 32 short independent
      // chains instead of one chain of 32 dependent products
      double hp[5];
      hp[0] = ipow(g2, step);
#pragma unroll
      for (int b = 1; b < 5; ++b) hp[b] = hp[b - 1] * hp[b - 1];
#pragma unroll
      for (int t = 0; t < kSpecPoints; ++t) {
        double y = x;
#pragma unroll
        for (int b = 0; b < 5; ++b)
          if (t & (1 << b)) y *= hp[b];
        if (t < count) acc[t] = fma(w, y, acc[t]);
      }
    }
  }
  __shared__ double sh[kSpecThreads / 32][kSpecPoints];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // transposed butterfly: 31 exchanges leave point `lane` of the warp in
  // acc[0], where 32 separate trees would take 160
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int t = 0; t < o; ++t) {
      const bool up = lane & o;
      const double give = up ? acc[t] : acc[t + o];
      acc[t] = (up ? acc[t + o] : acc[t]) + __shfl_xor_sync(0xffffffffu, give, o);
    }
  sh[wid][lane] = acc[0];
  __syncthreads();
  if (threadIdx.x < kSpecPoints) {
    double s = 0.0;
    for (int w2 = 0; w2 < kSpecThreads / 32; ++w2) s += sh[w2][threadIdx.x];
    partial[(long long)blockIdx.x * kSpecPoints + threadIdx.x] = s;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // the last block: out[t] = sum_b partial[b][t], warp w taking blocks w, w +
  // 8, ... (a row of 32 points per load) and the warps' sums added in order
  double s = 0.0;
#pragma unroll 8
  for (int b2 = wid; b2 < (int)gridDim.x; b2 += kSpecThreads / 32) s += __ldcg(partial + (long long)b2 * kSpecPoints + lane);
  sh[wid][lane] = s;
  __syncthreads();
  if (threadIdx.x < kSpecPoints) {
    double v = 0.0;
    for (int w2 = 0; w2 < kSpecThreads / 32; ++w2) v += sh[w2][threadIdx.x];
    sh[0][threadIdx.x] = v;  // this thread's own column
  }
  __syncwarp();
  if (threadIdx.x == 0) {
    *counter = 0u;
    SpecState Q = *state;
    spec_advance(Q, sh[0]);
    *state = Q;
  }
}

// rh -> -af (1 - g^d)/(1 - g) rh in place.  For g > 0 the factor is
// -expm1(d log1p(-omg))/omg (no cancellation near g = 1); a mode with
// omg == 0 (every axis periodic, the constant mode) takes d.
template <class T>
__global__ void spec_scale_kernel(double* Rh, int nx, int ny, int nz, const double* __restrict__ omx,
                                  const double* __restrict__ omy, const double* __restrict__ omz, double af,
                                  SpecState* state) {
  chain_begin();
  const long long d = state->d;
  if (state->trivial) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) stamps_of(state)->iterate = global_ns();
  const T n = T(nx) * T(ny) * T(nz);
  for (T q = T(blockIdx.x) * blockDim.x + threadIdx.x; q < n; q += T(gridDim.x) * blockDim.x) {
    int mx, my, mz;
    split3(q, nx, ny, mx, my, mz);
    const double omg = omx[mx] + omy[my] + omz[mz];
    // |g|^d <= exp(-d (1 - |g|)): below exp(-40) < 2^-57 it is nothing beside 1
    double f;
    if (omg == 0.0) {
      f = (double)d;
    } else if ((double)d * fmin(omg, 2.0 - omg) > 40.0) {
      f = 1.0 / omg;
    } else if (omg < 1.0) {
      f = -expm1((double)d * log1p(-omg)) / omg;
    } else {
      const double g = 1.0 - omg;  // in [-1, 0]
      f = (1.0 - ipow(g, d)) / omg;
    }
    Rh[q] = -af * f * Rh[q];
  }
}

int stream_blocks(long long n) {
  long long b = (n + kSpecThreads - 1) / kSpecThreads;
  return int(std::max<long long>(1, std::min<long long>(b, 148LL * 8)));
}

// The basis of one axis, folded (spec_axis_kernel): Pe[m][i] (ne x ne, the
// even functions on i < ne) and Po[m][i - s] (no x no, the odd ones on s <= i <
// no + s), and om, a_d (2 - sigma) per mode, in the order [even | odd].
//   open (s = 0): sqrt(2/(n+1)) sin(pi (f+1)(i+1)/(n+1)), even for even f;
//   periodic (s = 1): 1/sqrt(n), sqrt(2/n) cos(2 pi f i/n) and, n even,
//   (-1)^i/sqrt(n) even; sqrt(2/n) sin(2 pi f i/n) odd.
void folded_basis(int n, bool periodic, double a, AxisBasis& A, std::vector<double>& Pe, std::vector<double>& Po,
                  std::vector<double>& om) {
  const double pi = 3.14159265358979323846264338327950288;
  A.s = periodic ? 1 : 0;
  A.ne = periodic ? n / 2 + 1 : n - n / 2;
  A.no = n - A.ne;
  const int ne = A.ne, no = A.no;
  Pe.assign((size_t)ne * ne, 0.0);
  Po.assign((size_t)std::max(no, 1) * std::max(no, 1), 0.0);
  om.assign(n, 0.0);
  if (!periodic) {
    const double scale = std::sqrt(2.0 / (n + 1));
    const long long per = 2LL * (n + 1);
    for (int f = 0; f < n; ++f) {
      const int m = f / 2, cnt = f % 2 ? no : ne;
      for (int i = 0; i < cnt; ++i) {
        const long long p = ((long long)(f + 1) * (i + 1)) % per;  // sin(pi p/(n+1)) has period 2(n+1)
        (f % 2 ? Po[(size_t)m * no + i] : Pe[(size_t)m * ne + i]) = scale * std::sin(pi * (double)p / (double)(n + 1));
      }
      const double h = std::sin(pi * (f + 1) / (2.0 * (n + 1)));
      om[f % 2 ? ne + m : m] = a * 4.0 * h * h;  // a (2 - 2 cos(theta)) = 4 a sin^2(theta/2)
    }
    return;
  }
  for (int f = 0; f < ne; ++f) {
    const bool alone = f == 0 || 2 * f == n;
    for (int i = 0; i < ne; ++i) {
      const long long p = ((long long)f * i) % n;
      Pe[(size_t)f * ne + i] = f == 0       ? 1.0 / std::sqrt((double)n)
                               : 2 * f == n ? (i % 2 ? -1.0 : 1.0) / std::sqrt((double)n)
                                            : std::sqrt(2.0 / n) * std::cos(2.0 * pi * (double)p / n);
      if (!alone && i >= 1 && i <= no)
        Po[(size_t)(f - 1) * no + (i - 1)] = std::sqrt(2.0 / n) * std::sin(2.0 * pi * (double)p / n);
    }
    const double h = std::sin(pi * f / (double)n);
    om[f] = a * 4.0 * h * h;
    if (!alone) om[ne + f - 1] = om[f];
  }
}

void transpose(int n, const std::vector<double>& M, std::vector<double>& T) {
  T.assign(M.size(), 0.0);
  for (int r = 0; r < n; ++r)
    for (int c = 0; c < n; ++c) T[(size_t)c * n + r] = M[(size_t)r * n + c];
}

// One axis pass from `in` to `out` (out null: x, inverse, added to U's
// interior).  Axis d has outer extent O and inner extent I: x rows (I = 1), y
// O = nz slabs of nx columns, z one slab of nx ny columns.
cudaError_t axis_pass(picard_ctx* c, int d, bool forward, const double* in, double* out) {
  const SpectralPlan& S = c->spec;
  const AxisBasis& A = S.ax[d];
  const int nx = c->K.nx, ny = c->K.ny, nz = c->K.nz;
  const int n = d == 0 ? nx : d == 1 ? ny : nz;
  const long long I = d == 0 ? 1 : d == 1 ? nx : (long long)nx * ny;
  const int rows = d == 0 ? ny * nz : 0;
  auto tiles = [](long long v) { return (unsigned)((v + kAxTile - 1) / kAxTile); };
  const dim3 grid = d == 0 ? dim3(tiles(A.ne), tiles(rows)) : dim3(tiles(I), tiles(A.ne), d == 1 ? nz : 1);
  if (d == 0 && forward)
    return launch_chained(spec_axis_kernel<false, true, false>, grid, 256, 0, c->st, in, out, A.PeT, A.PoT, n, A.ne, A.no,
                          A.s, I, rows, c->K, nullptr, S.state);
  if (d == 0)
    return launch_chained(spec_axis_kernel<true, true, true>, grid, 256, 0, c->st, in, nullptr, A.Pe, A.Po, n, A.ne, A.no,
                          A.s, I, rows, c->K, c->U, S.state);
  if (forward)
    return launch_chained(spec_axis_kernel<false, false, false>, grid, 256, 0, c->st, in, out, A.Pe, A.Po, n, A.ne, A.no,
                          A.s, I, rows, c->K, nullptr, S.state);
  return launch_chained(spec_axis_kernel<true, false, false>, grid, 256, 0, c->st, in, out, A.PeT, A.PoT, n, A.ne, A.no,
                        A.s, I, rows, c->K, nullptr, S.state);
}

// Forward: Qz Qy Qx of T[0] into T[1] (x, y, z passes ping-ponging T[0] and
// T[1]); inverse: Qx^T Qy^T Qz^T of T[1], added to U's interior.
cudaError_t transform(picard_ctx* c, bool forward) {
  SpectralPlan& S = c->spec;
  cudaError_t e;
  if (forward) {
    if ((e = axis_pass(c, 0, true, S.T[0], S.T[1]))) return e;
    if ((e = axis_pass(c, 1, true, S.T[1], S.T[0]))) return e;
    return axis_pass(c, 2, true, S.T[0], S.T[1]);
  }
  if ((e = axis_pass(c, 2, false, S.T[1], S.T[0]))) return e;
  if ((e = axis_pass(c, 1, false, S.T[0], S.T[1]))) return e;
  return axis_pass(c, 0, false, S.T[1], nullptr);
}

// Evaluations that the search of spec_advance can need with this maxit: the
// doubling one, the ones at equal steps for the widest bracket it can leave,
// and f(smax).
int max_evaluations(int maxit) {
  if (maxit < 2) return 1;
  long long gap = 1;
  while (gap < maxit) gap <<= 1;
  int e = 2;
  for (; gap > 1; gap = (gap + kSpecPoints) / (kSpecPoints + 1)) ++e;
  return e;
}

}  // namespace

int spectral_alloc(picard_ctx* c) {
  SpectralPlan& S = c->spec;
  const KParams& K = c->K;
  const long long n = (long long)K.nx * K.ny * K.nz;
  const JacobiCoef J = jacobi_coef(K);
  const double a[3] = {J.ax, J.ay, J.az};
  const int len[3] = {K.nx, K.ny, K.nz};
  const bool per[3] = {!K.xflow, !K.yflow, !K.zflow};
  for (int d = 0; d < 3; ++d) {
    AxisBasis& A = S.ax[d];
    std::vector<double> Pe, Po, PeT, PoT, om;
    folded_basis(len[d], per[d], a[d], A, Pe, Po, om);
    transpose(A.ne, Pe, PeT);
    transpose(A.no, Po, PoT);
    double** dst[5] = {&A.Pe, &A.PeT, &A.Po, &A.PoT, &S.om[d]};
    const std::vector<double>* srcv[5] = {&Pe, &PeT, &Po, &PoT, &om};
    for (int t = 0; t < 5; ++t) {
      void* p = nullptr;
      PICARD_TRY(dev_alloc(c, &p, sizeof(double) * srcv[t]->size()));
      *dst[t] = static_cast<double*>(p);
      // no wait: an asynchronous copy from pageable memory returns once the
      // host data is staged, so the vectors may go out of scope
      PICARD_CUDA(cudaMemcpyAsync(*dst[t], srcv[t]->data(), sizeof(double) * srcv[t]->size(), cudaMemcpyHostToDevice,
                                  c->st));
      c->stats.h2d_bytes += (int64_t)(sizeof(double) * srcv[t]->size());
    }
  }
  void* p = nullptr;
  PICARD_TRY(dev_alloc(c, &p, sizeof(double) * n));
  S.T[0] = static_cast<double*>(p);
  PICARD_TRY(dev_alloc(c, &p, sizeof(double) * n));
  S.T[1] = static_cast<double*>(p);
  S.norm_blocks = std::min(stream_blocks(n), 148 * 4);
  PICARD_TRY(dev_alloc(c, &p, sizeof(double) * (size_t)S.norm_blocks * kSpecPoints));
  S.partial = static_cast<double*>(p);
  PICARD_TRY(dev_alloc(c, &p, kSpecBytes));
  S.state = static_cast<SpecState*>(p);
  PICARD_TRY(dev_alloc(c, &p, sizeof(unsigned int)));  // zeroed
  S.counter = static_cast<unsigned int*>(p);
  return PICARD_OK;
}

long long spectral_bytes(const KParams& K) {
  const long long n = (long long)K.nx * K.ny * K.nz;
  return 8LL * (2 * n + 2LL * ((long long)K.nx * K.nx + (long long)K.ny * K.ny + (long long)K.nz * K.nz) + K.nx +
                K.ny + K.nz + (long long)stream_blocks(n) * kSpecPoints + kSpecPoints);
}

int spec_issue(picard_ctx* c, double maxerr, int maxit) {
  SpectralPlan& S = c->spec;
  const KParams& K = c->K;
  const long long n = (long long)K.nx * K.ny * K.nz;
  const JacobiCoef J = jacobi_coef(K);
  const double ix = 1.0 / J.dx2, iy = 1.0 / J.dy2, iz = 1.0 / J.dz2, binv = 1.0 / (K.dV * kEps0);
  const int nb = stream_blocks(n);  // at most 32 norm_blocks partials
  if (S.queued - S.collected > 1) return fail(PICARD_ERR_STATE, "two closed-form solves are waiting to be collected");
  const int slot = S.queued & 1;
  auto* begin = fits32(n) ? spec_begin_kernel<unsigned> : spec_begin_kernel<long long>;
  PICARD_CUDA(launch_chained(begin, nb, kSpecThreads, 0, c->st, K, ix, iy, iz, binv, c->C, c->U, S.T[0], maxerr, maxit,
                             S.partial, S.counter, S.state));
  PICARD_CUDA(transform(c, true));
  auto* norms = fits32(n) ? spec_norms_kernel<unsigned> : spec_norms_kernel<long long>;
  for (int e = max_evaluations(maxit); e > 0; --e)
    PICARD_CUDA(launch_chained(norms, S.norm_blocks, kSpecThreads, 0, c->st, S.T[1], K.nx, K.ny, K.nz, S.om[0], S.om[1],
                               S.om[2], S.partial, S.counter, S.state));
  auto* scale = fits32(n) ? spec_scale_kernel<unsigned> : spec_scale_kernel<long long>;
  PICARD_CUDA(launch_chained(scale, nb, kSpecThreads, 0, c->st, S.T[1], K.nx, K.ny, K.nz, S.om[0], S.om[1], S.om[2],
                             J.af, S.state));
  PICARD_CUDA(transform(c, false));
  PICARD_CUDA(launch_refresh_periodic(c->K, c->U, c->st));
  PICARD_CUDA(cudaMemcpyAsync(c->h_pinned + kPinnedSpec + slot * kSpecSlots, S.state, kSpecBytes,
                              cudaMemcpyDeviceToHost, c->st));
  c->stats.d2h_bytes += kSpecBytes;
  ++S.queued;
  return PICARD_OK;
}

int spec_collect(picard_ctx* c, long long* sweeps) {
  *sweeps = 0;
  if (c->spec.queued == c->spec.collected) return PICARD_OK;
  const int slot = c->spec.collected++ & 1;
  SpecState Q;
  SpecStamps ns;
  std::memcpy(&Q, c->h_pinned + kPinnedSpec + slot * kSpecSlots, sizeof(Q));
  std::memcpy(&ns, c->h_pinned + kPinnedSpec + slot * kSpecSlots + sizeof(Q) / sizeof(double), sizeof(ns));
  if (!Q.trivial) {
    c->stats.spectral_transforms += 2;
    c->stats.spectral_transform_ms += 1e-6 * double((ns.search - ns.begin) + (ns.end - ns.iterate));
  }
  *sweeps = Q.d;
  return epot_account(c, Q.bnorm, Q.trivial ? Q.bnorm : std::sqrt(Q.r2_hit), Q.smax, Q.d, Q.converged != 0);
}

void spec_drain(picard_ctx* c, int64_t* sweeps_total) {
  if (c->spec.queued == c->spec.collected) return;
  if (cudaStreamSynchronize(c->st) != cudaSuccess) c->spec.collected = c->spec.queued;  // their results never came
  while (c->spec.queued != c->spec.collected) {
    long long sw = 0;
    (void)spec_collect(c, &sw);
    if (sweeps_total) *sweeps_total += sw;
  }
}

}  // namespace picard
