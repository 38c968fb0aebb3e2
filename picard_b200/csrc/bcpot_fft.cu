// bcpot_fft.cu -- BCpotentials (BCpotentials.f90:36-139) as FP64 FFT
// convolutions over the faces.
//
// The face potential of the reference is a direct sum over every interior
// cell; for the x0 face, node (0, j, k), with 0-based interior cells (a,b,c):
//   U = (2 tau eps0)^-1 sum_{a,b,c} C(a,b,c) D(a+1, b-j, c-k)
// and the x1 face takes D(a-Nx, ...) (BCpotentials.f90:53-63 with one rank;
// D(ox,oy,oz) the CalcDistance table, even in every offset).  For each plane
// a of cells along the face normal this is a 2-D correlation over the two
// tangential axes with the kernel slice D(s, ., .), s = a+1 (x0) or Nx-a (x1),
// so in the 2-D Fourier domain of the tangential axes (lengths LP, LQ: powers
// of two >= 2n-1, so the circular convolution reproduces every needed
// offset without wrap-around):
//   U^(kP,kQ) = sum_a C^_a(kP,kQ) E^_s(a)(kP,kQ)
// with E_s the slice laid out circularly; E_s is real and even, so its
// transform is real.  Per face pair: a real-to-complex FFT of every cell
// plane (rows along P keep LP/2+1 outputs, then columns along Q), the
// contraction over planes against the precomputed slice transforms (the
// constant (2 tau eps0)^-1 / (LP LQ) folded in), and one inverse FFT per face.
// FP64 throughout: FFTs of radix 8 and 4 in registers (fft_block), the
// twiddles computed on the host.  The slice transforms depend only on D and
// are computed on the first call after D changes.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "chain.cuh"
#include "context.cuh"

namespace picard {

namespace {

constexpr int kFftThreads = 256;
constexpr int kFftPer = 8;                           // elements per thread
constexpr int kFftElems = kFftThreads * kFftPer;     // elements per block: 2048 / L transforms of length L
constexpr int kMinLog = 3, kMaxLog = 11;             // transform lengths 8 .. 2048
constexpr int kMaxQ = 1024, kMaxP = 2048;            // accepted circular lengths along Q and P

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// a times -i (forward) or +i (inverse)
template <bool INV>
__device__ __forceinline__ double2 crot(double2 a) {
  return INV ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

// Transforms of length 4 and 8 in registers, natural order in and out.
template <bool INV>
__device__ __forceinline__ void fft4(double2& v0, double2& v1, double2& v2, double2& v3) {
  const double2 a = cadd(v0, v2), b = csub(v0, v2), c = cadd(v1, v3), d = crot<INV>(csub(v1, v3));
  v0 = cadd(a, c);
  v1 = cadd(b, d);
  v2 = csub(a, c);
  v3 = csub(b, d);
}
template <bool INV>
__device__ __forceinline__ void fft8(double2 v[8]) {
  const double h = 0.70710678118654752440;  // sqrt(1/2)
  fft4<INV>(v[0], v[2], v[4], v[6]);
  fft4<INV>(v[1], v[3], v[5], v[7]);
  const double2 o1 = v[3], o2 = v[5], o3 = v[7];  // the odd half, in its order 0, 1, 2, 3
  const double2 r1 = crot<INV>(o1), r3 = crot<INV>(o3);
  const double2 w1 = make_double2(h * (o1.x + r1.x), h * (o1.y + r1.y));
  const double2 w2 = crot<INV>(o2);
  const double2 w3 = make_double2(h * (r3.x - o3.x), h * (r3.y - o3.y));
  const double2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
  v[0] = cadd(e0, o0), v[4] = csub(e0, o0);
  v[1] = cadd(e1, w1), v[5] = csub(e1, w1);
  v[2] = cadd(e2, w2), v[6] = csub(e2, w2);
  v[3] = cadd(e3, w3), v[7] = csub(e3, w3);
}

// log2 of the radix of the pass that has `done` of `LOG` bits behind it: 8
// where three bits are left for it and the rest is not one bit, else 4 or 2.
__host__ __device__ constexpr int pass_bits(int left) {
  return left == 1 ? 1 : left == 2 || left == 4 ? 2 : 3;
}
constexpr int last_bits(int log) { return log <= 3 ? pass_bits(log) : last_bits(log - pass_bits(log)) ; }

// Shared index of element i of a transform: one 16-byte slot of padding for
// every eight, so that a pass's writes 8 apart fall into different banks.
__device__ __forceinline__ int fpad(int i) { return i + (i >> 3); }
// Slots per transform: odd, or for fewer than eight transforms per block 8 over
// their number mod 8, so that the transforms which a quarter-warp touches
// together lie in different banks.
template <int LOG>
__host__ __device__ constexpr int fstride() {
  constexpr int L = 1 << LOG, B = kFftElems / L, base = L + L / 8;
  if (B >= 8) return base | 1;
  constexpr int want = B == 4 ? 2 : B == 2 ? 4 : 0;
  return base + (want - base % 8 + 8) % 8;
}
template <int LOG>
constexpr size_t fsmem() {
  static_assert(sizeof(double2) * fstride<LOG>() * (kFftElems >> LOG) <= 48 * 1024, "default shared memory");
  return sizeof(double2) * (size_t)fstride<LOG>() * (kFftElems >> LOG);
}

// One Stockham pass of radix 2^BITS with 2^S of the length done, and the ones
// after it.  FIRST reads its inputs with load(b, i), the last one hands its
// outputs to store(u, b, i, value) (u: the element's number in the thread, the
// same for every call); between passes the block's transforms live in `x`.
// Butterflies are dealt with consecutive positions on consecutive threads, or,
// in the first pass with BLOAD and the last with BSTORE, with consecutive
// transforms.
template <int LOG, int S, bool INV, bool BLOAD, bool BSTORE, class Load, class Store>
__device__ __forceinline__ void fft_pass(double2* x, const double2* __restrict__ tw, Load&& load, Store&& store) {
  constexpr int BITS = pass_bits(LOG - S), R = 1 << BITS, NB = kFftPer / R, L = 1 << LOG, Ns = 1 << S;
  constexpr bool first = S == 0, last = S + BITS == LOG;
  constexpr int per = L >> BITS, B = kFftElems >> LOG;  // butterflies per transform, transforms per block
  constexpr bool bfast = (first && BLOAD) || (last && BSTORE && !first);
  double2 v[kFftPer];
#pragma unroll
  for (int u = 0; u < NB; ++u) {
    const int id = threadIdx.x + kFftThreads * u;
    const int b = bfast ? id % B : id / per, j = bfast ? id / B : id % per;
#pragma unroll
    for (int r = 0; r < R; ++r)
      v[u * R + r] = first ? load(b, j + r * per) : x[b * fstride<LOG>() + fpad(j + r * per)];
  }
#pragma unroll
  for (int u = 0; u < NB; ++u) {
    double2* w = v + u * R;
    if constexpr (!first) {
      const int id = threadIdx.x + kFftThreads * u;
      const int j = bfast ? id / B : id % per;
      const int k = (j & (Ns - 1)) << (LOG - S - BITS);
      auto twiddle = [&](int m) {
        double2 t = __ldg(tw + m * k);
        if (INV) t.y = -t.y;
        return t;
      };
      const double2 w1 = twiddle(1);
      w[1] = cmul(w[1], w1);
      if constexpr (R >= 4) {
        const double2 w2 = twiddle(2);
        const double2 w3 = cmul(w1, w2);
        w[2] = cmul(w[2], w2);
        w[3] = cmul(w[3], w3);
        if constexpr (R == 8) {
          const double2 w4 = twiddle(4);
          w[4] = cmul(w[4], w4);
          w[5] = cmul(w[5], cmul(w1, w4));
          w[6] = cmul(w[6], cmul(w2, w4));
          w[7] = cmul(w[7], cmul(w3, w4));
        }
      }
    }
    if constexpr (R == 8) {
      fft8<INV>(w);
    } else if constexpr (R == 4) {
      fft4<INV>(w[0], w[1], w[2], w[3]);
    } else {
      const double2 a = w[0];
      w[0] = cadd(a, w[1]);
      w[1] = csub(a, w[1]);
    }
  }
  if constexpr (!first) {
    if constexpr (!last) __syncthreads();  // every input of the pass is in registers
  }
#pragma unroll
  for (int u = 0; u < NB; ++u) {
    const int id = threadIdx.x + kFftThreads * u;
    const int b = bfast ? id % B : id / per, j = bfast ? id / B : id % per;
    const int idx = ((j & ~(Ns - 1)) << BITS) + (j & (Ns - 1));
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if constexpr (last)
        store(u * R + r, b, idx + r * Ns, v[u * R + r]);
      else
        x[b * fstride<LOG>() + fpad(idx + r * Ns)] = v[u * R + r];
    }
  }
  if constexpr (!last) {
    __syncthreads();
    fft_pass<LOG, S + BITS, INV, BLOAD, BSTORE>(x, tw, load, store);
  }
}

// What bounds the stages: latency at small sizes; at large ones the shared-memory
// pipe of the row transforms (75 % busy, an eighth of it conflicts) and, in the
// contraction, global loads that two blocks of 128 registers per SM do not hide
// (DRAM at a quarter of its rate).  Before, a stage was a
// generic radix-4 Stockham transform that crossed shared memory at every
// radix, in natural element order (30-44 % of its wavefronts were bank
// conflicts), with one real row per complex transform and a launch per face
// pair.  BCpotentials in us, before and now: 24^3 117 and 24, 77^3 378 and 93,
// 128^3 654 and 190, 256 x 128 x 128 1159 and 332, 200 x 140 x 140 2258 and 628.
//
// B = 2048 / L transforms of length L = 2^LOG (8 .. 2048) by the block: inputs
// load(b, i), outputs store(u, b, i, value), natural order, no scaling.  A
// length of up to 512 crosses shared memory at most twice.  The caller puts a
// block barrier between two calls on the same `x`.
template <int LOG, bool INV, bool BLOAD, bool BSTORE, class Load, class Store>
__device__ __forceinline__ void fft_block(double2* x, const double2* __restrict__ tw, Load&& load, Store&& store) {
  fft_pass<LOG, 0, INV, BLOAD, BSTORE>(x, tw, load, store);
}

// The stages of a run are chained launches (chain.cuh), so the bodies below read C
// and the stage buffers W, S and V by ordinary loads; the read-only path is for
// the twiddles and the slice transforms, which no kernel of the chain writes.

// Geometry of one face pair: A the normal axis, P and Q the tangential axes.
struct FaceGeom {
  int nA, nP, nQ;
  int LP, LQ, logP, logQ, HP;
  long long sA, sP, sQ;      // node-array strides (elements)
  long long dA, dP, dQ;      // D-table strides
  long long d0;              // D-table index of offset (0, 0, 0)
  long long base;            // node index of interior cell (0, 0, 0)
  long long face0, face1;    // node index of face node (p, q) = (0, 0) on the two faces
  int G;                     // plane groups of the contraction
};

// Distance along a circular axis of length L to offset index t (the kernel
// slice is nonzero for |offset| < n).
__device__ inline int circ_off(int t, int L, int n, bool& ok) {
  const int d = t <= L - t ? t : L - t;
  ok = d < n;
  return d;
}

// Stage 1: FFT along P of rows, two real rows in one complex transform: the
// block takes the row pairs (2 m, 2 m + 1) of plane index a for m in [bx B, bx B
// + B).  mode 0: the charge rows (a, q), q = by < nQ, from C; mode 1: the
// kernel rows (s, tQ) of slices s0 + a (a < count), tQ = by < LQ, from D.
// Output W[(a * rowsQ + q) * HP + kP], kP < HP.
template <int LOG>
__device__ void bcfft_rows_body(const FaceGeom& F, int mode, const double* src, int s0, int count,
                                const double2* __restrict__ tw, double2* W, int bx, int by) {
  extern __shared__ double2 smem[];
  constexpr int L = 1 << LOG, B = kFftElems >> LOG;
  const int q = by;
  const int rowsQ = mode == 0 ? F.nQ : F.LQ;
  const int na = mode == 0 ? F.nA : count;
  const int a0 = 2 * bx * B;
  bool okq = true;
  int dq = 0;
  if (mode == 1) dq = circ_off(q, F.LQ, F.nQ, okq);
  auto load = [&](int b, int p) {
    const int a = a0 + 2 * b;
    double2 v = make_double2(0.0, 0.0);
    if (mode == 0) {
      if (p < F.nP && a < na) {
        const double* c = src + (F.base + (long long)a * F.sA + (long long)p * F.sP + (long long)q * F.sQ);
        v.x = c[0];
        if (a + 1 < na) v.y = c[F.sA];
      }
    } else {
      bool okp;
      const int dp = circ_off(p, L, F.nP, okp);
      if (okp && okq && a < na) {
        const double* d = src + (F.d0 + (long long)(s0 + a) * F.dA + (long long)dp * F.dP + (long long)dq * F.dQ);
        v.x = d[0];
        if (a + 1 < na) v.y = d[F.dA];
      }
    }
    return v;
  };
  // the spectrum of the pair back to shared memory: both rows need Z[k] and Z[L - k]
  double2 z[kFftPer];
  int zb[kFftPer], zi[kFftPer];
  auto keep = [&](int u, int b, int i, double2 v) {
    z[u] = v;
    zb[u] = b;
    zi[u] = i;
  };
  if (F.sA == 1 && mode == 0)
    fft_block<LOG, false, true, false>(smem, tw, load, keep);
  else
    fft_block<LOG, false, false, false>(smem, tw, load, keep);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kFftPer; ++u) smem[zb[u] * fstride<LOG>() + fpad(zi[u])] = z[u];
  __syncthreads();
  constexpr int HP = L / 2 + 1;
  for (int e = threadIdx.x; e < B * HP; e += kFftThreads) {
    const int b = e / HP, k = e - b * HP, a = a0 + 2 * b;
    if (a >= na) break;
    const double2 p = smem[b * fstride<LOG>() + fpad(k)], m = smem[b * fstride<LOG>() + fpad((L - k) & (L - 1))];
    double2* w = W + ((long long)a * rowsQ + q) * HP + k;
    w[0] = make_double2(0.5 * (p.x + m.x), 0.5 * (p.y - m.y));
    if (a + 1 < na) w[(long long)rowsQ * HP] = make_double2(0.5 * (p.y + m.y), 0.5 * (m.x - p.x));
  }
}

// Plane t of the contraction's order: 0, nA - 1, 1, nA - 2, ... so that the
// slices of D that a plane reads for its two faces serve the next one too.
__device__ __forceinline__ int plane_at(int t, int nA) { return t & 1 ? nA - 1 - (t >> 1) : t >> 1; }

// Stage 2: FFT along Q of the columns kP in [bx B, bx B + B).
// mode 0 (contraction): the planes of group by; each thread keeps the sums of
// its (kP, kQ) elements against Dh[s0(a)] and Dh[s1(a)] and writes the group's
// partial to S[(g * 2 + f) * HP * LQ + kP * LQ + kQ].
// mode 1 (kernel transforms): slice by < count of W, real part times scale to
// Dh[(s0 + by) * HP * LQ + kP * LQ + kQ].
template <int LOG>
__device__ void bcfft_cols_body(const FaceGeom& F, int mode, const double2* W, int s0, int count, double scale,
                                const double2* __restrict__ tw, double* Dh, double2* S, int bx, int by) {
  extern __shared__ double2 smem[];
  constexpr int L = 1 << LOG, B = kFftElems >> LOG;
  const int k0 = bx * B;
  const int rowsQ = mode == 0 ? F.nQ : L;
  const long long plane = (long long)F.HP * L;
  const int per = (F.nA + F.G - 1) / F.G;
  const int t_lo = mode == 0 ? by * per : by, t_hi = mode == 0 ? min(F.nA, t_lo + per) : min(count, t_lo + 1);
  double2 acc0[kFftPer], acc1[kFftPer];
#pragma unroll
  for (int u = 0; u < kFftPer; ++u) acc0[u] = acc1[u] = make_double2(0.0, 0.0);
  for (int t = t_lo; t < t_hi; ++t) {
    const int a = mode == 0 ? plane_at(t, F.nA) : t;
    const double2* w = W + (long long)a * rowsQ * F.HP + k0;
    auto load = [&](int b, int q) {
      return k0 + b < F.HP && q < rowsQ ? w[(long long)q * F.HP + b] : make_double2(0.0, 0.0);
    };
    if (t > t_lo) __syncthreads();  // the plane before has read its last shared element
    if (mode == 0) {
      const double* d0 = Dh + (long long)a * plane + (long long)k0 * L;                // s = a + 1
      const double* d1 = Dh + (long long)(F.nA - 1 - a) * plane + (long long)k0 * L;   // s = nA - a
      fft_block<LOG, false, true, false>(smem, tw, load, [&](int u, int b, int kq, double2 v) {
        if (k0 + b < F.HP) {
          const double e0 = __ldg(d0 + b * L + kq), e1 = __ldg(d1 + b * L + kq);
          acc0[u].x = fma(v.x, e0, acc0[u].x);
          acc0[u].y = fma(v.y, e0, acc0[u].y);
          acc1[u].x = fma(v.x, e1, acc1[u].x);
          acc1[u].y = fma(v.y, e1, acc1[u].y);
        }
      });
    } else {
      double* d = Dh + (long long)(s0 + a) * plane + (long long)k0 * L;
      fft_block<LOG, false, true, false>(smem, tw, load, [&](int, int b, int kq, double2 v) {
        if (k0 + b < F.HP) d[b * L + kq] = v.x * scale;
      });
    }
  }
  if (mode != 0) return;
  // the elements of the last pass, in its order
  constexpr int BITS = last_bits(LOG), R = 1 << BITS, lastper = L >> BITS;
#pragma unroll
  for (int u = 0; u < kFftPer; ++u) {
    const int id = threadIdx.x + kFftThreads * (u / R), b = id / lastper, kq = id % lastper + (u % R) * lastper;
    if (k0 + b < F.HP) {
      const long long e = (long long)(k0 + b) * L + kq;
      S[((long long)by * 2 + 0) * plane + e] = acc0[u];
      S[((long long)by * 2 + 1) * plane + e] = acc1[u];
    }
  }
}

// Stage 3a: sum of the group partials (fixed order) and the inverse FFT along
// Q of columns kP in [bx B, bx B + B) of face f = by; V[(f*nQ + q)*HP + kP] for
// q < nQ.
template <int LOG>
__device__ void bcfft_invq_body(const FaceGeom& F, const double2* S, const double2* __restrict__ tw, double2* V,
                                int bx, int by) {
  extern __shared__ double2 smem[];
  constexpr int L = 1 << LOG, B = kFftElems >> LOG;
  const int k0 = bx * B, f = by;
  const long long plane = (long long)F.HP * L;
  fft_block<LOG, true, false, true>(
      smem, tw,
      [&](int b, int kq) {
        double2 v = make_double2(0.0, 0.0);
        if (k0 + b < F.HP) {
          const double2* s = S + (long long)f * plane + (long long)(k0 + b) * L + kq;
#pragma unroll 4
          for (int g = 0; g < F.G; ++g) {
            const double2 e = s[(long long)g * 2 * plane];
            v.x += e.x;
            v.y += e.y;
          }
        }
        return v;
      },
      [&](int, int b, int q, double2 v) {
        if (k0 + b < F.HP && q < F.nQ) V[((long long)f * F.nQ + q) * F.HP + k0 + b] = v;
      });
}

// Stage 3b: inverse real FFT along P of the row pairs (2 m, 2 m + 1) of face f =
// by, m in [bx B, bx B + B) (the spectrum's upper half from Hermitian
// symmetry): two real rows as the real and imaginary part of one transform.
template <int LOG>
__device__ void bcfft_invp_body(const FaceGeom& F, const double2* V, const double2* __restrict__ tw, double* U,
                                int bx, int by) {
  extern __shared__ double2 smem[];
  constexpr int L = 1 << LOG, B = kFftElems >> LOG, HP = L / 2 + 1;
  const int q0 = 2 * bx * B, f = by;
  const long long face = f == 0 ? F.face0 : F.face1;
  fft_block<LOG, true, false, false>(
      smem, tw,
      [&](int b, int k) {
        const int q = q0 + 2 * b;
        double2 z = make_double2(0.0, 0.0);
        if (q < F.nQ) {
          const bool up = k >= HP;
          const double2* r = V + ((long long)f * F.nQ + q) * HP + (up ? L - k : k);
          double2 v = r[0], w = q + 1 < F.nQ ? r[HP] : make_double2(0.0, 0.0);
          if (up) v.y = -v.y, w.y = -w.y;
          z = make_double2(v.x - w.y, v.y + w.x);  // v + i w
        }
        return z;
      },
      [&](int, int b, int p, double2 v) {
        const int q = q0 + 2 * b;
        if (p < F.nP && q < F.nQ) {
          double* u = U + (face + (long long)p * F.sP + (long long)q * F.sQ);
          u[0] = v.x;
          if (q + 1 < F.nQ) u[F.sQ] = v.y;
        }
      });
}

// One face pair in a launch: its geometry and buffers, and per stage (rows,
// columns + contraction, inverse along Q, inverse along P) the first block of
// its blocks in the launch and its blocks along x.
struct FftJob {
  FaceGeom F;
  const double* C;
  double2* W;
  const double2* twP;
  const double2* twQ;
  double* Dh;
  double2* S;
  double2* V;
  double* U;
  long long start[4];
  int bx[4];
};

template <int STAGE, int LOG>
__device__ __forceinline__ void bcfft_stage(const FftJob& J, int bx, int by) {
  const FaceGeom F = J.F;
  if constexpr (STAGE == 0) bcfft_rows_body<LOG>(F, 0, J.C, 0, F.nA, J.twP, J.W, bx, by);
  else if constexpr (STAGE == 1) bcfft_cols_body<LOG>(F, 0, J.W, 0, 0, 0.0, J.twQ, J.Dh, J.S, bx, by);
  else if constexpr (STAGE == 2) bcfft_invq_body<LOG>(F, J.S, J.twQ, J.V, bx, by);
  else bcfft_invp_body<LOG>(F, J.V, J.twP, J.U, bx, by);
}

// The blocks of one face pair in a stage of a batched launch.
struct FftSeg {
  long long start;  // its first block
  int job, bx;
};

// One stage of length 2^LOG for a table of face pairs in one launch: block b
// belongs to the segment with the largest start <= b (binary search), and runs
// block (local % bx, local / bx) of that job's stage.
template <int STAGE, int LOG>
__global__ void __launch_bounds__(kFftThreads, 2) bcfft_table_kernel(const FftJob* __restrict__ jobs,
                                                                     const FftSeg* __restrict__ segs, int n) {
  const long long b = blockIdx.x;
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (segs[mid].start <= b) lo = mid;
    else hi = mid - 1;
  }
  const FftSeg g = segs[lo];
  const long long local = b - g.start;
  bcfft_stage<STAGE, LOG>(jobs[g.job], int(local % g.bx), int(local / g.bx));
}

// The same for up to three face pairs of one run, the table in the parameters.
struct FftJobs3 {
  FftJob j[3];
  int n;
};
template <int STAGE, int LOG>
__global__ void __launch_bounds__(kFftThreads, 2) bcfft_run_kernel(const __grid_constant__ FftJobs3 T) {
  chain_begin();
  const long long b = blockIdx.x;
  int q = 0;
  while (q + 1 < T.n && T.j[q + 1].start[STAGE] <= b) ++q;
  const FftJob& J = T.j[q];
  const long long local = b - J.start[STAGE];
  bcfft_stage<STAGE, LOG>(J, int(local % J.bx[STAGE]), int(local / J.bx[STAGE]));
}

// Slice transforms (mode 1 of the row and column stages).
template <int LOG>
__global__ void __launch_bounds__(kFftThreads, 2) bcfft_slice_rows_kernel(FaceGeom F, const double* __restrict__ D,
                                                                          int s0, int count,
                                                                          const double2* __restrict__ tw,
                                                                          double2* __restrict__ W) {
  bcfft_rows_body<LOG>(F, 1, D, s0, count, tw, W, blockIdx.x, blockIdx.y);
}
template <int LOG>
__global__ void __launch_bounds__(kFftThreads, 2) bcfft_slice_cols_kernel(FaceGeom F, const double2* __restrict__ W,
                                                                          int s0, int count, double scale,
                                                                          const double2* __restrict__ tw,
                                                                          double* __restrict__ Dh) {
  bcfft_cols_body<LOG>(F, 1, W, s0, count, scale, tw, Dh, nullptr, blockIdx.x, blockIdx.y);
}

// f(std::integral_constant<int, log>) for the run-time length 2^log.
template <int LOG = kMinLog, class Fn>
int with_log(int log, Fn&& f) {
  if constexpr (LOG <= kMaxLog) {
    if (log == LOG) return f(std::integral_constant<int, LOG>());
    return with_log<LOG + 1>(log, f);
  } else {
    return fail(PICARD_ERR_BAD_ARG, "FFT BCpotentials: unsupported transform length");
  }
}

int pow2_at_least(int v) {
  int L = 1;
  while (L < v) L <<= 1;
  return L;
}
int ilog2(int L) {
  int l = 0;
  while ((1 << l) < L) ++l;
  return l;
}

int col_blocks(const FaceGeom& F) { return (F.HP + (kFftElems >> F.logQ) - 1) / (kFftElems >> F.logQ); }
// blocks of row pairs
int pair_blocks(const FaceGeom& F, int rows) { return (rows + 2 * (kFftElems >> F.logP) - 1) / (2 * (kFftElems >> F.logP)); }

// Whether the face pairs go through the row and contraction stages together:
// while their row transforms fit the L2 cache with room to spare.  Else one
// after another, so that each contraction finds its own row transforms in L2 and has
// three times the plane groups (face_geom).  BCpotentials in us, one after another
// and together: 64^3 (14 MB) 87 / 50, 64 x 128 x 100 (38 MB) 138 / 99, 60 x 60 x 250
// (45 MB) 173 / 163, 96^3 (54 MB) 141 / 117; above the line 100 x 200 x 80 (94 MB)
// 242 / 395, 120 x 120 x 150 (106 MB) 262 / 414, 256 x 128 x 128 (164 MB) 332 / 355.
// Pairs of equal transform lengths, which share their launches, gain from going
// together up to 97 MB (128^3 190 / 163), pairs of unequal ones lose from 54 MB on
// (100 x 130 x 60 177 / 248).
bool faces_together(const KParams& K) {
  auto half = [](int n) { return pow2_at_least(2 * n - 1) / 2 + 1LL; };
  const long long elems = (long long)K.nx * K.nz * half(K.ny) + (long long)K.ny * K.nz * half(K.nx) +
                          (long long)K.nz * K.ny * half(K.nx);
  return 16 * elems <= (64LL << 20);
}

FaceGeom face_geom(const KParams& K, int axis) {
  const int n[3] = {K.nx, K.ny, K.nz};
  const long long s[3] = {1, K.nxp, (long long)K.nxp * K.nyp};
  const long long DX = 2LL * K.nx + 1, DY = 2LL * K.ny + 1;
  const long long ds[3] = {1, DX, DX * DY};
  const int P = axis == 0 ? 1 : 0, Q = axis == 2 ? 1 : 2;
  FaceGeom F;
  F.nA = n[axis];
  F.nP = n[P];
  F.nQ = n[Q];
  F.LP = std::max(1 << kMinLog, pow2_at_least(2 * F.nP - 1));
  F.LQ = std::max(1 << kMinLog, pow2_at_least(2 * F.nQ - 1));
  F.logP = ilog2(F.LP);
  F.logQ = ilog2(F.LQ);
  F.HP = F.LP / 2 + 1;
  F.sA = s[axis];
  F.sP = s[P];
  F.sQ = s[Q];
  F.dA = ds[axis];
  F.dP = ds[P];
  F.dQ = ds[Q];
  F.d0 = (long long)K.nx + DX * ((long long)K.ny + DY * (long long)K.nz);
  F.base = 1 + K.nxp * (1 + (long long)K.nyp * 1);
  F.face0 = F.base - F.sA;                       // plane 0 along A, tangential (1, 1)
  F.face1 = F.base + (long long)F.nA * F.sA;     // plane nA + 1
  // plane groups of the contraction: two blocks per SM, counting the other face
  // pairs of a launch; on small grids no more than eight partials, which the
  // inverse along Q sums before it starts.  BCpotentials in us with at most 4 / 8 /
  // 16 / 32 groups: 24^3 29.2 / 29.1 / 29.7 / 32.5, 40^3 48 / 37.6 / 38.4 / 43.9, 64^3 59
  // / 50.2 / 44.4 / 50.0, 128^3 405 / 252 / 185 / 190 (72^3 and 96^3 fill the SMs with
  // eight)
  const int share = col_blocks(F) * (faces_together(K) ? 3 : 1);
  F.G = std::max(1, std::min(std::min(F.nA, F.nA <= 64 ? 8 : 32), 2 * 148 / share));
  return F;
}

bool fits(const FaceGeom& F) { return F.LP <= kMaxP && F.LQ <= kMaxQ; }

}  // namespace

// Device scratch of the FFT BCpotentials: per face axis the slice transforms,
// shared stage buffers, twiddle tables.
long long bcpot_fft_bytes(const KParams& K) {
  const int flows[3] = {K.xflow, K.yflow, K.zflow};
  long long dh = 0, w = 0, s = 0, v = 0, tw = 0;
  for (int a = 0; a < 3; ++a) {
    if (!flows[a]) continue;
    FaceGeom F = face_geom(K, a);
    dh += (long long)F.nA * F.HP * F.LQ * 8;
    w += std::max((long long)F.nA * F.nQ, (long long)F.LQ) * F.HP * 16;
    s += (long long)F.G * 2 * F.HP * F.LQ * 16;
    v += 2LL * F.nQ * F.HP * 16;
    tw += (long long)(F.LP + F.LQ) * 16;
  }
  return dh + w + s + v + tw;
}

int bcpot_fft_supported(const KParams& K) {
  const int flows[3] = {K.xflow, K.yflow, K.zflow};
  for (int a = 0; a < 3; ++a)
    if (flows[a] && !fits(face_geom(K, a))) return 0;
  return 1;
}

namespace {

// One face pair's plan and buffers: its own stage buffers, so that the face
// pairs of a run can go through a batched stage at the same time.
struct AxisPlan {
  FaceGeom F;
  double* Dh = nullptr;
  double2* twP = nullptr;
  double2* twQ = nullptr;
  double2* W = nullptr;  // row transforms
  long long w_elems = 0;
  double2* S = nullptr;  // the contraction's group partials
  double2* V = nullptr;  // face spectra after the inverse along Q
};

void twiddles(int L, std::vector<double2>& t) {
  const double pi = 3.14159265358979323846264338327950288;
  t.assign(std::max(1, L), make_double2(1.0, 0.0));
  for (int k = 0; k < L; ++k) {
    // exp(-2 pi i k / L) from the FP64 cosine and sine of the angle
    const double ang = 2.0 * pi * (double)k / (double)L;
    t[k] = make_double2(std::cos(ang), -std::sin(ang));
  }
}

}  // namespace

struct BcFft {
  AxisPlan ax[3];
  bool ready = false;  // slice transforms of the current D
};

int bcpot_fft_alloc(picard_ctx* c) {
  if (c->bcfft) return PICARD_OK;
  if (!bcpot_fft_supported(c->K)) return fail(PICARD_ERR_BAD_ARG, "FFT BCpotentials: a face is longer than 1024 cells");
  BcFft* B = new BcFft();
  c->bcfft = B;
  const KParams& K = c->K;
  const int flows[3] = {K.xflow, K.yflow, K.zflow};
  for (int a = 0; a < 3; ++a) {
    if (!flows[a]) continue;
    AxisPlan& A = B->ax[a];
    A.F = face_geom(K, a);
    const FaceGeom& F = A.F;
    void* p = nullptr;
    PICARD_TRY(dev_alloc(c, &p, sizeof(double) * (size_t)F.nA * F.HP * F.LQ));
    A.Dh = static_cast<double*>(p);
    std::vector<double2> t;
    twiddles(F.LP, t);
    PICARD_TRY(dev_alloc(c, &p, sizeof(double2) * t.size()));
    A.twP = static_cast<double2*>(p);
    // no wait: an asynchronous copy from pageable memory returns once the host
    // data is staged, so the vector may be refilled
    PICARD_CUDA(cudaMemcpyAsync(A.twP, t.data(), sizeof(double2) * t.size(), cudaMemcpyHostToDevice, c->st));
    c->stats.h2d_bytes += (int64_t)(sizeof(double2) * t.size());
    twiddles(F.LQ, t);
    PICARD_TRY(dev_alloc(c, &p, sizeof(double2) * t.size()));
    A.twQ = static_cast<double2*>(p);
    PICARD_CUDA(cudaMemcpyAsync(A.twQ, t.data(), sizeof(double2) * t.size(), cudaMemcpyHostToDevice, c->st));
    c->stats.h2d_bytes += (int64_t)(sizeof(double2) * t.size());
    // at least one kernel slice's rows, for the slice transforms
    const long long w = std::max((long long)F.nA * F.nQ, (long long)F.LQ) * F.HP;
    PICARD_TRY(dev_alloc(c, &p, sizeof(double2) * (size_t)w));
    A.W = static_cast<double2*>(p);
    A.w_elems = w;
    PICARD_TRY(dev_alloc(c, &p, sizeof(double2) * (size_t)F.G * 2 * F.HP * F.LQ));
    A.S = static_cast<double2*>(p);
    PICARD_TRY(dev_alloc(c, &p, sizeof(double2) * 2 * (size_t)F.nQ * F.HP));
    A.V = static_cast<double2*>(p);
  }
  return PICARD_OK;
}

void bcpot_fft_free(picard_ctx* c) {
  delete c->bcfft;
  c->bcfft = nullptr;
}

void bcpot_fft_invalidate(picard_ctx* c) {
  if (c->bcfft) c->bcfft->ready = false;
}

// Slice transforms of D for every face axis: chunks of slices through the
// row and column stages (mode 1).
static int prepare(picard_ctx* c) {
  BcFft* B = c->bcfft;
  const double K0 = 1.0 / (2.0 * kTau * kEps0);
  for (int a = 0; a < 3; ++a) {
    AxisPlan& A = B->ax[a];
    if (!A.Dh) continue;
    const FaceGeom& F = A.F;
    const double scale = K0 / ((double)F.LP * (double)F.LQ);
    const int chunk = int(std::max<long long>(1, A.w_elems / ((long long)F.LQ * F.HP)));
    for (int s0 = 0; s0 < F.nA; s0 += chunk) {
      const int cnt = std::min(chunk, F.nA - s0);
      note_launch();
      // slice index a <-> normal offset s0 + a + 1 (the D table at offset a + 1 along A)
      PICARD_TRY(with_log(F.logP, [&](auto lg) {
        constexpr int LOG = decltype(lg)::value;
        bcfft_slice_rows_kernel<LOG><<<dim3(pair_blocks(F, cnt), F.LQ), kFftThreads, fsmem<LOG>(), c->st>>>(
            F, c->D + F.dA, s0, cnt, A.twP, A.W);
        return check_cuda(cudaGetLastError(), "bcfft_slice_rows_kernel");
      }));
      note_launch();
      PICARD_TRY(with_log(F.logQ, [&](auto lg) {
        constexpr int LOG = decltype(lg)::value;
        bcfft_slice_cols_kernel<LOG><<<dim3(col_blocks(F), cnt), kFftThreads, fsmem<LOG>(), c->st>>>(
            F, A.W, s0, cnt, scale, A.twQ, A.Dh);
        return check_cuda(cudaGetLastError(), "bcfft_slice_cols_kernel");
      }));
    }
  }
  B->ready = true;
  return PICARD_OK;
}

namespace {

FftJob make_job(picard_ctx* c, const AxisPlan& A) {
  FftJob J;
  J.F = A.F;
  J.C = c->C;
  J.W = A.W;
  J.twP = A.twP;
  J.twQ = A.twQ;
  J.Dh = A.Dh;
  J.S = A.S;
  J.V = A.V;
  J.U = c->U;
  const FaceGeom& F = A.F;
  J.bx[0] = pair_blocks(F, F.nA);
  J.bx[1] = J.bx[2] = col_blocks(F);
  J.bx[3] = pair_blocks(F, F.nQ);
  return J;
}
int stage_rows(const FaceGeom& F, int stage) { return stage == 0 ? F.nQ : stage == 1 ? F.G : 2; }
int stage_log(const FaceGeom& F, int stage) { return stage == 0 || stage == 3 ? F.logP : F.logQ; }

template <int STAGE>
int launch_run_stage(FftJobs3& T, int log, long long blocks, cudaStream_t st) {
  return with_log(log, [&](auto lg) {
    constexpr int LOG = decltype(lg)::value;
    return check_cuda(launch_chained(bcfft_run_kernel<STAGE, LOG>, (unsigned)blocks, kFftThreads, fsmem<LOG>(), st, T),
                      "bcfft_run_kernel");
  });
}
// Stages [STAGE, END) of jobs [first, last) of `J`, one launch per stage and
// transform length.
template <int STAGE, int END>
int run_stages(const std::vector<FftJob>& J, size_t first, size_t last, cudaStream_t st) {
  if constexpr (STAGE < END) {
    for (int log = kMinLog; log <= kMaxLog; ++log) {
      FftJobs3 T;
      T.n = 0;
      long long blocks = 0;
      for (size_t q = first; q < last; ++q) {
        const FftJob& j = J[q];
        if (stage_log(j.F, STAGE) != log) continue;
        T.j[T.n] = j;
        T.j[T.n].start[STAGE] = blocks;
        blocks += (long long)j.bx[STAGE] * stage_rows(j.F, STAGE);
        ++T.n;
      }
      if (T.n) PICARD_TRY(launch_run_stage<STAGE>(T, log, blocks, st));
    }
    return run_stages<STAGE + 1, END>(J, first, last, st);
  }
  return PICARD_OK;
}

}  // namespace

int bc_potentials_fft(picard_ctx* c) {
  PICARD_TRY(bcpot_fft_alloc(c));
  BcFft* B = c->bcfft;
  if (!B->ready) PICARD_TRY(prepare(c));
  PICARD_CUDA(launch_zero(c->U, c->K.nodes, c->st));  // BCpotentials.f90:36
  std::vector<FftJob> jobs;
  for (int a = 0; a < 3; ++a)
    if (B->ax[a].Dh) jobs.push_back(make_job(c, B->ax[a]));
  const size_t n = jobs.size(), step = faces_together(c->K) ? 3 : 1;
  for (size_t q = 0; q < n; q += step) PICARD_TRY((run_stages<0, 2>(jobs, q, std::min(n, q + step), c->st)));
  PICARD_TRY((run_stages<2, 4>(jobs, 0, n, c->st)));
  return PICARD_OK;
}

namespace {

// The stages of a whole batch, one launch per stage and transform length that
// occurs; segs[stage][log]: [first, last) of its segments in the table.
struct SegRange {
  int first = 0, count = 0;
  long long blocks = 0;
};
template <int STAGE = 0>
int table_stages(const FftJob* jobs, const FftSeg* segs, const SegRange (*range)[kMaxLog + 1], cudaStream_t st) {
  if constexpr (STAGE < 4) {
    for (int log = kMinLog; log <= kMaxLog; ++log) {
      const SegRange& r = range[STAGE][log];
      if (!r.count) continue;
      note_launch();
      PICARD_TRY(with_log(log, [&](auto lg) {
        constexpr int LOG = decltype(lg)::value;
        bcfft_table_kernel<STAGE, LOG><<<(unsigned)r.blocks, kFftThreads, fsmem<LOG>(), st>>>(jobs, segs + r.first,
                                                                                              r.count);
        return check_cuda(cudaGetLastError(), "bcfft_table_kernel");
      }));
    }
    return table_stages<STAGE + 1>(jobs, segs, range, st);
  }
  return PICARD_OK;
}

}  // namespace

// BCpotentials of many runs: the FFT runs' face pairs advance stage by stage,
// each stage one launch per transform length over all of them on the batch
// stream (after every such run's U is zeroed and its slice transforms exist,
// on its own stream); the other runs take their own method on their own
// streams.
int bc_potentials_batch(picard_ctx** ctxs, int n, cudaStream_t bst, cudaEvent_t* rev, cudaEvent_t bev) {
  std::vector<FftJob> jobs;
  std::vector<int> fft_runs;
  for (int r = 0; r < n; ++r) {
    picard_ctx* c = ctxs[r];
    if (c->bcpot_tensor != PICARD_BCPOT_FFT) {
      PICARD_TRY(bc_potentials_async(c));
      continue;
    }
    PICARD_TRY(bcpot_fft_alloc(c));
    BcFft* B = c->bcfft;
    if (!B->ready) PICARD_TRY(prepare(c));
    PICARD_CUDA(launch_zero(c->U, c->K.nodes, c->st));  // BCpotentials.f90:36
    PICARD_CUDA(cudaEventRecord(rev[r], c->st));
    PICARD_CUDA(cudaStreamWaitEvent(bst, rev[r], 0));
    fft_runs.push_back(r);
    for (int a = 0; a < 3; ++a)
      if (B->ax[a].Dh) jobs.push_back(make_job(c, B->ax[a]));
  }
  if (jobs.empty()) return PICARD_OK;
  std::vector<FftSeg> segs;
  SegRange range[4][kMaxLog + 1];
  for (int stage = 0; stage < 4; ++stage)
    for (int log = kMinLog; log <= kMaxLog; ++log) {
      SegRange& r = range[stage][log];
      r.first = (int)segs.size();
      for (size_t q = 0; q < jobs.size(); ++q) {
        if (stage_log(jobs[q].F, stage) != log) continue;
        segs.push_back(FftSeg{r.blocks, (int)q, jobs[q].bx[stage]});
        r.blocks += (long long)jobs[q].bx[stage] * stage_rows(jobs[q].F, stage);
      }
      r.count = (int)segs.size() - r.first;
    }
  // the table lives on the batch stream until its last launch
  const size_t jb = sizeof(FftJob) * jobs.size(), sb = sizeof(FftSeg) * segs.size();
  std::vector<unsigned char> table(jb + sb);
  std::memcpy(table.data(), jobs.data(), jb);
  std::memcpy(table.data() + jb, segs.data(), sb);
  void* dj = nullptr;
  PICARD_CUDA(cudaMallocAsync(&dj, table.size(), bst));
  PICARD_CUDA(cudaMemcpyAsync(dj, table.data(), table.size(), cudaMemcpyHostToDevice, bst));
  const FftJob* dev = static_cast<const FftJob*>(dj);
  PICARD_TRY(table_stages(dev, reinterpret_cast<const FftSeg*>(static_cast<unsigned char*>(dj) + jb), range, bst));
  PICARD_CUDA(cudaFreeAsync(dj, bst));
  PICARD_CUDA(cudaEventRecord(bev, bst));
  for (int r : fft_runs) PICARD_CUDA(cudaStreamWaitEvent(ctxs[r]->st, bev, 0));
  return PICARD_OK;
}

}  // namespace picard
