// particles_exact.cu -- FP64 particle kernels with the reference's arithmetic.
//
// Compiled with --fmad=false: every multiply and add is rounded separately,
// in the order the reference writes its expressions, so positions, cell
// indices and the removed / wrapped particle sets equal the FP64 oracle's.
// This unit also holds the stochastic generators (init, inflow, produce),
// which both particle layouts share: particles are generated in FP64 and
// converted to the CELL32 layout only when stored.
#include <cuda_runtime.h>

#include <climits>
#include <cmath>

#include "chain.cuh"
#include "common.cuh"
#include "kernels.cuh"
#include "outflow.cuh"

namespace picard {

namespace {

constexpr int kThreads = 256;

inline int grid_for(long long n, int threads = kThreads) {
  long long b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > 2147483647LL) b = 2147483647LL;
  return int(b);
}

// ------------------------------------------------------------ generation

// Tools.f90:30-48 normal(): r1 for the angle, r2 = 1 - u in (0, 1].
__device__ double normal_from(Site& s, uint32_t n) {
  double r1 = s.u(n);
  double r2 = 1.0 - s.u(n + 1);
  return sqrt(-2.0 * log(r2)) * sin(kTau * r1);
}

// Tools.f90:2-28 Gaussian()
__device__ void gaussian_from(Site& s, uint32_t n, double u[3], const double v[3], double t, double m) {
  if (t > 0.0 && m > 0.0) {
    double a = m / (2.0 * kKb * t);
    double pw = sqrt(1.0 / a);
    for (int c = 0; c < 3; ++c) u[c] = normal_from(s, n + 2 * c);
    double r2 = sqrt(2.0);
    for (int c = 0; c < 3; ++c) u[c] = u[c] * pw / r2;
    for (int c = 0; c < 3; ++c) u[c] = u[c] + v[c];
  } else {
    for (int c = 0; c < 3; ++c) u[c] = v[c];
  }
}

// -dt/2 rotation with |v - ve| restored (ParticlesInitialize.f90:73-80).
__device__ void half_rotate(double v[3], const double ve[3], const double tB[3]) {
  double vmin[3], vmid[3];
  for (int c = 0; c < 3; ++c) vmin[c] = v[c] - ve[c];
  vmid[0] = vmin[0] + vmin[1] * tB[2] - vmin[2] * tB[1];
  vmid[1] = vmin[1] + vmin[2] * tB[0] - vmin[0] * tB[2];
  vmid[2] = vmin[2] + vmin[0] * tB[1] - vmin[1] * tB[0];
  double smid = vmid[0] * vmid[0] + vmid[1] * vmid[1] + vmid[2] * vmid[2];
  if (smid > 0.0) {
    double smin = vmin[0] * vmin[0] + vmin[1] * vmin[1] + vmin[2] * vmin[2];
    double f = sqrt(smin / smid);
    for (int c = 0; c < 3; ++c) vmid[c] = vmid[c] * f;
  }
  for (int c = 0; c < 3; ++c) v[c] = vmid[c] + ve[c];
}

// Member `m` of the group (ss, pp) at cell `a`: m = 0 is the ion,
// 1..epp its electrons, epp+1.. its protons.  ParticlesInitialize.f90:65-113,
// BCinflow.f90:66-114.
// In two parts: the position, which all members of a group share, and the
// velocity of member m.
__device__ __forceinline__ void gen_position(const KParams& P, Site& ion, double x0, double y0, double z0, double x[3]) {
  x[0] = x0 + P.dx * ion.u(0);
  x[1] = y0 + P.dy * ion.u(1);
  x[2] = z0 + P.dz * ion.u(2);
}
__device__ inline int member_species(const KParams& P, int ss, int m) {
  return m == 0 ? ss - 1 : (m <= P.epp[ss - 1] ? 0 : 1);  // the ion; 0 = electron, 1 = proton
}
__device__ void gen_velocity(const KParams& P, uint32_t tag, uint32_t it, uint32_t a, int ss, int pp, int m,
                             const Site& ion, double v[3], int& sp) {
  int s0 = ss - 1;
  // The ion draws its velocity from its own site after the position (from
  // u(3)); an electron or proton from a site of its own (from u(0)).  One
  // code path for both, so that a warp holding ions and their members runs
  // the Gaussian draws and the rotation once, not once per kind.
  const bool is_ion = m == 0;
  const int t = member_species(P, ss, m);
  Site src = is_ion ? ion : Site(P.seed, a, (uint32_t(ss) << 24) | (uint32_t(pp) << 8) | uint32_t(m), it, tag);
  gaussian_from(src, is_ion ? 3u : 0u, v, P.v0[s0], P.kelvin[t], P.mass[t]);
  half_rotate(v, P.ve, P.tB[t]);
  sp = t;
}
__device__ void gen_member(const KParams& P, uint32_t tag, uint32_t it, uint32_t a, int ss, int pp, int m, double x0,
                           double y0, double z0, double x[3], double v[3], int& sp) {
  Site ion(P.seed, a, (uint32_t(ss) << 24) | (uint32_t(pp) << 8), it, tag);
  gen_position(P, ion, x0, y0, z0, x);
  gen_velocity(P, tag, it, a, ss, pp, m, ion, v, sp);
}

// Slot of (ss, pp, member) inside one cell's block of created particles.
__device__ inline void decode_group(const KParams& P, const int* prefix, int local, int& ss, int& pp, int& m) {
  int s0 = 0;
  while (s0 < P.species - 1 && local >= prefix[s0 + 1]) ++s0;
  int g = 1 + P.epp[s0] + P.hpp[s0];
  int r = local - prefix[s0];
  ss = s0 + 1;
  pp = r / g + 1;
  m = r % g;
}

// Stores one FP64 particle in either layout.
__device__ inline void store_f64(PartF64 o, long long slot, const double x[3], const double v[3], int sp) {
  o.x[slot] = x[0];
  o.y[slot] = x[1];
  o.z[slot] = x[2];
  o.vx[slot] = v[0];
  o.vy[slot] = v[1];
  o.vz[slot] = v[2];
  o.sp[slot] = int8_t(sp);
}

// Base node (floor) and in-cell fraction of one coordinate, for CELL32.
// Position x on an axis -> CIC base node i and the 32-bit fixed-point offset
// f = round((t - floor t) 2^32) of t = (x - lmin)/d + 1/2 (a carry moves to
// the next node).  Far-out positions are pinned one node beyond the guard
// layer, where BCoutflow removes them.
__device__ inline void to_cell(double x, double lmin, double d, int nmax, int& i, uint32_t& f) {
  double t = (x - lmin) / d + 0.5;
  if (!(t > -2.0)) t = -2.0;  // NaN too
  if (t > nmax + 3.0) t = nmax + 3.0;
  double fl = floor(t);
  i = int(fl);
  unsigned long long q = (unsigned long long)__double2ull_rn((t - fl) * 4294967296.0);
  if (q >> 32) {
    q = 0;
    i += 1;
  }
  f = uint32_t(q);
  if (i < -1) {
    i = -1;
    f = 0u;
  }
  if (i > nmax + 1) {
    i = nmax + 1;
    f = 0xFFFFFFFFu;
  }
}

__device__ inline void store_c32(const KParams& P, PartC32 o, long long slot, const double x[3], const double v[3],
                                 int sp) {
  int i, j, k;
  uint32_t fx, fy, fz;
  to_cell(x[0], P.Lx_min, P.dx, P.nx, i, fx);
  to_cell(x[1], P.Ly_min, P.dy, P.ny, j, fy);
  to_cell(x[2], P.Lz_min, P.dz, P.nz, k, fz);
  o.cell[slot] = pack_cell(i, j, k);
  o.fx[slot] = fx;
  o.fy[slot] = fy;
  o.fz[slot] = fz;
  o.vx[slot] = float(v[0]);
  o.vy[slot] = float(v[1]);
  o.vz[slot] = float(v[2]);
  o.sp[slot] = int8_t(sp);
}

struct GroupPrefix {
  int p[9];
};

__host__ inline GroupPrefix group_prefix(const KParams& P) {
  GroupPrefix g;
  g.p[0] = 0;
  for (int s = 0; s < 8; ++s) g.p[s + 1] = g.p[s] + (s < P.species ? P.ipp[s] * (1 + P.epp[s] + P.hpp[s]) : 0);
  return g;
}

// ParticlesInitialize.f90:54-119: one thread per created particle, slot =
// start + (interior cell in k, j, i order) * per_cell + slot inside the cell.
template <class Store>
__global__ void init_kernel(KParams P, GroupPrefix G, long long start, long long total, Store store) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  int per_cell = G.p[P.species];
  long long c = t / per_cell;
  int local = int(t - c * per_cell);
  int ii = int(c % P.nx) + 2;
  int jj = int((c / P.nx) % P.ny) + 2;
  int kk = int(c / ((long long)P.nx * P.ny)) + 2;
  double x0 = P.Lx_min + P.dx * (ii - 2);
  double y0 = P.Ly_min + P.dy * (jj - 2);
  double z0 = P.Lz_min + P.dz * (kk - 2);
  uint32_t a = uint32_t(node_index(P, ii - 1, jj - 1, kk - 1));
  int ss, pp, m, sp;
  decode_group(P, G.p, local, ss, pp, m);
  double x[3], v[3];
  gen_member(P, kTagInit, 0u, a, ss, pp, m, x0, y0, z0, x, v, sp);
  store(start + t, x, v, sp);
}

struct StoreF64 {
  PartF64 o;
  __device__ void operator()(long long slot, const double x[3], const double v[3], int sp) const {
    store_f64(o, slot, x, v, sp);
  }
};
struct StoreC32 {
  KParams P;
  PartC32 o;
  __device__ void operator()(long long slot, const double x[3], const double v[3], int sp) const {
    store_c32(P, o, slot, x, v, sp);
  }
};

// Guard cell number g of the enumeration -> 1-based (ii, jj, kk) and the
// lower-edge coordinates of the cell (BCinflow.f90:56-61, 127-132, ...).
// Candidate indices of one BCinflow call are decoded in 32-bit arithmetic.
constexpr long long kMaxInflowCandidates = 0xFFFFFFFFLL;

// Guard cell g of the inflow enumeration, and the axis of its face; the launchers
// keep every candidate index (and so g) below 2^32, so the decode divides in 32 bits.
__device__ inline int inflow_cell(const KParams& P, const InflowTable& T, uint32_t g, int& ii, int& jj, int& kk,
                                  double& x0, double& y0, double& z0) {
  int f = 0;
  while (f < T.nfaces - 1 && (long long)g >= T.f[f + 1].first) ++f;
  const InflowFace& F = T.f[f];
  const uint32_t l = g - uint32_t(F.first), inner = uint32_t(F.i_n);
  const uint32_t lo = l / inner;
  int o = F.o_lo + int(lo);
  int in = F.i_lo + int(l - lo * inner);
  if (F.axis == 0) {  // outer kk, inner jj
    ii = F.fixed;
    kk = o;
    jj = in;
    x0 = F.edge;
    y0 = P.Ly_min + P.dy * (jj - 2);
    z0 = P.Lz_min + P.dz * (kk - 2);
  } else if (F.axis == 1) {  // outer kk, inner ii
    jj = F.fixed;
    kk = o;
    ii = in;
    x0 = P.Lx_min + P.dx * (ii - 2);
    y0 = F.edge;
    z0 = P.Lz_min + P.dz * (kk - 2);
  } else {  // outer jj, inner ii
    kk = F.fixed;
    jj = o;
    ii = in;
    x0 = P.Lx_min + P.dx * (ii - 2);
    y0 = P.Ly_min + P.dy * (jj - 2);
    z0 = F.edge;
  }
  return F.axis;
}

// BCinflow.f90:23-476 (append every candidate, reference order).
template <class Store>
__global__ void inflow_kernel(KParams P, InflowTable T, int iteration, long long start, long long total, Store store) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const uint32_t tu = uint32_t(t), pc = uint32_t(T.per_cell), g = tu / pc;
  const int local = int(tu - g * pc);
  int ii, jj, kk;
  double x0, y0, z0;
  inflow_cell(P, T, g, ii, jj, kk, x0, y0, z0);
  uint32_t a = uint32_t(node_index(P, ii - 1, jj - 1, kk - 1));
  int ss, pp, m, sp;
  decode_group(P, T.group_prefix, local, ss, pp, m);
  double x[3], v[3];
  gen_member(P, kTagInflow, uint32_t(iteration), a, ss, pp, m, x0, y0, z0, x, v, sp);
  store(start + t, x, v, sp);
}

// BCoutflow.f90:28-66 predicate (true = keep).
__device__ inline bool outflow_keep(const KParams& P, double x, double y, double z) {
  bool del = false;
  if (P.xflow && (x < P.xmin || x > P.xmax)) del = true;
  if (P.yflow && (y < P.ymin || y > P.ymax)) del = true;
  if (P.zflow && (z < P.zmin || z > P.zmax)) del = true;
  if (x < 2.0 * P.Lx_min - P.Lx_max || x > 2.0 * P.Lx_max - P.Lx_min) del = true;
  if (y < 2.0 * P.Ly_min - P.Ly_max || y > 2.0 * P.Ly_max - P.Ly_min) del = true;
  if (z < 2.0 * P.Lz_min - P.Lz_max || z > 2.0 * P.Lz_max - P.Lz_min) del = true;
  return !del;
}

// ParticlesTransfer.f90:494-519
__device__ inline void transfer_wrap(const KParams& P, double& x, double& y, double& z) {
  const double Lx = P.xmax - P.xmin, Ly = P.ymax - P.ymin, Lz = P.zmax - P.zmin;
  if (z < P.zmin) z = z + Lz;
  if (z > P.zmax) z = z - Lz;
  if (y < P.ymin) y = y + Ly;
  if (y > P.ymax) y = y - Ly;
  if (x < P.xmin) x = x + Lx;
  if (x > P.xmax) x = x - Lx;
}

// How far a created particle can move in one step along each axis, by its
// species.  A Gaussian draw is at most sqrt(-2 ln 2^-53) < 8.58 standard
// deviations (the uniform it comes from is at least 2^-53), and the half
// rotation keeps |v - ve|, so |v_c| <= |ve_c| + |v0 - ve| + sqrt(3) 8.58 sigma;
// a millionth more covers the rounding.
struct InflowReach {
  double r[8][3];
};

InflowReach inflow_reach(const KParams& P) {
  InflowReach R;
  for (int t = 0; t < 8; ++t) {
    double drift = 0.0;  // over the ion species that create members of species t
    for (int s = 0; s < P.species; ++s) {
      double d2 = 0.0;
      for (int c = 0; c < 3; ++c) d2 += (P.v0[s][c] - P.ve[c]) * (P.v0[s][c] - P.ve[c]);
      drift = std::fmax(drift, std::sqrt(d2));
    }
    const double sigma = P.kelvin[t] > 0.0 && P.mass[t] > 0.0 ? std::sqrt(kKb * P.kelvin[t] / P.mass[t]) : 0.0;
    for (int c = 0; c < 3; ++c)
      R.r[t][c] = std::fabs(P.dt) * (std::fabs(P.ve[c]) + drift + 14.9 * sigma) * (1.0 + 1e-6);
  }
  return R;
}

// Candidate t of the fast-path inflow: its group member and the draw site of
// its position.
struct InflowSite {
  int ss, pp, m, axis;
  uint32_t a;
  double x0, y0, z0;
};
__device__ __forceinline__ InflowSite inflow_site(const KParams& P, const InflowTable& T, uint32_t t) {
  const uint32_t pc = uint32_t(T.per_cell), g = t / pc;
  InflowSite S;
  int ii, jj, kk;
  S.axis = inflow_cell(P, T, g, ii, jj, kk, S.x0, S.y0, S.z0);
  S.a = uint32_t(node_index(P, ii - 1, jj - 1, kk - 1));
  decode_group(P, T.group_prefix, int(t - g * pc), S.ss, S.pp, S.m);
  return S;
}

// Whether the candidate starts near enough to its face to cross it in one step
// with some velocity (a comparison that is never true for a NaN bound gives
// nothing up then).  One Philox block decides.
__device__ __forceinline__ bool inflow_near(const KParams& P, const InflowTable& T, const InflowReach& R,
                                            int iteration, uint32_t t) {
  const InflowSite S = inflow_site(P, T, t);
  Site ion(P.seed, S.a, (uint32_t(S.ss) << 24) | (uint32_t(S.pp) << 8), uint32_t(iteration), kTagInflow);
  const int ax = S.axis;
  const double q = (ax == 0 ? S.x0 : ax == 1 ? S.y0 : S.z0) + (ax == 0 ? P.dx : ax == 1 ? P.dy : P.dz) * ion.u(uint32_t(ax));
  const double lo = ax == 0 ? P.xmin : ax == 1 ? P.ymin : P.zmin, hi = ax == 0 ? P.xmax : ax == 1 ? P.ymax : P.zmax;
  const double r = R.r[member_species(P, S.ss, S.m)][ax];
  return !(q < lo - r || q > hi + r);
}

// BCinflow + AdvancePosition + BCoutflow + ParticlesTransfer of candidate t:
// generated, advanced by dt, tested and wrapped; true = it survives.
__device__ inline bool inflow_candidate(const KParams& P, const InflowTable& T, int iteration, uint32_t t, double x[3],
                                        double v[3], int& sp) {
  const InflowSite S = inflow_site(P, T, t);
  gen_member(P, kTagInflow, uint32_t(iteration), S.a, S.ss, S.pp, S.m, S.x0, S.y0, S.z0, x, v, sp);
  x[0] = x[0] + v[0] * P.dt;
  x[1] = x[1] + v[1] * P.dt;
  x[2] = x[2] + v[2] * P.dt;
  if (!outflow_keep(P, x[0], x[1], x[2])) return false;
  transfer_wrap(P, x[0], x[1], x[2]);
  return true;
}

// ------------------------------------------------------------- produce

// ParticlesProduce.f90:46-58: distance of the cell centre from the source,
// averaged over 8 sub-points when the cell is close to it.
__device__ void haser_radius(const KParams& P, double x0, double y0, double z0, double& r1, double& r2) {
  double xc = x0 + 0.5 * P.dx, yc = y0 + 0.5 * P.dy, zc = z0 + 0.5 * P.dz;
  r2 = xc * xc + yc * yc + zc * zc;
  r1 = sqrt(r2);
  double q = 4.0 * r1;
  if (q * q * q < P.dV) {
    const double fa[8][3] = {{0.25, 0.25, 0.25}, {0.25, 0.25, 0.75}, {0.25, 0.75, 0.25}, {0.75, 0.25, 0.25},
                             {0.25, 0.75, 0.75}, {0.75, 0.25, 0.75}, {0.75, 0.75, 0.25}, {0.75, 0.75, 0.75}};
    double s = 0.0;
    for (int t = 0; t < 8; ++t) {
      double a = x0 + fa[t][0] * P.dx, b = y0 + fa[t][1] * P.dy, c = z0 + fa[t][2] * P.dz;
      s = s + sqrt(a * a + b * b + c * c);
    }
    r1 = s * 0.125;
    r2 = r1 * r1;
  }
}

// ParticlesProduce.f90:62-73: number of ions of species ss created in cell a.
__device__ int produce_number(const KParams& P, int iteration, uint32_t a, int ss, double r1, double r2) {
  int s0 = ss - 1;
  double nden = 0.0;
  if (P.vn[s0] > 0.0) nden = P.Qn[s0] / (2.0 * kTau * r2 * P.vn[s0]) * exp(-P.nu_d[s0] * r1 / P.vn[s0]);
  if (!(P.n2p[s0] > 0.0)) return 0;
  double rate = P.nu_i[s0] * nden * P.dV / P.n2p[s0];
  if (P.produce_dt_scaled) rate = rate * P.dt;
  if (rate == 0.0) return 0;  // int(u) with u < 1
  Site r(P.seed, a, uint32_t(ss), uint32_t(iteration), kTagProduceCount);
  return int(rate + r.u(0));
}

__device__ inline void interior_cell(const KParams& P, long long c, int& ii, int& jj, int& kk, double& x0,
                                     double& y0, double& z0) {
  ii = int(c % P.nx) + 2;
  jj = int((c / P.nx) % P.ny) + 2;
  kk = int(c / ((long long)P.nx * P.ny)) + 2;
  x0 = P.Lx_min + P.dx * (ii - 2);
  y0 = P.Ly_min + P.dy * (jj - 2);
  z0 = P.Lz_min + P.dz * (kk - 2);
}

__global__ void produce_count_kernel(KParams P, int iteration, int* counts) {
  chain_begin();
  long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long cells = (long long)P.nx * P.ny * P.nz;
  if (c >= cells) return;
  int ii, jj, kk;
  double x0, y0, z0, r1, r2;
  interior_cell(P, c, ii, jj, kk, x0, y0, z0);
  haser_radius(P, x0, y0, z0, r1, r2);
  uint32_t a = uint32_t(node_index(P, ii - 1, jj - 1, kk - 1));
  int total = 0;
  for (int ss = 1; ss <= P.species; ++ss) {
    int k = produce_number(P, iteration, a, ss, r1, r2);
    if (k > 0) total += k * (1 + P.epp[ss - 1] + P.hpp[ss - 1]);
  }
  counts[c] = total;
}

// ParticlesProduce.f90:75-103 for every ion of one cell, in (ss, pp) order.
template <class Store>
__global__ void produce_emit_kernel(KParams P, int iteration, const int* offsets, const int* count, long long capacity,
                                    int* err, Store store) {
  chain_begin();
  long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long cells = (long long)P.nx * P.ny * P.nz;
  if (c >= cells) return;
  const long long start = *count;
  int next = (c + 1 < cells) ? offsets[c + 1] : -1;
  int mine = offsets[c];
  if (next == mine) return;
  int ii, jj, kk;
  double x0, y0, z0, r1, r2;
  interior_cell(P, c, ii, jj, kk, x0, y0, z0);
  haser_radius(P, x0, y0, z0, r1, r2);
  uint32_t a = uint32_t(node_index(P, ii - 1, jj - 1, kk - 1));
  long long slot = start + mine;
  if (slot + ((next >= 0 ? next : offsets[cells]) - mine) > capacity) {
    atomicCAS(err, 0, int(kDevCapacity));
    return;
  }
  for (int ss = 1; ss <= P.species; ++ss) {
    int s0 = ss - 1;
    int k = produce_number(P, iteration, a, ss, r1, r2);
    for (int pp = 1; pp <= k; ++pp) {
      Site r(P.seed, a, (uint32_t(ss) << 24) | uint32_t(pp), uint32_t(iteration), kTagProduceParticle);
      double rnd[7];
      for (int q = 0; q < 7; ++q) rnd[q] = r.u(uint32_t(q));
      double xi[3], vi[3];
      xi[0] = x0 + P.dx * rnd[0];
      xi[1] = y0 + P.dy * rnd[1];
      xi[2] = z0 + P.dz * rnd[2];
      double rn = sqrt(xi[0] * xi[0] + xi[1] * xi[1] + xi[2] * xi[2]);
      double un = sqrt(rnd[3] * rnd[3] + rnd[4] * rnd[4] + rnd[5] * rnd[5]);
      for (int q = 0; q < 3; ++q) vi[q] = P.vn[s0] * xi[q] / rn + P.ui[s0] * rnd[3 + q] / un;
      for (int q = 0; q < 3; ++q) xi[q] = xi[q] + vi[q] * P.dt * rnd[6];
      store(slot++, xi, vi, s0);
      for (int ee = 1; ee <= P.epp[s0] + P.hpp[s0]; ++ee) {
        bool el = ee <= P.epp[s0];
        double u = el ? P.ue[s0] : P.uh[s0];
        double xe[3], vv[3];
        for (int q = 0; q < 3; ++q) vv[q] = vi[q] - (u + P.ui[s0]) * rnd[3 + q] / un;
        for (int q = 0; q < 3; ++q) xe[q] = xi[q] - vi[q] * P.dt * rnd[6] + vv[q] * P.dt * rnd[6];
        store(slot++, xe, vv, el ? 0 : 1);
      }
    }
  }
}

// ------------------------------------------------------ FP64 layout kernels

__global__ void advance_position_f64_kernel(PartF64 a, long long n, double dt) {
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    a.x[p] = a.x[p] + a.vx[p] * dt;
    a.y[p] = a.y[p] + a.vy[p] * dt;
    a.z[p] = a.z[p] + a.vz[p] * dt;
  }
}

__global__ void transfer_f64_kernel(KParams P, PartF64 a, long long n) {
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    double x = a.x[p], y = a.y[p], z = a.z[p];
    transfer_wrap(P, x, y, z);
    a.x[p] = x;
    a.y[p] = y;
    a.z[p] = z;
  }
}

// Exclusive scan of one int per thread over the block; total = the block's sum.
__device__ inline int block_exclusive_scan(int v, int* smem_warp, int& total) {
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) smem_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = (lane < (blockDim.x >> 5)) ? smem_warp[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    smem_warp[lane] = w;
  }
  __syncthreads();
  int warp_prefix = warp > 0 ? smem_warp[warp - 1] : 0;
  total = smem_warp[(blockDim.x >> 5) - 1];
  __syncthreads();
  return warp_prefix + x - v;
}

// BCoutflow.f90:28-66 and ParticlesTransfer.f90:494-519 on the FP64 layout,
// for the in-place removal of outflow.cuh.
struct OutflowF64 {
  KParams P;
  PartF64 a;
  using Key = double3;
  static constexpr bool kQuads = false;
  __device__ Key load_key(long long p) const { return make_double3(a.x[p], a.y[p], a.z[p]); }
  __device__ bool keep_wrap(long long p, double3 key, int wrap) const {
    const double x = key.x, y = key.y, z = key.z;
    if (!outflow_keep(P, x, y, z)) return false;
    if (wrap) {
      double wx = x, wy = y, wz = z;
      transfer_wrap(P, wx, wy, wz);
      if (wx != x || wy != y || wz != z) {
        a.x[p] = wx;
        a.y[p] = wy;
        a.z[p] = wz;
      }
    }
    return true;
  }
  __device__ void move(long long d, long long s) const {
    a.x[d] = a.x[s];
    a.y[d] = a.y[s];
    a.z[d] = a.z[s];
    a.vx[d] = a.vx[s];
    a.vy[d] = a.vy[s];
    a.vz[d] = a.vz[s];
    a.sp[d] = a.sp[s];
  }
};

// The fused inflow in one generation: every block takes up to 2,048 candidates, lists
// in order those that start near enough to the domain to reach it in one step
// (inflow_near: most do not, whatever velocity they would draw), generates the
// listed ones in full, and writes the survivors, in candidate order, to its own
// stretch of a staging area (FP64 position and velocity, species); after the
// scan of the block counts, the place pass stores them at *count + the block's
// offset + their rank.
//
// What bounds it: instruction issue (55 % of the slots, FP64 6 %), most of it the
// integer decode of the candidates.  Listing first matters
// as much as the early test itself: with a test ahead of the draws but 256
// candidates a block, nearly every block still waited for one lane's logarithm
// and sine.  256 x 128 x 128, 10.7 M candidates: 164 us, 267 with the test
// alone, 612 when every candidate drew its velocity.
// A block takes `items` candidates per thread, one for every four blocks an SM that
// the candidates would fill: 1 on small grids, so that the device fills, up to 8.
// us with 1 / 2 / 4 / 8 candidates a thread: 16^3 (16 k candidates) 8.1 / 9.2 / 10.9 /
// 14.2, 32^3 (222 k) 16.5 / 13.8 / 14.5 / 18.4, 48^3 (390 k) 21.8 / 20.7 / 17.0 / 19.8,
// 77^3 (970 k) 43 / 34 / 29 / 27, 256 x 128 x 128 (5.4 M) 198 / 145 / 109 / 90.
constexpr int kInflowItems = 8;
inline int inflow_items(long long candidates) {
  const long long q = candidates / (148LL * 4 * kThreads);
  return q < 1 ? 1 : q > kInflowItems ? kInflowItems : int(q);
}
__global__ void __launch_bounds__(kThreads) inflow_stage_kernel(KParams P, InflowTable T, InflowReach R, int iteration,
                                                                long long total, int items, int* block_counts,
                                                                double* stage, int8_t* stage_sp, long long stride) {
  chain_begin();
  constexpr int kWords = kInflowItems * kThreads / 32;
  static_assert(kWords == 64, "two words per lane of the scanning warp");
  __shared__ int warp_sums[32];
  __shared__ uint16_t list[kInflowItems * kThreads];
  __shared__ unsigned near[kWords];   // bit l of word w: candidate 32 w + l starts near enough
  __shared__ int before[kWords + 1];  // listed candidates before each word's
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long base = (long long)blockIdx.x * items * kThreads;
  for (int q = 0; q < kInflowItems; ++q) {
    unsigned m = 0;
    if (q < items) {
      const long long t = base + q * kThreads + threadIdx.x;
      m = __ballot_sync(0xffffffffu, t < total && inflow_near(P, T, R, iteration, uint32_t(t)));
    }
    if (lane == 0) near[q * (kThreads / 32) + warp] = m;
  }
  __syncthreads();
  if (warp == 0) {
    const int c0 = __popc(near[2 * lane]), v = c0 + __popc(near[2 * lane + 1]);
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    before[2 * lane] = x - v;
    before[2 * lane + 1] = x - v + c0;
    if (lane == 31) before[kWords] = x;
  }
  __syncthreads();
  for (int q = 0; q < items; ++q) {
    const int w = q * (kThreads / 32) + warp;
    if (near[w] >> lane & 1u) list[before[w] + __popc(near[w] & ((1u << lane) - 1u))] = uint16_t(32 * w + lane);
  }
  const int listed = before[kWords];
  __syncthreads();
  int done = 0;
  for (int first = 0; first < listed; first += kThreads) {
    const int e = first + threadIdx.x;
    double x[3], v[3];
    int sp = 0;
    const bool keep = e < listed && inflow_candidate(P, T, iteration, uint32_t(base) + list[e], x, v, sp);
    int sum;
    const int rank = block_exclusive_scan(keep ? 1 : 0, warp_sums, sum);
    if (keep) {
      const long long q = base + done + rank;
      stage[q] = x[0];
      stage[q + stride] = x[1];
      stage[q + 2 * stride] = x[2];
      stage[q + 3 * stride] = v[0];
      stage[q + 4 * stride] = v[1];
      stage[q + 5 * stride] = v[2];
      stage_sp[q] = int8_t(sp);
    }
    done += sum;
  }
  if (threadIdx.x == 0) block_counts[blockIdx.x] = done;
}

template <class Store>
__global__ void __launch_bounds__(kThreads) inflow_place_kernel(int tile, const int* block_counts, const int* offsets,
                                                                const int* count, long long capacity, int* err,
                                                                const double* stage, const int8_t* stage_sp,
                                                                long long stride, Store store) {
  chain_begin();
  for (int r = threadIdx.x; r < block_counts[blockIdx.x]; r += blockDim.x) {
    const long long q = (long long)blockIdx.x * tile + r;
    const double x[3] = {stage[q], stage[q + stride], stage[q + 2 * stride]};
    const double v[3] = {stage[q + 3 * stride], stage[q + 4 * stride], stage[q + 5 * stride]};
    const long long slot = (long long)*count + offsets[blockIdx.x] + r;
    if (slot < capacity)
      store(slot, x, v, int(stage_sp[q]));
    else
      atomicCAS(err, 0, int(kDevCapacity));
  }
}

// CIC weights of ParticlesGridify.f90:70-88 (F1..F8 before the 1/dV).
struct Cic64 {
  int i, j, k;  // 0-based base node
  double F[8];
};

// One axis: base node int((x - lo)/d + 1/2) and fmod(x - lo + d/2, d), both
// exactly as the reference's arithmetic gives them.  The quotient by the
// reciprocal decides unless it lies within 1e-6 of an integer (its error is a
// few ulp of at most 2^31), where the division does; the remainder is one FMA
// (exact when it lies in [0, d)), else fmod's.  Three library fmod calls and
// divisions a particle were most of the deposit's and the push's instructions.
__device__ __forceinline__ void cic_axis(double x, double lo, double d, double inv, int& i, double& rest) {
  const double a = x - lo, t2 = a * inv + 0.5;
  i = int(t2);
  if (!(fabs(t2 - rint(t2)) >= 1e-6)) i = int(a / d + 0.5);
  const double t = a + 0.5 * d;
  rest = fma(-double(i), d, t);
  if (!(rest >= 0.0 && rest < d)) rest = fmod(t, d);
}

// Base node and the distances `r` from it on each axis.
struct Cic64Axes {
  int i, j, k;
  double r[3];
};
__device__ __forceinline__ void cic_axes(const KParams& P, double x, double y, double z, Cic64Axes& c) {
  cic_axis(x, P.Lx_min, P.dx, 1.0 / P.dx, c.i, c.r[0]);
  cic_axis(y, P.Ly_min, P.dy, 1.0 / P.dy, c.j, c.r[1]);
  cic_axis(z, P.Lz_min, P.dz, 1.0 / P.dz, c.k, c.r[2]);
}

__device__ inline void cic64(const KParams& P, double x, double y, double z, Cic64& w) {
  Cic64Axes c;
  cic_axes(P, x, y, z, c);
  const double rest0 = c.r[0], rest1 = c.r[1], rest2 = c.r[2];
  const double d0 = P.dx - rest0, d1 = P.dy - rest1, d2 = P.dz - rest2;
  w.i = c.i;
  w.j = c.j;
  w.k = c.k;
  w.F[0] = d0 * d1 * d2;
  w.F[1] = rest0 * d1 * d2;
  w.F[2] = d0 * rest1 * d2;
  w.F[3] = d0 * d1 * rest2;
  w.F[4] = rest0 * rest1 * d2;
  w.F[5] = d0 * rest1 * rest2;
  w.F[6] = rest0 * d1 * rest2;
  w.F[7] = rest0 * rest1 * rest2;
}

__constant__ int kOff[8][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {1, 1, 0}, {0, 1, 1}, {1, 0, 1}, {1, 1, 1}};

__device__ inline int clamp_gather(int i, int n) { return i < 0 ? 0 : (i > n + 1 ? n + 1 : i); }

// AdvanceVelocity.f90:39-121 (mode 0), AdvanceVelocityExp (mode 1),
// AdvanceVelocityImp (mode 2).  E is three planes (Ex, Ey, Ez) of nodes.
__global__ void advance_velocity_f64_kernel(KParams P, PartF64 a, long long n, const double* __restrict__ E,
                                            double dt, double deltat, int mode) {
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    Cic64 w;
    cic64(P, a.x[p], a.y[p], a.z[p], w);
    double Ep[3];
    for (int c = 0; c < 3; ++c) {
      const double* Ec = E + (long long)c * P.nodes;
      double s = 0.0;
      for (int q = 0; q < 8; ++q) {
        int i = clamp_gather(w.i + kOff[q][0], P.nx), j = clamp_gather(w.j + kOff[q][1], P.ny),
            k = clamp_gather(w.k + kOff[q][2], P.nz);
        double e = Ec[node_index(P, i, j, k)];
        s = (q == 0) ? e * w.F[0] : s + e * w.F[q];
      }
      Ep[c] = s / P.dV;
    }
    int s = a.sp[p];
    double v[3] = {a.vx[p], a.vy[p], a.vz[p]};
    if (P.fluid[s]) {
      if (P.gyration[s]) {
        const double* B = P.B0;
        double vb = v[0] * B[0] + v[1] * B[1] + v[2] * B[2];
        double vm[3], vd[3];
        for (int c = 0; c < 3; ++c) vm[c] = vb * B[c];
        vd[0] = vm[0] + (Ep[1] * B[2] - Ep[2] * B[1]);
        vd[1] = vm[1] + (Ep[2] * B[0] - Ep[0] * B[2]);
        vd[2] = vm[2] + (Ep[0] * B[1] - Ep[1] * B[0]);
        double ib = 1.0 / (B[0] * B[0] + B[1] * B[1] + B[2] * B[2]);
        a.vx[p] = vd[0] * ib;
        a.vy[p] = vd[1] * ib;
        a.vz[p] = vd[2] * ib;
      }
      continue;
    }
    double etadt2, tB[3];
    if (mode == 0) {
      etadt2 = 0.5 * dt * P.eta[s];
      for (int c = 0; c < 3; ++c) tB[c] = P.tB[s][c];
    } else {
      etadt2 = 0.5 * dt * P.eta[s] * 2.0 * deltat / dt;
      for (int c = 0; c < 3; ++c) tB[c] = P.tB[s][c] * 2.0 * deltat / dt;
    }
    double vmin[3], vmid[3];
    if (mode == 0) {
      const double* sB = P.sB[s];
      double vplus[3];
      for (int c = 0; c < 3; ++c) vmin[c] = v[c] - P.ve[c] + etadt2 * Ep[c];
      vmid[0] = vmin[0] + vmin[1] * tB[2] - vmin[2] * tB[1];
      vmid[1] = vmin[1] + vmin[2] * tB[0] - vmin[0] * tB[2];
      vmid[2] = vmin[2] + vmin[0] * tB[1] - vmin[1] * tB[0];
      vplus[0] = vmin[0] + vmid[1] * sB[2] - vmid[2] * sB[1];
      vplus[1] = vmin[1] + vmid[2] * sB[0] - vmid[0] * sB[2];
      vplus[2] = vmin[2] + vmid[0] * sB[1] - vmid[1] * sB[0];
      for (int c = 0; c < 3; ++c) v[c] = vplus[c] + P.ve[c] + etadt2 * Ep[c];
    } else {
      if (mode == 1)
        for (int c = 0; c < 3; ++c) vmin[c] = v[c] - P.ve[c];
      else
        for (int c = 0; c < 3; ++c) vmin[c] = v[c] - P.ve[c] + etadt2 * Ep[c];
      vmid[0] = vmin[0] + vmin[1] * tB[2] - vmin[2] * tB[1];
      vmid[1] = vmin[1] + vmin[2] * tB[0] - vmin[0] * tB[2];
      vmid[2] = vmin[2] + vmin[0] * tB[1] - vmin[1] * tB[0];
      double smid = vmid[0] * vmid[0] + vmid[1] * vmid[1] + vmid[2] * vmid[2];
      if (smid > 0.0) {
        double smin = vmin[0] * vmin[0] + vmin[1] * vmin[1] + vmin[2] * vmin[2];
        double f = sqrt(smin / smid);
        for (int c = 0; c < 3; ++c) vmid[c] = vmid[c] * f;
      }
      if (mode == 1)
        for (int c = 0; c < 3; ++c) v[c] = vmid[c] + P.ve[c] + etadt2 * Ep[c];
      else
        for (int c = 0; c < 3; ++c) v[c] = vmid[c] + P.ve[c];
    }
    a.vx[p] = v[0];
    a.vy[p] = v[1];
    a.vz[p] = v[2];
  }
}

// Deposit index of node i on an axis of n cells: open axes fold the ghost
// layers onto the first / last interior node (ParticlesGridify.f90:149-171),
// periodic axes fold them onto the opposite interior node (ibid. 167-170).
__device__ inline int fold_index(int i, int n, int open) {
  if (open) return i < 1 ? 1 : (i > n ? n : i);
  // periodic: the interior node congruent to i modulo n -- one period for
  // the ghost layers, a closed-form remainder for anything farther out
  if (i < 1)
    i += n;
  else if (i > n)
    i -= n;
  if (i >= 1 && i <= n) return i;
  long long r = ((long long)i - 1) % n;
  return int(r < 0 ? r + n : r) + 1;
}

// True when x lies within half a cell of [L_min, L_max] (NaN: false).  There
// the CIC base node is 0 .. n and both stencil nodes lie inside the
// ghost-padded box, with non-negative weights.  The reference deposits after
// BCoutflow and ParticlesTransfer, which leave every particle inside
// [min, max], so its particles always pass.
__device__ inline bool within_half_cell(double x, double lo, double hi, double d) {
  return x >= lo - 0.5 * d && x < hi + 0.5 * d;
}

// F (a product of three distances) -> round(F/dV 2^40), scale = 2^40/dV: one
// FMA against 1.5 2^52 leaves the integer in the low mantissa bits (|result| <
// 2^51).  Every FP64 deposit takes its weights from here, so their sums agree
// bit for bit.
__device__ __forceinline__ long long fixed_bits_f64(double F, double scale) {
  return __double_as_longlong(fma(F, scale, 6755399441055744.0));
}
__device__ __forceinline__ long long fixed_f64(double F, double scale) {
  return fixed_bits_f64(F, scale) - 0x4338000000000000LL;
}

// The deposit of FP64 positions (ParticlesGridify.f90:65-123), shared-memory
// tiled as the CELL32 one (deposit_tile_c32_kernel): a warp takes 64
// consecutive particles, two to a lane in 16-byte loads, finds the box of their
// CIC stencils, adds the weights in 20-bit halves to its own tile, lane
// l visiting the corners in the order q ^ (l & 7), and flushes each touched
// node to global memory once.  A box that does not fit keeps the particles
// around the warp's middle cell and adds the others' corners directly.
//
// CALLER: positions and 1-based species of another owner (gridify_noalloc):
// species outside 1 .. species, and positions farther than half a cell outside
// the domain, are skipped.  VEC: the arrays allow 16-byte loads.
//
// What bounds it: instruction issue (70 % of the slots; FP64 arithmetic, then
// 16 shared atomics a particle).  8 M particles on 64^3: 193 us, against 1684
// for one particle per lane with warp aggregation by match_any and two
// partial-mask reductions per corner, three fmod calls and eleven divisions; 1
// M on 32^3 44 and 218, 2 M on 90^3 (under three per cell) 126 and 648, 4 M in
// no order 221 and 1424.  Two particles per lane at 64 registers beat four (80
// registers 248 us, 106 registers 261) and eight (128 registers, 521).
constexpr int kTileF64 = 768;   // entries per warp (two u32 halves)
constexpr int kTileWarps = 8;
constexpr int kTilePer = 2;     // particles per lane
constexpr int kTileCtas = 4;    // CTAs per SM (64 registers, 48 KB)

template <bool CALLER, bool VEC, class Sp>
__global__ void __launch_bounds__(256, kTileCtas) deposit_tile_f64_kernel(KParams P, const double* __restrict__ x,
                                                                  const double* __restrict__ y,
                                                                  const double* __restrict__ z,
                                                                  const Sp* __restrict__ sp, long long n,
                                                                  unsigned long long* Nacc, int reach) {
  extern __shared__ unsigned int f64_tile[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned int* lo = f64_tile + warp * 2 * kTileF64;
  constexpr int kHi = kTileF64;
  const bool sx = lane & 1, sy = lane & 2, sz = lane & 4;
  const double scale = kDepositScale / P.dV;
  int zeroed = 0;  // entries below this are zero between chunks: the flush clears what it reads
  const long long warps = (long long)gridDim.x * kTileWarps;
  for (long long base = ((long long)blockIdx.x * kTileWarps + warp) * (32 * kTilePer); base < n;
       base += warps * (32 * kTilePer)) {
    // pairs of consecutive particles: base + 2 lane
    double px[kTilePer], py[kTilePer], pz[kTilePer];
    int s[kTilePer];
    Cic64Axes c[kTilePer];
    unsigned live = 0;
    const bool full = base + 32 * kTilePer <= n;
#pragma unroll
    for (int h = 0; h < kTilePer / 2; ++h) {
      const long long p = base + 64 * h + 2 * lane;
      if (VEC && full) {
        const double2 vx = __ldcs(reinterpret_cast<const double2*>(x + p)), vy = __ldcs(reinterpret_cast<const double2*>(y + p)),
                      vz = __ldcs(reinterpret_cast<const double2*>(z + p));
        px[2 * h] = vx.x, px[2 * h + 1] = vx.y;
        py[2 * h] = vy.x, py[2 * h + 1] = vy.y;
        pz[2 * h] = vz.x, pz[2 * h + 1] = vz.y;
        s[2 * h] = int(sp[p]), s[2 * h + 1] = int(sp[p + 1]);
        live |= 3u << (2 * h);
      } else {
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const bool in = p + t < n;
          px[2 * h + t] = in ? x[p + t] : 0.0;
          py[2 * h + t] = in ? y[p + t] : 0.0;
          pz[2 * h + t] = in ? z[p + t] : 0.0;
          s[2 * h + t] = in ? int(sp[p + t]) : 0;
          if (in) live |= 1u << (2 * h + t);
        }
      }
    }
    int imin = INT_MAX, imax = INT_MIN, jmin = INT_MAX, jmax = INT_MIN, kmin = INT_MAX, kmax = INT_MIN;
    int smin = INT_MAX, smax = INT_MIN;
    unsigned near = 0;
    auto widen = [&](int m) {
      near |= 1u << m;
      imin = min(imin, c[m].i), imax = max(imax, c[m].i);
      jmin = min(jmin, c[m].j), jmax = max(jmax, c[m].j);
      kmin = min(kmin, c[m].k), kmax = max(kmax, c[m].k);
      smin = min(smin, s[m]), smax = max(smax, s[m]);
    };
#pragma unroll
    for (int m = 0; m < kTilePer; ++m) {
      if (CALLER) {
        s[m] -= 1;
        if (!(s[m] >= 0 && s[m] < P.species && within_half_cell(px[m], P.Lx_min, P.Lx_max, P.dx) &&
              within_half_cell(py[m], P.Ly_min, P.Ly_max, P.dy) && within_half_cell(pz[m], P.Lz_min, P.Lz_max, P.dz)))
          live &= ~(1u << m);
      }
      cic_axes(P, px[m], py[m], pz[m], c[m]);
      // only non-negative weights go to the tile
      const bool in = c[m].r[0] >= 0.0 && c[m].r[0] <= P.dx && c[m].r[1] >= 0.0 && c[m].r[1] <= P.dy &&
                      c[m].r[2] >= 0.0 && c[m].r[2] <= P.dz;
      if ((live >> m & 1u) && in) widen(m);
    }
    auto reduce_box = [&]() -> int {
      imin = __reduce_min_sync(0xffffffffu, imin), imax = __reduce_max_sync(0xffffffffu, imax);
      jmin = __reduce_min_sync(0xffffffffu, jmin), jmax = __reduce_max_sync(0xffffffffu, jmax);
      kmin = __reduce_min_sync(0xffffffffu, kmin), kmax = __reduce_max_sync(0xffffffffu, kmax);
      smin = __reduce_min_sync(0xffffffffu, smin), smax = __reduce_max_sync(0xffffffffu, smax);
      if (imax < imin) return 0;  // nothing near
      const long long bi = (long long)imax - imin + 2, bj = (long long)jmax - jmin + 2, bk = (long long)kmax - kmin + 2;
      if (bi > 64 || bj > 64 || bk > 64) return 0;
      const int v = int(bi * bj * bk) * (smax - smin + 1);
      return v <= kTileF64 ? v : 0;
    };
    int vol = reduce_box();
    if (vol == 0) {
      // the particles around the first near one of the middle lane that has one
      const unsigned have = __ballot_sync(0xffffffffu, near != 0u);
      if (have) {
        const unsigned upper = have & 0xffff0000u;
        const int src = upper ? __ffs(upper) - 1 : 31 - __clz(have);
        int mi = 0, mj = 0, mk = 0;
#pragma unroll
        for (int m = kTilePer - 1; m >= 0; --m)
          if (near >> m & 1u) mi = c[m].i, mj = c[m].j, mk = c[m].k;
        mi = __shfl_sync(0xffffffffu, mi, src), mj = __shfl_sync(0xffffffffu, mj, src), mk = __shfl_sync(0xffffffffu, mk, src);
        const unsigned was = near;
        near = 0;
        imin = jmin = kmin = smin = INT_MAX;
        imax = jmax = kmax = smax = INT_MIN;
#pragma unroll
        for (int m = 0; m < kTilePer; ++m)
          if ((was >> m & 1u) && abs(c[m].i - mi) <= reach && abs(c[m].j - mj) <= 2 && abs(c[m].k - mk) <= 2) widen(m);
        vol = reduce_box();
      }
      if (vol == 0) near = 0;
    }
    if (vol > 0) {
      const int bi = imax - imin + 2, bj = jmax - jmin + 2, bk = kmax - kmin + 2;
      const int sj = bi, sk = bi * bj, ss = sk * bk;
      if (vol > zeroed) {
        for (int e = zeroed + lane; e < vol; e += 32) lo[e] = 0u, lo[e + kHi] = 0u;
        zeroed = vol;
        __syncwarp();
      }
      const int first = (sx ? 1 : 0) + (sy ? sj : 0) + (sz ? sk : 0) - (imin + jmin * sj + kmin * sk + smin * ss);
      const int ex = sx ? -1 : 1, ey = sy ? -sj : sj, ez = sz ? -sk : sk;
#pragma unroll
      for (int m = 0; m < kTilePer; ++m) {
        if (!(near >> m & 1u)) continue;
        const double r0 = c[m].r[0], r1 = c[m].r[1], r2 = c[m].r[2];
        const double d0 = P.dx - r0, d1 = P.dy - r1, d2 = P.dz - r2;
        const double ax[2] = {sx ? r0 : d0, sx ? d0 : r0}, ay[2] = {sy ? r1 : d1, sy ? d1 : r1},
                     az[2] = {sz ? r2 : d2, sz ? d2 : r2};
        unsigned int* e0 = lo + (first + c[m].i + c[m].j * sj + c[m].k * sk + s[m] * ss);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const long long u = fixed_bits_f64((ax[q & 1] * ay[q >> 1 & 1]) * az[q >> 2], scale);
          unsigned int* e = e0 + ((q & 1) ? ex : 0) + ((q & 2) ? ey : 0) + ((q & 4) ? ez : 0);
          // low 20 bits; the high ones under a constant top bit that the sum masks off
          atomicAdd(e, unsigned(u) & 0xFFFFFu);
          atomicAdd(e + kHi, unsigned(u >> 20));
        }
      }
      __syncwarp();
      // v / d = (v inv) >> 16 for v < 1024, d <= 64
      const uint32_t ri = (65535u + bi) / uint32_t(bi), rj = (65535u + bj) / uint32_t(bj), rk = (65535u + bk) / uint32_t(bk);
      for (int e = lane; e < vol; e += 32) {
        const unsigned l = lo[e], h = lo[e + kHi];
        if ((l | h) == 0u) continue;
        lo[e] = 0u, lo[e + kHi] = 0u;
        const int r1 = int((uint32_t(e) * ri) >> 16), r2 = int((uint32_t(r1) * rj) >> 16),
                  r3 = int((uint32_t(r2) * rk) >> 16);
        const int i = fold_index(e - r1 * bi + imin, P.nx, P.xflow), j = fold_index(r1 - r2 * bj + jmin, P.ny, P.yflow),
                  k = fold_index(r2 - r3 * bk + kmin, P.nz, P.zflow);
        const unsigned long long v = ((unsigned long long)(h & 0x7FFFFFFFu) << 20) + (unsigned long long)l;
        atomicAdd(Nacc + (long long)(r3 + smin) * P.nodes + node_index(P, i, j, k), v);
      }
      __syncwarp();
    }
    unsigned far = live & ~near;
    if (__any_sync(0xffffffffu, far != 0u)) {
#pragma unroll
      for (int m = 0; m < kTilePer; ++m) {
        if (!(far >> m & 1u)) continue;
        unsigned long long* plane = Nacc + (long long)s[m] * P.nodes;
#pragma unroll 1
        for (int q = 0; q < 8; ++q) {
          const double F = (((q & 1) ? c[m].r[0] : P.dx - c[m].r[0]) * ((q & 2) ? c[m].r[1] : P.dy - c[m].r[1])) *
                           ((q & 4) ? c[m].r[2] : P.dz - c[m].r[2]);
          const int i = fold_index(c[m].i + (q & 1), P.nx, P.xflow), j = fold_index(c[m].j + (q >> 1 & 1), P.ny, P.yflow),
                    k = fold_index(c[m].k + (q >> 2), P.nz, P.zflow);
          atomicAdd(plane + node_index(P, i, j, k), (unsigned long long)fixed_f64(F, scale));
        }
      }
    }
  }
}

template <bool CALLER, class Sp>
cudaError_t launch_deposit_tile_f64(const KParams& P, const double* x, const double* y, const double* z, const Sp* sp,
                                    long long n, unsigned long long* acc, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const size_t smem = size_t(kTileWarps) * 2 * sizeof(unsigned int) * kTileF64;  // within the default 48 KB
  const long long chunk = (long long)kTileWarps * 32 * kTilePer, chunks = (n + chunk - 1) / chunk;
  const int grid = int(chunks < 148LL * kTileCtas ? chunks : 148LL * kTileCtas);
  // the window reaches as far along x as one warp's particles do at this density, and two cells
  const long long span = 32LL * kTilePer * P.nx * P.ny * P.nz / n + 2;
  const int reach = int(span < 15 ? span : 15);
  const uintptr_t bits = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(z);
  note_launch();
  if (bits % 16 == 0)
    deposit_tile_f64_kernel<CALLER, true, Sp><<<grid, 256, smem, st>>>(P, x, y, z, sp, n, acc, reach);
  else
    deposit_tile_f64_kernel<CALLER, false, Sp><<<grid, 256, smem, st>>>(P, x, y, z, sp, n, acc, reach);
  return cudaGetLastError();
}

// The flux of GridifyAll (ParticlesGridifyAll.f90:65-160): w v in fixed point, 24
// atomics a particle straight to global memory, which bound it; its N comes from the
// tiles above.  GridifyAll's two passes in us, against one kernel with both sums (N
// aggregated by match_any; 89 registers since the remainders are FMAs, 64 before):
// 1.05 M particles on 32^3 177 (290, 208), 8.4 M on 64^3 1165 (2075, 1370), 18 M on
// 100 x 90 x 128 2080 (5230, 3300).
__global__ void __launch_bounds__(256, 4) flux_f64_kernel(KParams P, PartF64 a, long long n, unsigned long long* Facc) {
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    Cic64 c;
    cic64(P, a.x[p], a.y[p], a.z[p], c);
    const double vel[3] = {a.vx[p], a.vy[p], a.vz[p]};
    unsigned long long* plane = Facc + (long long)a.sp[p] * 3 * P.nodes;
    for (int q = 0; q < 8; ++q) {
      const int i = fold_index(c.i + kOff[q][0], P.nx, P.xflow), j = fold_index(c.j + kOff[q][1], P.ny, P.yflow),
                k = fold_index(c.k + kOff[q][2], P.nz, P.zflow);
      const long long node = node_index(P, i, j, k);
      const double F = c.F[q] / P.dV;
      for (int d = 0; d < 3; ++d)
        atomicAdd(plane + (long long)d * P.nodes + node, (unsigned long long)__double2ll_rn(F * vel[d] * kFluxScale));
    }
  }
}

// Block partial sums of sum(n2p*mass*|v|^2) (picard.f90:661-664).
__global__ void energy_particles_f64_kernel(KParams P, PartF64 a, long long n, double* partial) {
  __shared__ double sh[32];
  double acc = 0.0;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    int s = a.sp[p];
    double v2 = a.vx[p] * a.vx[p] + a.vy[p] * a.vy[p] + a.vz[p] * a.vz[p];
    acc += P.n2p[s] * P.mass[s] * v2;
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < int(blockDim.x >> 5); ++w) t += sh[w];
    partial[blockIdx.x] = t;
  }
}

// One block of 256 threads (a single thread walking the 2,368 partials took 61
// us): strided sums, then a tree, in an order that depends on nb alone.
__global__ void finish_sum_kernel(const double* partial, int nb, double scale, double* out) {
  __shared__ double sh[256];
  double t = 0.0;
  for (int b = threadIdx.x; b < nb; b += 256) t += partial[b];
  sh[threadIdx.x] = t;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0] * scale;
}

__global__ void cell_indices_f64_kernel(KParams P, PartF64 a, long long n, int* ijk) {
  long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  ijk[3 * p + 0] = 1 + int((a.x[p] - P.Lx_min) / P.dx + 0.5);
  ijk[3 * p + 1] = 1 + int((a.y[p] - P.Ly_min) / P.dy + 0.5);
  ijk[3 * p + 2] = 1 + int((a.z[p] - P.Lz_min) / P.dz + 0.5);
}

// CalcDistance.f90:28-87 (one thread per (ii, jj, kk) of the positive octant).
__global__ void calc_distance_kernel(KParams P, double* D) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int Nx = P.nx, Ny = P.ny, Nz = P.nz;
  long long total = (long long)(Nx + 1) * (Ny + 1) * (Nz + 1);
  if (t >= total) return;
  int ii = int(t % (Nx + 1)) + 1, jj = int((t / (Nx + 1)) % (Ny + 1)) + 1, kk = int(t / ((long long)(Nx + 1) * (Ny + 1))) + 1;
  const long long DX = 2 * Nx + 1, DY = 2 * Ny + 1;
  double di = double(ii - 1), dj = double(jj - 1), dk = double(kk - 1);
  double a = di * P.dx, b = dj * P.dy, c = dk * P.dz;
  double an = (Nx - di) * P.dx, bn = (Ny - dj) * P.dy, cn = (Nz - dk) * P.dz;
  auto inv = [](double x, double y, double z) { return 1.0 / sqrt(x * x + y * y + z * z); };
  double t0 = (ii == 1 && jj == 1 && kk == 1) ? 0.0 : inv(a, b, c);
  const int xf = P.xflow != 0, yf = P.yflow != 0, zf = P.zflow != 0;
  if (xf) {
    if (!yf && !zf) {
      t0 = t0 + inv(a, bn, c);
      t0 = t0 + inv(a, b, cn);
      t0 = t0 + inv(a, bn, cn);
    } else if (!yf) {
      t0 = t0 + inv(a, bn, c);
    } else if (!zf) {
      t0 = t0 + inv(a, b, cn);
    }
  } else if (yf) {
    if (!zf) {
      t0 = t0 + inv(an, b, c);
      t0 = t0 + inv(a, b, cn);
      t0 = t0 + inv(an, b, cn);
    } else {
      t0 = t0 + inv(an, b, c);
    }
  } else if (zf) {
    t0 = t0 + inv(an, b, c);
    t0 = t0 + inv(a, bn, c);
    t0 = t0 + inv(an, bn, c);
  } else {
    t0 = t0 + inv(an, b, c);
    t0 = t0 + inv(a, bn, c);
    t0 = t0 + inv(a, b, cn);
    t0 = t0 + inv(an, bn, c);
    t0 = t0 + inv(a, bn, cn);
    t0 = t0 + inv(an, b, cn);
    t0 = t0 + inv(an, bn, cn);
  }
  int pi = Nx + 1 + (ii - 1), pj = Ny + 1 + (jj - 1), pk = Nz + 1 + (kk - 1);
  int ni = Nx + 1 - (ii - 1), nj = Ny + 1 - (jj - 1), nk = Nz + 1 - (kk - 1);
  auto at = [&](int i, int j, int k) { return (long long)(i - 1) + DX * ((long long)(j - 1) + DY * (long long)(k - 1)); };
  D[at(pi, pj, pk)] = t0;
  D[at(ni, pj, pk)] = t0;
  D[at(pi, nj, pk)] = t0;
  D[at(pi, pj, nk)] = t0;
  D[at(ni, nj, pk)] = t0;
  D[at(pi, nj, nk)] = t0;
  D[at(ni, pj, nk)] = t0;
  D[at(ni, nj, nk)] = t0;
}

// CELL32 -> FP64 positions: x = Lx_min + (i + f/2^32 - 0.5) dx.
__global__ void c32_to_f64_kernel(KParams P, PartC32 a, long long n, PartF64 o) {
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    int i, j, k;
    unpack_cell(a.cell[p], i, j, k);
    o.x[p] = P.Lx_min + ((double)i + off_f64(a.fx[p]) - 0.5) * P.dx;
    o.y[p] = P.Ly_min + ((double)j + off_f64(a.fy[p]) - 0.5) * P.dy;
    o.z[p] = P.Lz_min + ((double)k + off_f64(a.fz[p]) - 0.5) * P.dz;
    o.vx[p] = a.vx[p];
    o.vy[p] = a.vy[p];
    o.vz[p] = a.vz[p];
    o.sp[p] = a.sp[p];
  }
}

__global__ void f64_to_c32_kernel(KParams P, PartF64 a, long long n, PartC32 o) {
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    double x[3] = {a.x[p], a.y[p], a.z[p]};
    double v[3] = {a.vx[p], a.vy[p], a.vz[p]};
    store_c32(P, o, p, x, v, a.sp[p]);
  }
}

}  // namespace

int compact_blocks(long long n) { return int((n + kOutflowTile - 1) / kOutflowTile); }

int inflow_blocks(long long candidates) { return grid_for(candidates, inflow_items(candidates) * kThreads); }

cudaError_t launch_calc_distance(const KParams& P, double* D, cudaStream_t st) {
  long long total = (long long)(P.nx + 1) * (P.ny + 1) * (P.nz + 1);
  note_launch();
  calc_distance_kernel<<<grid_for(total), kThreads, 0, st>>>(P, D);
  return cudaGetLastError();
}

cudaError_t launch_init_f64(const KParams& P, PartF64 out, long long start, cudaStream_t st) {
  GroupPrefix G = group_prefix(P);
  long long total = (long long)P.nx * P.ny * P.nz * G.p[P.species];
  if (total == 0) return cudaSuccess;
  note_launch();
  init_kernel<<<grid_for(total), kThreads, 0, st>>>(P, G, start, total, StoreF64{out});
  return cudaGetLastError();
}

cudaError_t launch_init_c32(const KParams& P, PartC32 out, long long start, cudaStream_t st) {
  GroupPrefix G = group_prefix(P);
  long long total = (long long)P.nx * P.ny * P.nz * G.p[P.species];
  if (total == 0) return cudaSuccess;
  note_launch();
  init_kernel<<<grid_for(total), kThreads, 0, st>>>(P, G, start, total, StoreC32{P, out});
  return cudaGetLastError();
}

cudaError_t launch_inflow_f64(const KParams& P, const InflowTable& T, int iteration, PartF64 out, long long start,
                              cudaStream_t st) {
  long long total = T.cells * T.per_cell;
  if (total == 0) return cudaSuccess;
  if (total > kMaxInflowCandidates) return cudaErrorInvalidValue;
  note_launch();
  inflow_kernel<<<grid_for(total), kThreads, 0, st>>>(P, T, iteration, start, total, StoreF64{out});
  return cudaGetLastError();
}

cudaError_t launch_inflow_c32(const KParams& P, const InflowTable& T, int iteration, PartC32 out, long long start,
                              cudaStream_t st) {
  long long total = T.cells * T.per_cell;
  if (total == 0) return cudaSuccess;
  if (total > kMaxInflowCandidates) return cudaErrorInvalidValue;
  note_launch();
  inflow_kernel<<<grid_for(total), kThreads, 0, st>>>(P, T, iteration, start, total, StoreC32{P, out});
  return cudaGetLastError();
}

cudaError_t launch_produce_count(const KParams& P, int iteration, int* counts, cudaStream_t st) {
  long long cells = (long long)P.nx * P.ny * P.nz;
  return launch_chained(produce_count_kernel, grid_for(cells), kThreads, 0, st, P, iteration, counts);
}

__global__ void add_count_kernel(int* count, const int* add, long long capacity) {
  chain_begin();
  long long v = (long long)*count + *add;
  *count = int(v < capacity ? v : capacity);
}

template <class Store>
static cudaError_t inflow_fused(const KParams& P, const InflowTable& T, int iteration, Store store, int* count,
                                long long capacity, int* block_counts, int* block_offsets, int* err,
                                const InflowStage& S, cudaStream_t st) {
  const long long total = T.cells * T.per_cell;
  if (total == 0) return cudaSuccess;
  if (total > kMaxInflowCandidates) return cudaErrorInvalidValue;
  const int nb = inflow_blocks(total);
  const InflowReach R = inflow_reach(P);
  cudaError_t e;
  const int items = inflow_items(total), tile = items * kThreads;
  const long long stride = (long long)nb * tile;
  e = launch_chained(inflow_stage_kernel, nb, kThreads, 0, st, P, T, R, iteration, total, items, block_counts, S.x, S.sp,
                     stride);
  if (e != cudaSuccess) return e;
  e = launch_scan_int(block_counts, block_offsets, nb, block_offsets + nb, block_offsets + nb + 1, st);
  if (e != cudaSuccess) return e;
  e = launch_chained(inflow_place_kernel<Store>, nb, kThreads, 0, st, tile, block_counts, block_offsets, count, capacity,
                     err, S.x, S.sp, stride, store);
  if (e != cudaSuccess) return e;
  return launch_chained(add_count_kernel, 1, 1, 0, st, count, block_offsets + nb, capacity);
}

cudaError_t launch_inflow_fused_c32(const KParams& P, const InflowTable& T, int iteration, PartC32 out, int* count,
                                    long long capacity, int* block_counts, int* block_offsets, int* err,
                                    const InflowStage& stage, cudaStream_t st) {
  return inflow_fused(P, T, iteration, StoreC32{P, out}, count, capacity, block_counts, block_offsets, err, stage,
                      st);
}

cudaError_t launch_inflow_fused_f64(const KParams& P, const InflowTable& T, int iteration, PartF64 out, int* count,
                                    long long capacity, int* block_counts, int* block_offsets, int* err,
                                    const InflowStage& stage, cudaStream_t st) {
  return inflow_fused(P, T, iteration, StoreF64{out}, count, capacity, block_counts, block_offsets, err, stage, st);
}

long long inflow_stage_slots(long long candidates) { return (long long)inflow_blocks(candidates) * inflow_items(candidates) * kThreads; }

cudaError_t launch_produce_emit_f64(const KParams& P, int iteration, const int* offsets, PartF64 out, int* count,
                                    long long capacity, int* err, cudaStream_t st) {
  long long cells = (long long)P.nx * P.ny * P.nz;
  cudaError_t e = launch_chained(produce_emit_kernel<StoreF64>, grid_for(cells), kThreads, 0, st, P, iteration, offsets, count,
                                 capacity, err, StoreF64{out});
  if (e != cudaSuccess) return e;
  return launch_chained(add_count_kernel, 1, 1, 0, st, count, offsets + cells, capacity);
}

cudaError_t launch_produce_emit_c32(const KParams& P, int iteration, const int* offsets, PartC32 out, int* count,
                                    long long capacity, int* err, cudaStream_t st) {
  long long cells = (long long)P.nx * P.ny * P.nz;
  cudaError_t e = launch_chained(produce_emit_kernel<StoreC32>, grid_for(cells), kThreads, 0, st, P, iteration, offsets, count,
                                 capacity, err, StoreC32{P, out});
  if (e != cudaSuccess) return e;
  return launch_chained(add_count_kernel, 1, 1, 0, st, count, offsets + cells, capacity);
}

static int persistent_grid(long long n) {
  long long b = (n + kThreads - 1) / kThreads;
  if (b > 148LL * 16) b = 148LL * 16;
  return b < 1 ? 1 : int(b);
}

cudaError_t launch_advance_position_f64(const KParams& P, PartF64 a, long long n, double dt, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  note_launch();
  advance_position_f64_kernel<<<persistent_grid(n), kThreads, 0, st>>>(a, n, dt);
  return cudaGetLastError();
}

cudaError_t launch_transfer_f64(const KParams& P, PartF64 a, long long n, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  note_launch();
  transfer_f64_kernel<<<persistent_grid(n), kThreads, 0, st>>>(P, a, n);
  return cudaGetLastError();
}

cudaError_t launch_outflow_f64(const KParams& P, PartF64 a, long long n, uint2* words, int* block_counts,
                               int* block_offsets, int* count, int wrap, int* err, cudaStream_t st,
                               const OutflowSplit* split) {
  return launch_outflow_inplace(OutflowF64{P, a}, n, words, block_counts, block_offsets, count, wrap, err, st, split);
}

cudaError_t launch_advance_velocity_f64(const KParams& P, PartF64 a, long long n, const double* E, double dt,
                                        double deltat, int mode, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  note_launch();
  advance_velocity_f64_kernel<<<persistent_grid(n), kThreads, 0, st>>>(P, a, n, E, dt, deltat, mode);
  return cudaGetLastError();
}

cudaError_t launch_deposit_f64(const KParams& P, PartF64 a, long long n, unsigned long long* Nacc,
                               unsigned long long* Facc, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const cudaError_t e = launch_deposit_tile_f64<false>(P, a.x, a.y, a.z, a.sp, n, Nacc, st);
  if (e != cudaSuccess || !Facc) return e;
  note_launch();
  flux_f64_kernel<<<persistent_grid(n), kThreads, 0, st>>>(P, a, n, Facc);
  return cudaGetLastError();
}

cudaError_t launch_energy_particles_f64(const KParams& P, PartF64 a, long long n, ReduceBuf rb, cudaStream_t st) {
  int nb = persistent_grid(n > 0 ? n : 1);
  if (nb > rb.max_blocks) nb = rb.max_blocks;
  note_launch();
  energy_particles_f64_kernel<<<nb, kThreads, 0, st>>>(P, a, n, rb.partial);
  note_launch();
  finish_sum_kernel<<<1, 256, 0, st>>>(rb.partial, nb, 0.5, rb.result);
  return cudaGetLastError();
}

cudaError_t launch_cell_indices_f64(const KParams& P, PartF64 a, long long n, int* ijk, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  note_launch();
  cell_indices_f64_kernel<<<grid_for(n), kThreads, 0, st>>>(P, a, n, ijk);
  return cudaGetLastError();
}

}  // namespace picard

namespace picard {
cudaError_t launch_c32_to_f64(const KParams& P, PartC32 a, long long n, PartF64 out, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  note_launch();
  c32_to_f64_kernel<<<persistent_grid(n), kThreads, 0, st>>>(P, a, n, out);
  return cudaGetLastError();
}
cudaError_t launch_f64_to_c32(const KParams& P, PartF64 a, long long n, PartC32 out, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  note_launch();
  f64_to_c32_kernel<<<persistent_grid(n), kThreads, 0, st>>>(P, a, n, out);
  return cudaGetLastError();
}
}  // namespace picard

// ---------------------------------------------------------------------------
// Allocation-free deposit: picard_gpu_particles_gridify_noalloc.
//
// Some callers cannot allocate device memory at the point where they need a
// charge deposit: a host whose device memory is owned by another runtime's
// fixed pool (a Fortran program that manages its arrays through OpenACC or
// CUDA Fortran data regions), a serving loop that has already promised all of
// the HBM to resident runs, or a pipeline that cannot afford the device-wide
// synchronisation cudaFree implies.  For them this entry point takes the
// particle arrays and the output grids from the caller and keeps its only
// scratch -- the int64 fixed-point accumulators -- in the file-scope array
// below, so it calls no cudaMalloc, cudaFree or allocating library routine.
#include <string>

namespace picard {
KParams make_kparams(const picard_params& p);
int fail(int code, const std::string& msg);

namespace {

// Every device that loads the library holds this array (16 MiB) until the
// process exits.  All calls share it, so calls that overlap on the GPU race.
static __device__ __align__(256) unsigned long long g_noalloc_acc[PICARD_NOALLOC_MAX_WORDS];

// N(s, node) = n2p_s * acc * 2^-40 in the reference layout (species fastest),
// with the ghost folds of ParticlesGridify.f90:149-278; C = sum_s q_s N_s.
__global__ void finish_noalloc_kernel(KParams P, const unsigned long long* acc, double* N, double* C) {
  long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= P.nodes) return;
  int i = int(g % P.nxp), j = int((g / P.nxp) % P.nyp), k = int(g / ((long long)P.nxp * P.nyp));
  auto mirror = [](int v, int nn, int open) { return (v >= 1 && v <= nn) ? v : (open ? -1 : (v < 1 ? v + nn : v - nn)); };
  int mi = mirror(i, P.nx, P.xflow), mj = mirror(j, P.ny, P.yflow), mk = mirror(k, P.nz, P.zflow);
  double c = 0.0;
  for (int s = 0; s < P.species; ++s) {
    double v = 0.0;
    if (mi >= 0 && mj >= 0 && mk >= 0) {
      long long a = (long long)acc[(long long)s * P.nodes + node_index(P, mi, mj, mk)];
      v = P.n2p[s] * ((double)a * (1.0 / kDepositScale));
    }
    N[(long long)s + (long long)P.species * g] = v;
    c = c + v * P.charge[s];
  }
  C[g] = c;
}

}  // namespace
}  // namespace picard

extern "C" int picard_gpu_particles_gridify_noalloc(const picard_params* p, const double* x, const double* y,
                                                    const double* z, const int32_t* int_particles, int32_t num_local,
                                                    double* N, double* C, void* stream) {
  using namespace picard;
  if (!p) return fail(PICARD_ERR_BAD_ARG, "params is NULL");
  if (!(p->dxyz[0] > 0.0 && p->dxyz[1] > 0.0 && p->dxyz[2] > 0.0))
    return fail(PICARD_ERR_BAD_ARG, "params not derived (call picard_params_derive first)");
  if (p->species < 2 || p->species > 8) return fail(PICARD_ERR_BAD_ARG, "species must be in 2..8");
  if (p->nx < 1 || p->ny < 1 || p->nz < 1) return fail(PICARD_ERR_BAD_ARG, "grid dimensions must be positive");
  const long long nodes = (long long)(p->nx + 2) * (p->ny + 2) * (p->nz + 2);
  const long long words = nodes * p->species;
  if (words > (long long)PICARD_NOALLOC_MAX_WORDS)
    return fail(PICARD_ERR_BAD_ARG, "the allocation-free deposit needs species*(Nx+2)*(Ny+2)*(Nz+2) = " +
                                        std::to_string(words) + " accumulator words; its fixed scratch holds " +
                                        std::to_string((long long)PICARD_NOALLOC_MAX_WORDS));
  if (num_local < 0) return fail(PICARD_ERR_BAD_ARG, "num_local must be >= 0");
  if (num_local > 0 && (!x || !y || !z || !int_particles)) return fail(PICARD_ERR_BAD_ARG, "particle array is NULL");
  if (!N || !C) return fail(PICARD_ERR_BAD_ARG, "output array is NULL");
  // The array's host-side name is not a device address.  Its address on the
  // current device is looked up on every call (a table lookup once the
  // library's device code is loaded), so nothing cached outlives a
  // cudaDeviceReset.  The first call on a device loads that code: make it
  // before any stream capture.
  void* q = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&q, g_noalloc_acc);
  if (e != cudaSuccess) return fail(PICARD_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
  unsigned long long* acc = static_cast<unsigned long long*>(q);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const KParams K = make_kparams(*p);
  // the array keeps the previous call's sums: clear the part this call uses
  e = cudaMemsetAsync(acc, 0, sizeof(unsigned long long) * (size_t)words, st);
  if (e != cudaSuccess) return fail(PICARD_ERR_CUDA, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
  e = launch_deposit_tile_f64<true>(K, x, y, z, int_particles, num_local, acc, st);
  if (e != cudaSuccess) return fail(PICARD_ERR_CUDA, std::string("deposit launch: ") + cudaGetErrorString(e));
  note_launch();
  finish_noalloc_kernel<<<grid_for(nodes), kThreads, 0, st>>>(K, acc, N, C);
  e = cudaGetLastError();
  if (e != cudaSuccess) return fail(PICARD_ERR_CUDA, std::string("deposit launch: ") + cudaGetErrorString(e));
  return PICARD_OK;
}
