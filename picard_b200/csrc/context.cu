// context.cu -- the C ABI of include/picard_gpu.h: context life cycle,
// transfers in the reference layouts, and one entry point per reference
// subroutine (each cites the routine it replaces).
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "context.cuh"
#include "picard_gpu.h"
#include "pinned.cuh"

using namespace picard;

#include <atomic>
#include <thread>

namespace picard {

static thread_local std::string g_last_error;
static std::atomic<long long> g_launches{0};

void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
long long launches_so_far() { return g_launches.load(std::memory_order_relaxed); }

int fail(int code, const std::string& msg) {
  g_last_error = msg;
  return code;
}

int check_cuda(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return PICARD_OK;
  // reported here: clear the runtime's last-error slot so that a later,
  // unrelated launch check does not report it again (sticky errors stay)
  (void)cudaGetLastError();
  return fail(PICARD_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

KParams make_kparams(const picard_params& p) {
  KParams K;
  std::memset(&K, 0, sizeof(K));
  K.nx = p.nx;
  K.ny = p.ny;
  K.nz = p.nz;
  K.nxp = p.nx + 2;
  K.nyp = p.ny + 2;
  K.nzp = p.nz + 2;
  K.nodes = (long long)K.nxp * K.nyp * K.nzp;
  K.species = p.species;
  K.xflow = p.xflow != 0;
  K.yflow = p.yflow != 0;
  K.zflow = p.zflow != 0;
  K.produce_dt_scaled = p.produce_dt_scaled;
  K.xmin = p.xmin; K.xmax = p.xmax; K.ymin = p.ymin; K.ymax = p.ymax; K.zmin = p.zmin; K.zmax = p.zmax;
  K.Lx_min = p.Lx_min; K.Lx_max = p.Lx_max; K.Ly_min = p.Ly_min; K.Ly_max = p.Ly_max;
  K.Lz_min = p.Lz_min; K.Lz_max = p.Lz_max;
  K.dx = p.dxyz[0];
  K.dy = p.dxyz[1];
  K.dz = p.dxyz[2];
  K.dV = p.dxyz[0] * p.dxyz[1] * p.dxyz[2];
  K.dt = p.dt;
  for (int c = 0; c < 3; ++c) {
    K.ve[c] = p.ve[c];
    K.E0[c] = p.E0[c];
    K.B0[c] = p.B0[c];
  }
  const double* m = p.mass;
  for (int s = 0; s < 8; ++s) {
    K.gyration[s] = p.gyration[s] != 0;
    K.fluid[s] = p.fluid[s] != 0;
    K.ipp[s] = p.ipp[s];
    K.epp[s] = p.epp[s];
    K.hpp[s] = p.hpp[s];
    K.mass[s] = p.mass[s];
    K.charge[s] = p.charge[s];
    K.kelvin[s] = p.kelvin[s];
    K.n2p[s] = p.n2p[s];
    K.eta[s] = p.eta[s];
    for (int c = 0; c < 3; ++c) {
      K.v0[s][c] = p.v0[s][c];
      K.tB[s][c] = p.tB[s][c];
      K.sB[s][c] = p.sB[s][c];
    }
    K.vn[s] = p.vn[s];
    K.Qn[s] = p.Qn[s];
    K.nu_i[s] = p.nu_i[s];
    K.nu_d[s] = p.nu_d[s];
    K.Ek[s] = p.Ek[s];
    K.ue[s] = K.uh[s] = K.ui[s] = 0.0;
  }
  // ParticlesProduce.f90:26-36
  for (int s = 0; s < p.species; ++s) {
    K.ue[s] = std::sqrt(2.0 * m[s] * p.Ek[s] * (1.0 / (m[0] * (m[s] + m[0]))));
    K.uh[s] = std::sqrt(2.0 * m[s] * p.Ek[s] * (1.0 / (m[1] * (m[s] + m[1]))));
    if (p.epp[s] > 0)
      K.ui[s] = std::sqrt(2.0 * m[0] * p.Ek[s] * (1.0 / (m[s] * (m[s] + m[0]))));
    else if (p.hpp[s] > 0)
      K.ui[s] = std::sqrt(2.0 * m[1] * p.Ek[s] * (1.0 / (m[s] * (m[s] + m[1]))));
  }
  K.seed = p.seed;
  return K;
}

// The guard shell BCinflow.f90 fills on one rank, in its loop order.
InflowTable make_inflow_table(const picard_params& p) {
  InflowTable T;
  std::memset(&T, 0, sizeof(T));
  const double dx = p.dxyz[0], dy = p.dxyz[1], dz = p.dxyz[2];
  const int Nx = p.nx, Ny = p.ny, Nz = p.nz;
  int ypos = (p.yflow && (p.Ly_max + 0.5 * dy > p.ymax)) ? 1 : 0;
  int yneg = (p.yflow && (p.Ly_min - 0.5 * dy < p.ymin)) ? 1 : 0;
  int zpos = (p.zflow && (p.Lz_max + 0.5 * dz > p.zmax)) ? 1 : 0;
  int zneg = (p.zflow && (p.Lz_min - 0.5 * dz < p.zmin)) ? 1 : 0;
  auto add = [&](int axis, int fixed, int o_lo, int o_n, int i_lo, int i_n, double edge) {
    InflowFace& F = T.f[T.nfaces++];
    F.axis = axis;
    F.fixed = fixed;
    F.o_lo = o_lo;
    F.o_n = o_n;
    F.i_lo = i_lo;
    F.i_n = i_n;
    F.edge = edge;
    F.first = T.cells;
    T.cells += (long long)o_n * i_n;
  };
  if (p.xflow && (p.Lx_max + 0.5 * dx > p.xmax))
    add(0, Nx + 2, 2 - zneg, Nz + zneg + zpos, 2 - yneg, Ny + yneg + ypos, p.Lx_max);
  if (p.xflow && (p.Lx_min - 0.5 * dx < p.xmin))
    add(0, 1, 2 - zneg, Nz + zneg + zpos, 2 - yneg, Ny + yneg + ypos, p.Lx_min - dx);
  if (ypos > 0) add(1, Ny + 2, 2, Nz + zpos, 2, Nx, p.Ly_max);
  if (yneg > 0) add(1, 1, 2 - zneg, Nz + zneg, 2, Nx, p.Ly_min - dy);
  if (zpos > 0) add(2, Nz + 2, 2 - yneg, Ny + yneg, 2, Nx, p.Lz_max);
  if (zneg > 0) add(2, 1, 2, Ny + ypos, 2, Nx, p.Lz_min - dz);
  T.group_prefix[0] = 0;
  for (int s = 0; s < 8; ++s)
    T.group_prefix[s + 1] = T.group_prefix[s] + (s < p.species ? p.ipp[s] * (1 + p.epp[s] + p.hpp[s]) : 0);
  T.per_cell = T.group_prefix[p.species];
  return T;
}

}  // namespace picard

namespace {

struct CudaPinned {
  static void* alloc(size_t bytes) {
    void* p = nullptr;
    if (cudaHostAlloc(&p, bytes, cudaHostAllocPortable) == cudaSuccess) return p;
    (void)cudaGetLastError();
    return nullptr;
  }
  static void free(void* p) { cudaFreeHost(p); }
};
// never destroyed: blocks kept at exit go with the process, after the driver
PinnedPool<CudaPinned>& pinned() {
  static auto* p = new PinnedPool<CudaPinned>();
  return *p;
}

template <class T>
int dalloc(picard_ctx* c, T*& p, size_t n) {
  void* q = nullptr;
  size_t bytes = std::max<size_t>(n, 1) * sizeof(T);
  // stream-ordered: creating or destroying a context does not synchronise
  // the device, so contexts of concurrent runs come and go independently
  cudaError_t e = cudaMallocAsync(&q, bytes, c->st);
  if (e != cudaSuccess) return check_cuda(e, ("cudaMallocAsync(" + std::to_string(bytes) + " B)").c_str());
  c->allocs.push_back(q);
  e = cudaMemsetAsync(q, 0, bytes, c->st);
  if (e != cudaSuccess) return check_cuda(e, "cudaMemsetAsync");
  p = static_cast<T*>(q);
  return PICARD_OK;
}

// Frees one allocation of dalloc on the context's stream.
void release(picard_ctx* c, void* q) {
  auto it = std::find(c->allocs.begin(), c->allocs.end(), q);
  if (it == c->allocs.end()) return;
  c->allocs.erase(it);
  cudaFreeAsync(q, c->st);
}

}  // namespace

namespace picard {
int dev_alloc(picard_ctx* c, void** p, size_t bytes) {
  unsigned char* q = nullptr;
  PICARD_TRY(dalloc(c, q, bytes));
  *p = q;
  return PICARD_OK;
}
}  // namespace picard

namespace {

struct Sizes {
  long long cap, nodes, cells, dsize;
  int species, nb_compact, nb_jacobi, nb_inflow;
};

Sizes sizes_of(const picard_params& p) {
  Sizes s;
  s.cap = p.max_per_proc;
  s.nodes = (long long)(p.nx + 2) * (p.ny + 2) * (p.nz + 2);
  s.cells = (long long)p.nx * p.ny * p.nz;
  s.dsize = (long long)(2 * p.nx + 1) * (2 * p.ny + 1) * (2 * p.nz + 1);
  s.species = p.species;
  s.nb_compact = compact_blocks(s.cap) + 1;
  const InflowTable T = make_inflow_table(p);
  s.nb_inflow = T.cells * T.per_cell > 0 ? inflow_blocks(T.cells * T.per_cell) : 0;
  KParams K = make_kparams(p);
  s.nb_jacobi = jacobi_geom(K).nblocks;
  return s;
}

int validate(const picard_params* p, int layout, int solver) {
  if (!p) return fail(PICARD_ERR_BAD_ARG, "params is NULL");
  if (p->nx < 1 || p->ny < 1 || p->nz < 1) return fail(PICARD_ERR_BAD_ARG, "grid dimensions must be positive");
  if (p->species < 2 || p->species > 8) return fail(PICARD_ERR_BAD_ARG, "species must be in 2..8");
  if (p->max_per_proc < 1) return fail(PICARD_ERR_BAD_ARG, "max_per_proc must be positive");
  if (layout != PICARD_LAYOUT_F64 && layout != PICARD_LAYOUT_CELL32) return fail(PICARD_ERR_BAD_ARG, "unknown layout");
  if (solver != PICARD_SOLVER_F64 && solver != PICARD_SOLVER_F32_REFINE && solver != PICARD_SOLVER_SPECTRAL)
    return fail(PICARD_ERR_BAD_ARG, "unknown solver");
  if (layout == PICARD_LAYOUT_CELL32 &&
      (p->nx + 2 > (int)kCellMaskX || p->ny + 2 > (int)kCellMaskY || p->nz + 2 > (int)kCellMaskZ))
    return fail(PICARD_ERR_BAD_ARG, "CELL32 layout holds at most 2045 x 2045 x 1021 cells");
  if (!(p->dxyz[0] > 0.0 && p->dxyz[1] > 0.0 && p->dxyz[2] > 0.0))
    return fail(PICARD_ERR_BAD_ARG, "params not derived (call picard_params_derive first)");
  return PICARD_OK;
}

int sync_count(picard_ctx* c) {
  PICARD_CUDA(cudaMemcpyAsync(c->h_pinned_i, c->d_count, sizeof(int), cudaMemcpyDeviceToHost, c->st));
  PICARD_CUDA(cudaStreamSynchronize(c->st));
  c->stats.d2h_bytes += sizeof(int);
  c->num_local = c->h_pinned_i[0];
  return PICARD_OK;
}

// The host's count to the device, in stream order (the value travels with the
// launch: nothing to wait for).
__global__ void set_count_kernel(int* count, int value) { *count = value; }

int push_count(picard_ctx* c) {
  note_launch();
  set_count_kernel<<<1, 1, 0, c->st>>>(c->d_count, int(c->num_local));
  return check_cuda(cudaGetLastError(), "set_count_kernel");
}

int report_dev_err(picard_ctx* c, int e) {
  if (e == kDevCapacity) {
    cudaMemsetAsync(c->d_err, 0, sizeof(int), c->st);
    return fail(PICARD_ERR_CAPACITY, "particle capacity max_per_proc exceeded on the device");
  }
  if (e == kDevTimeout) {
    cudaMemsetAsync(c->d_err, 0, sizeof(int), c->st);
    return fail(PICARD_ERR_TIMEOUT, "a bounded device wait gave up");
  }
  if (e == kDevRange) {
    cudaMemsetAsync(c->d_err, 0, sizeof(int), c->st);
    return fail(PICARD_ERR_STATE, "a particle move left its range on the device and was skipped");
  }
  return PICARD_OK;
}

int check_dev_err(picard_ctx* c) {
  PICARD_CUDA(cudaMemcpyAsync(c->h_pinned_i + 2, c->d_err, sizeof(int), cudaMemcpyDeviceToHost, c->st));
  PICARD_CUDA(cudaStreamSynchronize(c->st));
  c->stats.d2h_bytes += sizeof(int);
  return report_dev_err(c, c->h_pinned_i[2]);
}

int check_dev_err_timeout(picard_ctx* c) {
  PICARD_CUDA(cudaMemcpyAsync(c->h_pinned_i + 5, c->d_err, sizeof(int), cudaMemcpyDeviceToHost, c->st));
  PICARD_CUDA(cudaStreamSynchronize(c->st));
  c->stats.d2h_bytes += sizeof(int);
  if (c->h_pinned_i[5] == kDevTimeout) {
    cudaMemsetAsync(c->d_err, 0, sizeof(int), c->st);
    return fail(PICARD_ERR_TIMEOUT, "a tensor-core BCpotentials block timed out waiting for its MMAs");
  }
  return PICARD_OK;
}

int ensure_capacity(picard_ctx* c, long long add) {
  if (c->num_local + add > c->capacity)
    return fail(PICARD_ERR_CAPACITY, "particle count " + std::to_string(c->num_local + add) +
                                         " would exceed max_per_proc " + std::to_string(c->capacity));
  return PICARD_OK;
}

}  // namespace

namespace picard {
bool has_neutral_source(const KParams& K) {
  // ParticlesProduce.f90:62-73: the number of ions is int(rate + u), u < 1, and
  // the rate is 0 without an outflow speed, a production or an ionisation rate
  for (int s = 0; s < K.species; ++s)
    if (K.n2p[s] > 0.0 && K.vn[s] > 0.0 && !(K.Qn[s] == 0.0) && !(K.nu_i[s] == 0.0)) return true;
  return false;
}

int check_dev_err_public(picard_ctx* c) { return check_dev_err(c); }

int bc_potentials_async(picard_ctx* c) {
  if (c->bcpot_tensor == PICARD_BCPOT_FFT) return bc_potentials_fft(c);
  if (c->bcpot_tensor == PICARD_BCPOT_TENSOR) {
    if (!c->tc_cs) {
      long long cs = 0, pe = 0;
      bcpot_tc_scratch(c->K, &cs, &pe);
      unsigned short* csb = nullptr;
      PICARD_TRY(dalloc(c, csb, (size_t)cs));
      PICARD_TRY(dalloc(c, c->tc_partial, (size_t)pe));
      c->tc_cs = csb;
    }
    PICARD_CUDA(launch_bc_potentials_tc(c->K, c->C, c->D, c->U, c->tc_cs, c->tc_partial, c->d_err, c->st));
    return PICARD_OK;
  }
  const long long want = bc_direct_scratch(c->K);
  if (!c->bc_scratch && dalloc(c, c->bc_scratch, (size_t)want) != PICARD_OK) {
    // no room: the right-hand side's array, which the next solve writes before it reads it
    PICARD_CUDA(launch_bc_potentials(c->K, c->C, c->D, c->U, c->b, c->K.nodes, c->st));
    return PICARD_OK;
  }
  PICARD_CUDA(launch_bc_potentials(c->K, c->C, c->D, c->U, c->bc_scratch, want, c->st));
  return PICARD_OK;
}

static cudaError_t launch_outflow_split(picard_ctx* c, long long n, const OutflowSplit* sp) {
  if (c->layout == PICARD_LAYOUT_F64)
    return launch_outflow_f64(c->K, c->f64, n, c->out_words, c->blk_counts, c->blk_offsets, c->d_count, 0, c->d_err,
                              c->st, sp);
  return launch_outflow_c32(c->K, c->c32, n, c->out_words, c->blk_counts, c->blk_offsets, c->d_count, 0, c->d_err,
                            c->st, sp);
}

cudaError_t launch_outflow(picard_ctx* c, int wrap) {
  if (c->layout == PICARD_LAYOUT_F64)
    return launch_outflow_f64(c->K, c->f64, c->num_local, c->out_words, c->blk_counts, c->blk_offsets, c->d_count,
                              wrap, c->d_err, c->st);
  return launch_outflow_c32(c->K, c->c32, c->num_local, c->out_words, c->blk_counts, c->blk_offsets, c->d_count, wrap,
                            c->d_err, c->st);
}

cudaError_t launch_inflow_fused(picard_ctx* c, int iteration) {
  const long long cand = (long long)c->inflow.cells * c->inflow.per_cell;
  if (cand > 0 && !c->inflow_stage.x) {
    const long long slots = inflow_stage_slots(cand);
    double* x = nullptr;
    int8_t* sp = nullptr;
    if (dalloc(c, x, (size_t)(6 * slots)) != PICARD_OK || dalloc(c, sp, (size_t)slots) != PICARD_OK)
      return cudaErrorMemoryAllocation;
    c->inflow_stage.x = x;
    c->inflow_stage.sp = sp;
  }
  if (c->layout == PICARD_LAYOUT_F64)
    return launch_inflow_fused_f64(c->K, c->inflow, iteration, c->f64, c->d_count, c->capacity, c->inflow_counts,
                                   c->inflow_offsets, c->d_err, c->inflow_stage, c->st);
  return launch_inflow_fused_c32(c->K, c->inflow, iteration, c->c32, c->d_count, c->capacity, c->inflow_counts,
                                 c->inflow_offsets, c->d_err, c->inflow_stage, c->st);
}

// The count and the error word lie side by side: one copy.
int count_issue(picard_ctx* c) {
  PICARD_CUDA(cudaMemcpyAsync(c->h_pinned_i + 8, c->d_count, 2 * sizeof(int), cudaMemcpyDeviceToHost, c->st));
  c->stats.d2h_bytes += 2 * sizeof(int);
  return PICARD_OK;
}

int count_collect(picard_ctx* c) {
  PICARD_CUDA(cudaStreamSynchronize(c->st));
  PICARD_TRY(report_dev_err(c, c->h_pinned_i[9]));
  c->num_local = c->h_pinned_i[8];
  return PICARD_OK;
}
}  // namespace picard

// ======================================================================= ABI

extern "C" {

const char* picard_gpu_last_error(void) { return g_last_error.c_str(); }

int picard_gpu_pool_keep(int32_t device, uint64_t bytes) {
  int count = 0;
  PICARD_CUDA(cudaGetDeviceCount(&count));
  if (device < 0 || device >= count) return fail(PICARD_ERR_BAD_ARG, "no such device");
  cudaMemPool_t pool;
  PICARD_CUDA(cudaDeviceGetDefaultMemPool(&pool, device));
  PICARD_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &bytes));
  pinned().set_keep(device, (size_t)bytes);
  return PICARD_OK;
}

int picard_gpu_footprint(const picard_params* p, int32_t layout, int32_t solver, uint64_t* bytes) {
  PICARD_TRY(validate(p, layout, solver));
  if (!bytes) return fail(PICARD_ERR_BAD_ARG, "bytes is NULL");
  Sizes s = sizes_of(*p);
  double per_particle = layout == PICARD_LAYOUT_F64 ? 49.0 : 29.0;
  double b = per_particle * (double)s.cap;
  b += (double)s.nodes * (8.0 * s.species /*Nacc*/ + 8.0 * s.species /*N*/ + 8 * 3 /*C,U,b*/ + 24 /*E*/ + 8 /*U1*/);
  if (layout == PICARD_LAYOUT_CELL32) b += 16.0 * s.nodes;
  if (solver == PICARD_SOLVER_F64) b += 8.0 * s.nodes;
  else if (solver == PICARD_SOLVER_SPECTRAL) b += (double)spectral_bytes(make_kparams(*p));
  else b += 16.0 * (double)f32_elems(make_kparams(*p));
  b += 8.0 * (double)s.dsize;
  b += 8.0 * (double)s.cells;                // produce counts + offsets
  b += 8.0 * (double)s.nb_compact * (3 + kOutflowWordsPerBlock);  // BCoutflow scratch
  b += 8.0 * (double)s.nb_inflow * 2;        // fused BCinflow scan
  {
    const InflowTable T = make_inflow_table(*p);  // fused BCinflow survivors' staging area
    const long long cand = (long long)T.cells * T.per_cell;
    if (cand > 0) b += 49.0 * (double)inflow_stage_slots(cand);
  }
  b += 8.0 * (kMaxSweepsPerRound + 1.0) * s.nb_jacobi;  // sweep partials
  if (layout == PICARD_LAYOUT_CELL32) {      // BCpotentials scratch of the layout's default method
    const KParams K = make_kparams(*p);
    if (bcpot_fft_supported(K)) {
      b += (double)bcpot_fft_bytes(K);
    } else {
      long long cs = 0, pe = 0;
      bcpot_tc_scratch(K, &cs, &pe);
      b += 2.0 * (double)cs + 8.0 * (double)pe;
    }
  }
  *bytes = (uint64_t)b;
  return PICARD_OK;
}

int picard_gpu_create(const picard_params* p, int32_t layout, int32_t solver, picard_ctx** out) {
  PICARD_TRY(validate(p, layout, solver));
  if (!out) return fail(PICARD_ERR_BAD_ARG, "out is NULL");
  picard_ctx* c = new picard_ctx();
  pinned().context(1);
  c->prm = *p;
  c->K = make_kparams(*p);
  c->layout = layout;
  c->solver = solver;
  c->capacity = p->max_per_proc;
  c->inflow = make_inflow_table(*p);
  c->G = jacobi_geom(c->K);
  c->bcpot_tensor = layout != PICARD_LAYOUT_CELL32 ? PICARD_BCPOT_DIRECT
                    : bcpot_fft_supported(c->K)   ? PICARD_BCPOT_FFT
                                                  : PICARD_BCPOT_TENSOR;
  int rc = PICARD_OK;
  auto bail = [&](int code) {
    picard_gpu_destroy(c);
    return code;
  };
  if (cudaGetDevice(&c->device) != cudaSuccess) return bail(fail(PICARD_ERR_CUDA, "no CUDA device"));
  if ((rc = check_cuda(cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking), "cudaStreamCreate"))) return bail(rc);
  Sizes s = sizes_of(*p);
  const long long cap = s.cap;
  // one particle buffer: BCoutflow removes in place
  if (layout == PICARD_LAYOUT_F64) {
    PartF64& a = c->f64;
    if ((rc = dalloc(c, a.x, cap)) || (rc = dalloc(c, a.y, cap)) || (rc = dalloc(c, a.z, cap)) ||
        (rc = dalloc(c, a.vx, cap)) || (rc = dalloc(c, a.vy, cap)) || (rc = dalloc(c, a.vz, cap)) ||
        (rc = dalloc(c, a.sp, cap)))
      return bail(rc);
  } else {
    PartC32& a = c->c32;
    if ((rc = dalloc(c, a.cell, cap)) || (rc = dalloc(c, a.fx, cap)) || (rc = dalloc(c, a.fy, cap)) ||
        (rc = dalloc(c, a.fz, cap)) || (rc = dalloc(c, a.vx, cap)) || (rc = dalloc(c, a.vy, cap)) ||
        (rc = dalloc(c, a.vz, cap)) || (rc = dalloc(c, a.sp, cap)))
      return bail(rc);
  }
  const long long nn = s.nodes;
  if ((rc = dalloc(c, c->d_count, 2)) || (rc = dalloc(c, c->d_info, (1 + kJumpRounds) * kInfoStride)) ||
      (rc = dalloc(c, c->Nacc, nn * s.species)) || (rc = dalloc(c, c->N, nn * s.species)) ||
      (rc = dalloc(c, c->C, nn)) || (rc = dalloc(c, c->U, nn)) || (rc = dalloc(c, c->E, 3 * nn)) ||
      (rc = dalloc(c, c->D, s.dsize)) || (rc = dalloc(c, c->b, nn)) || (rc = dalloc(c, c->U1, nn)))
    return bail(rc);
  c->d_err = c->d_count + 1;  // read together with the count
  if (layout == PICARD_LAYOUT_CELL32 && (rc = dalloc(c, c->E32, nn))) return bail(rc);
  if (solver == PICARD_SOLVER_F64) {
    if ((rc = dalloc(c, c->Usnap, nn))) return bail(rc);
  } else if (solver == PICARD_SOLVER_SPECTRAL) {
    if ((rc = spectral_alloc(c))) return bail(rc);
  } else {
    const long long fe = f32_elems(c->K);
    if ((rc = dalloc(c, c->w[0], fe)) || (rc = dalloc(c, c->w[1], fe)) || (rc = dalloc(c, c->r, 2 * fe))) return bail(rc);
    if (c->G.tma) {
      int e0 = make_tensor_map(&c->tmw[0], c->w[0], c->K, 40, 10, c->G.zc + 2);
      int e1 = make_tensor_map(&c->tmw[1], c->w[1], c->K, 40, 10, c->G.zc + 2);
      int e2 = make_tensor_map(&c->tmr[0], c->r, c->K, 32, 8, c->G.zc);
      int e3 = make_tensor_map(&c->tmr[1], c->r + fe, c->K, 32, 8, c->G.zc);
      e0 |= make_tensor_map(&c->tmw2[0], c->w[0], c->K, 72, 10, c->G.zc + 2);
      e1 |= make_tensor_map(&c->tmw2[1], c->w[1], c->K, 72, 10, c->G.zc + 2);
      e2 |= make_tensor_map(&c->tmr2[0], c->r, c->K, 64, 8, c->G.zc);
      e3 |= make_tensor_map(&c->tmr2[1], c->r + fe, c->K, 64, 8, c->G.zc);
      if (c->G.zc <= 8) {
        e0 |= make_tensor_map(&c->tmw3[0], c->w[0], c->K, 72, 12, c->G.zc + 4);
        e1 |= make_tensor_map(&c->tmw3[1], c->w[1], c->K, 72, 12, c->G.zc + 4);
        e2 |= make_tensor_map(&c->tmr3[0], c->r, c->K, 72, 10, c->G.zc + 2);
        e3 |= make_tensor_map(&c->tmr3[1], c->r + fe, c->K, 72, 10, c->G.zc + 2);
      }
      if (e0 || e1 || e2 || e3)
        return bail(fail(PICARD_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string(e0 | e1 | e2 | e3) + ")"));
    }
  }
  if ((rc = dalloc(c, c->partials, (size_t)(c->m_max + 1) * c->G.nblocks)) ||
      (rc = dalloc(c, c->r2, c->m_max + 1)))
    return bail(rc);
  int scan_extra = scan_scratch_ints(s.nb_compact) + 4;
  if ((rc = dalloc(c, c->blk_counts, s.nb_compact)) ||
      (rc = dalloc(c, c->blk_offsets, 2 * (size_t)s.nb_compact + 2 + scan_extra)) ||
      (rc = dalloc(c, c->out_words, (size_t)kOutflowWordsPerBlock * s.nb_compact)))
    return bail(rc);
  if (s.nb_inflow > 0 &&
      ((rc = dalloc(c, c->inflow_counts, s.nb_inflow)) ||
       (rc = dalloc(c, c->inflow_offsets, (size_t)s.nb_inflow + 2 + scan_scratch_ints(s.nb_inflow) + 4))))
    return bail(rc);
  int cells = int(s.cells);
  if ((rc = dalloc(c, c->cell_counts, cells)) ||
      (rc = dalloc(c, c->cell_offsets, (size_t)cells + 2 + scan_scratch_ints(cells) + 4)))
    return bail(rc);
  c->red_blocks = std::max<int>(148 * 16, rhs_blocks(c->K));
  if ((rc = dalloc(c, c->red_partial, c->red_blocks)) || (rc = dalloc(c, c->red_result, 8))) return bail(rc);
  static_assert(sizeof(double) * (kMaxSweepsPerRound + 64) + sizeof(int) * 16 <= kPinnedBlock[0], "mailbox");
  c->h_pinned = static_cast<double*>(pinned().get(0));
  if (!c->h_pinned) return bail(fail(PICARD_ERR_CUDA, "no pinned host memory"));
  c->h_pinned_i = reinterpret_cast<int*>(c->h_pinned + c->m_max + 64);
  for (int e = 0; e < 4; ++e)
    if ((rc = check_cuda(cudaEventCreate(&c->ev[e]), "cudaEventCreate"))) return bail(rc);
  for (int e = 0; e < 12; ++e)
    if ((rc = check_cuda(cudaEventCreate(&c->pev[e]), "cudaEventCreate"))) return bail(rc);
  if ((rc = tune_sweep(c, false))) return bail(rc);
  if ((rc = check_cuda(cudaStreamSynchronize(c->st), "create"))) return bail(rc);
  c->launches_at_reset = launches_so_far();
  *out = c;
  return PICARD_OK;
}

int picard_gpu_destroy(picard_ctx* c) {
  if (!c) return PICARD_OK;
  if (c->st) {
    for (void* q : c->allocs) cudaFreeAsync(q, c->st);
    cudaStreamSynchronize(c->st);
  }
  bcpot_fft_free(c);
  pinned().put(0, c->h_pinned);
  pinned().context(-1);
  for (int e = 0; e < 4; ++e)
    if (c->ev[e]) cudaEventDestroy(c->ev[e]);
  for (int e = 0; e < 12; ++e)
    if (c->pev[e]) cudaEventDestroy(c->pev[e]);
  if (c->st) cudaStreamDestroy(c->st);
  delete c;
  return PICARD_OK;
}

int picard_gpu_synchronize(picard_ctx* c) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  PICARD_CUDA(cudaStreamSynchronize(c->st));
  return PICARD_OK;
}

int picard_gpu_get_stats(picard_ctx* c, picard_stats* out) {
  if (!c || !out) return fail(PICARD_ERR_BAD_ARG, "NULL argument");
  *out = c->stats;
  out->kernel_launches = launches_so_far() - c->launches_at_reset;
  out->last_sweeps = c->last_sweeps;
  return PICARD_OK;
}

int picard_gpu_reset_stats(picard_ctx* c) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  c->stats = picard_stats{};
  c->launches_at_reset = launches_so_far();
  return PICARD_OK;
}

int picard_gpu_get_stream(picard_ctx* c, void** stream) {
  if (!c || !stream) return fail(PICARD_ERR_BAD_ARG, "NULL argument");
  *stream = (void*)c->st;
  return PICARD_OK;
}

int picard_gpu_get_num_local(picard_ctx* c, int32_t* n) {
  if (!c || !n) return fail(PICARD_ERR_BAD_ARG, "NULL argument");
  *n = int32_t(c->num_local);
  return PICARD_OK;
}

// ------------------------------------------------------------ transfers

int picard_gpu_set_particles(picard_ctx* c, const double* rp, const int32_t* ip, int32_t n) {
  if (!c || (n > 0 && (!rp || !ip))) return fail(PICARD_ERR_BAD_ARG, "NULL argument");
  if (n < 0 || n > c->capacity) return fail(PICARD_ERR_CAPACITY, "num_local exceeds max_per_proc");
  std::vector<double> soa((size_t)6 * n);
  std::vector<int8_t> sp(n);
  for (int32_t p = 0; p < n; ++p) {
    for (int q = 0; q < 6; ++q) soa[(size_t)q * n + p] = rp[(size_t)8 * p + q];
    if (ip[p] < 1 || ip[p] > c->prm.species) return fail(PICARD_ERR_BAD_ARG, "int_particles holds an unknown species");
    sp[p] = int8_t(ip[p] - 1);
  }
  PartF64 dst;
  std::vector<void*> tmp;
  if (c->layout == PICARD_LAYOUT_F64) {
    dst = c->f64;
  } else {
    double* buf = nullptr;
    int8_t* sb = nullptr;
    PICARD_CUDA(cudaMallocAsync(&buf, sizeof(double) * 6 * std::max<int32_t>(n, 1), c->st));
    PICARD_CUDA(cudaMallocAsync(&sb, std::max<int32_t>(n, 1), c->st));
    tmp = {buf, sb};
    dst.x = buf;
    dst.y = buf + n;
    dst.z = buf + 2 * (size_t)n;
    dst.vx = buf + 3 * (size_t)n;
    dst.vy = buf + 4 * (size_t)n;
    dst.vz = buf + 5 * (size_t)n;
    dst.sp = sb;
  }
  double* cols[6] = {dst.x, dst.y, dst.z, dst.vx, dst.vy, dst.vz};
  for (int q = 0; q < 6; ++q)
    PICARD_CUDA(cudaMemcpyAsync(cols[q], soa.data() + (size_t)q * n, sizeof(double) * n, cudaMemcpyHostToDevice, c->st));
  PICARD_CUDA(cudaMemcpyAsync(dst.sp, sp.data(), n, cudaMemcpyHostToDevice, c->st));
  if (c->layout == PICARD_LAYOUT_CELL32) PICARD_CUDA(launch_f64_to_c32(c->K, dst, n, c->c32, c->st));
  for (void* q : tmp) cudaFreeAsync(q, c->st);
  PICARD_CUDA(cudaStreamSynchronize(c->st));
  c->stats.h2d_bytes += (int64_t)n * 49;
  c->num_local = n;
  return push_count(c);
}

int picard_gpu_get_particles(picard_ctx* c, double* rp, int32_t* ip, int32_t capacity, int32_t* num_local) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  const long long n = c->num_local;
  if (num_local) *num_local = int32_t(n);
  if (!rp && !ip) return PICARD_OK;
  if (capacity < n) return fail(PICARD_ERR_CAPACITY, "host arrays smaller than num_local");
  PartF64 src;
  std::vector<void*> tmp;
  if (c->layout == PICARD_LAYOUT_F64) {
    src = c->f64;
  } else {
    double* buf = nullptr;
    int8_t* sb = nullptr;
    PICARD_CUDA(cudaMallocAsync(&buf, sizeof(double) * 6 * std::max<long long>(n, 1), c->st));
    PICARD_CUDA(cudaMallocAsync(&sb, std::max<long long>(n, 1), c->st));
    tmp = {buf, sb};
    src.x = buf;
    src.y = buf + n;
    src.z = buf + 2 * n;
    src.vx = buf + 3 * n;
    src.vy = buf + 4 * n;
    src.vz = buf + 5 * n;
    src.sp = sb;
    PICARD_CUDA(launch_c32_to_f64(c->K, c->c32, n, src, c->st));
  }
  std::vector<double> soa((size_t)6 * n);
  std::vector<int8_t> sp(n);
  double* cols[6] = {src.x, src.y, src.z, src.vx, src.vy, src.vz};
  for (int q = 0; q < 6; ++q)
    PICARD_CUDA(cudaMemcpyAsync(soa.data() + (size_t)q * n, cols[q], sizeof(double) * n, cudaMemcpyDeviceToHost, c->st));
  PICARD_CUDA(cudaMemcpyAsync(sp.data(), src.sp, n, cudaMemcpyDeviceToHost, c->st));
  for (void* q : tmp) cudaFreeAsync(q, c->st);
  PICARD_CUDA(cudaStreamSynchronize(c->st));
  c->stats.d2h_bytes += (int64_t)n * 49;
  for (long long p = 0; p < n; ++p) {
    if (rp) {
      for (int q = 0; q < 6; ++q) rp[(size_t)8 * p + q] = soa[(size_t)q * n + p];
      rp[(size_t)8 * p + 6] = 0.0;
      rp[(size_t)8 * p + 7] = 0.0;
    }
    if (ip) ip[p] = int32_t(sp[p]) + 1;
  }
  return PICARD_OK;
}

static int field_geometry(picard_ctx* c, int which, double** dev, int* ncomp, long long* n) {
  const long long nn = c->K.nodes;
  const int S = c->prm.species;
  switch (which) {
    case PICARD_FIELD_U: *dev = c->U; *ncomp = 1; *n = nn; return PICARD_OK;
    case PICARD_FIELD_C: *dev = c->C; *ncomp = 1; *n = nn; return PICARD_OK;
    case PICARD_FIELD_E: *dev = c->E; *ncomp = 3; *n = nn; return PICARD_OK;
    case PICARD_FIELD_N: *dev = c->N; *ncomp = S; *n = nn; return PICARD_OK;
    case PICARD_FIELD_F:
      if (!c->F) return fail(PICARD_ERR_STATE, "flux F exists after picard_gpu_particles_gridify_all");
      *dev = c->F; *ncomp = 3 * S; *n = nn; return PICARD_OK;
    case PICARD_FIELD_D:
      *dev = c->D; *ncomp = 1;
      *n = (long long)(2 * c->prm.nx + 1) * (2 * c->prm.ny + 1) * (2 * c->prm.nz + 1);
      return PICARD_OK;
  }
  return fail(PICARD_ERR_BAD_ARG, "unknown field");
}

// Device planes [comp][node] <-> reference order (comp fastest).  For F the
// device plane index is s*3 + c and the reference order is F(s, c, node).
static inline size_t ref_index(int which, int S, int plane, long long g) {
  if (which == PICARD_FIELD_F) {
    int s = plane / 3, c = plane % 3;
    return (size_t)s + (size_t)S * ((size_t)c + 3 * (size_t)g);
  }
  int ncomp = which == PICARD_FIELD_E ? 3 : (which == PICARD_FIELD_N ? S : 1);
  return (size_t)plane + (size_t)ncomp * (size_t)g;
}

// Elements [first, first + count) of a field in the reference order, from its
// planes: component c of node g lies in plane c, or for F (fs species) in plane
// (c % fs) * 3 + c / fs.  Written straight to pinned host memory in whole lines.
__global__ void __launch_bounds__(256) field_piece_kernel(const double* __restrict__ planes, long long nodes, int ncomp,
                                                          int fs, long long first, long long count,
                                                          double* __restrict__ out) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < count; t += (long long)gridDim.x * blockDim.x) {
    const long long e = first + t, g = e / ncomp;
    const int c = int(e - g * ncomp);
    const int plane = fs ? (c % fs) * 3 + c / fs : c;
    out[t] = planes[plane * nodes + g];
  }
}

int picard_gpu_get_field(picard_ctx* c, int32_t which, double* out) {
  if (!c || !out) return fail(PICARD_ERR_BAD_ARG, "NULL argument");
  double* dev;
  int ncomp;
  long long n;
  PICARD_TRY(field_geometry(c, which, &dev, &ncomp, &n));
  // Pieces of up to 4 MB through pinned memory, the components brought into the
  // reference order on the device; up to four host threads copy them on, each
  // with its own pinned block, so the pieces of one are under way while another's
  // are copied; one that gets no pinned block copies its pieces through pageable
  // memory.  (U of 256 x 128 x 128 2.5 ms, N 6.2; one pageable copy into a
  // scratch array and a loop over it took 21 and 79.)
  const long long total = (long long)ncomp * n, piece = (long long)(kPinnedBlock[1] / sizeof(double));
  const long long pieces = (total + piece - 1) / piece;
  const int fs = which == PICARD_FIELD_F ? c->prm.species : 0;
  const int workers = int(std::min<long long>(4, (pieces + 1) / 2));
  std::array<int, 4> status{};  // PICARD_OK
  std::array<std::string, 4> message;
  std::atomic<long long> next{0};
  // elements [first, first + count) without pinned memory: their nodes of every plane, put in order here
  auto copy_pageable = [&](std::vector<double>& h, long long first, long long count) -> cudaError_t {
    const long long g0 = first / ncomp, nodes = (first + count - 1) / ncomp + 1 - g0;
    h.resize((size_t)(ncomp * nodes));
    cudaError_t e = cudaSuccess;
    for (int pl = 0; pl < ncomp && e == cudaSuccess; ++pl)
      e = cudaMemcpyAsync(h.data() + pl * nodes, dev + pl * n + g0, sizeof(double) * nodes, cudaMemcpyDeviceToHost, c->st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->st);
    if (e != cudaSuccess) return e;
    for (int pl = 0; pl < ncomp; ++pl)
      for (long long g = 0; g < nodes; ++g) {
        const long long at = (long long)ref_index(which, c->prm.species, pl, g0 + g);
        if (at >= first && at < first + count) out[at] = h[(size_t)(pl * nodes + g)];
      }
    return cudaSuccess;
  };
  auto work = [&](int w) {
    auto run = [&]() -> int {
      double* stage = static_cast<double*>(pinned().get(1));
      std::vector<double> h;  // where there is no pinned block
      cudaEvent_t done = nullptr;
      int rc = check_cuda(cudaEventCreateWithFlags(&done, cudaEventDisableTiming), "cudaEventCreate");
      for (long long q; rc == PICARD_OK && (q = next.fetch_add(1)) < pieces;) {
        const long long first = q * piece, count = std::min(piece, total - first);
        cudaError_t e;
        if (!stage) {
          rc = check_cuda(copy_pageable(h, first, count), "field copy");
          continue;
        }
        if (ncomp == 1) {
          e = cudaMemcpyAsync(stage, dev + first, sizeof(double) * count, cudaMemcpyDeviceToHost, c->st);
        } else {
          note_launch();
          field_piece_kernel<<<int(std::min<long long>((count + 255) / 256, 148LL * 8)), 256, 0, c->st>>>(
              dev, n, ncomp, fs, first, count, stage);
          e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaEventRecord(done, c->st);
        if (e == cudaSuccess) e = cudaEventSynchronize(done);
        rc = check_cuda(e, "field copy");
        if (rc == PICARD_OK) std::memcpy(out + first, stage, sizeof(double) * count);
      }
      if (done) cudaEventDestroy(done);
      if (rc != PICARD_OK) cudaStreamSynchronize(c->st);  // nothing writes to the block any more
      pinned().put(1, stage);
      return rc;
    };
    int device = c->device;  // the calling thread's device is put back
    try {
      status[w] = check_cuda(cudaGetDevice(&device), "cudaGetDevice");
      if (status[w] == PICARD_OK && device != c->device) status[w] = check_cuda(cudaSetDevice(c->device), "cudaSetDevice");
      if (status[w] == PICARD_OK) status[w] = run();
      if (status[w] != PICARD_OK) message[w] = picard_gpu_last_error();
    } catch (const std::exception&) {
      status[w] = PICARD_ERR_CUDA;  // out of host memory
    }
    if (device != c->device) cudaSetDevice(device);
  };
  std::array<std::thread, 3> others;
  for (int w = 1; w < workers; ++w) {
    try {
      others[w - 1] = std::thread(work, w);
    } catch (const std::exception&) {
      break;  // fewer threads share the pieces
    }
  }
  work(0);
  for (std::thread& th : others)
    if (th.joinable()) th.join();
  for (size_t w = 0; w < status.size(); ++w)
    if (status[w] != PICARD_OK) return fail(status[w], message[w].empty() ? "field copy" : message[w]);
  c->stats.d2h_bytes += (int64_t)(sizeof(double) * total);
  return PICARD_OK;
}

int picard_gpu_set_field(picard_ctx* c, int32_t which, const double* in) {
  if (!c || !in) return fail(PICARD_ERR_BAD_ARG, "NULL argument");
  if (which == PICARD_FIELD_F && !c->F) PICARD_TRY(dalloc(c, c->F, (size_t)3 * c->prm.species * c->K.nodes));
  double* dev;
  int ncomp;
  long long n;
  PICARD_TRY(field_geometry(c, which, &dev, &ncomp, &n));
  std::vector<double> h((size_t)ncomp * n);
  for (int pl = 0; pl < ncomp; ++pl)
    for (long long g = 0; g < n; ++g) h[(size_t)pl * n + g] = in[ref_index(which, c->prm.species, pl, g)];
  PICARD_CUDA(cudaMemcpyAsync(dev, h.data(), sizeof(double) * h.size(), cudaMemcpyHostToDevice, c->st));
  c->stats.h2d_bytes += (int64_t)(sizeof(double) * h.size());
  if (which == PICARD_FIELD_D) bcpot_fft_invalidate(c);
  if (which == PICARD_FIELD_E && c->E32) {
    std::vector<float4> e32(n);
    for (long long g = 0; g < n; ++g)
      e32[g] = make_float4(float(h[g]), float(h[n + g]), float(h[2 * n + g]), 0.0f);
    PICARD_CUDA(cudaMemcpyAsync(c->E32, e32.data(), sizeof(float4) * n, cudaMemcpyHostToDevice, c->st));
    PICARD_CUDA(cudaStreamSynchronize(c->st));
  }
  PICARD_CUDA(cudaStreamSynchronize(c->st));
  return PICARD_OK;
}

// ------------------------------------------------ one entry per subroutine

// CalcDistance.f90:1-95
int picard_gpu_calc_distance(picard_ctx* c) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  PICARD_CUDA(launch_calc_distance(c->K, c->D, c->st));
  bcpot_fft_invalidate(c);
  return PICARD_OK;
}

// ParticlesInitialize.f90:2-125
int picard_gpu_particles_initialize(picard_ctx* c) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  long long per_cell = c->inflow.group_prefix[c->prm.species];
  long long total = (long long)c->prm.nx * c->prm.ny * c->prm.nz * per_cell;
  PICARD_TRY(ensure_capacity(c, total));
  if (c->layout == PICARD_LAYOUT_F64)
    PICARD_CUDA(launch_init_f64(c->K, c->f64, c->num_local, c->st));
  else
    PICARD_CUDA(launch_init_c32(c->K, c->c32, c->num_local, c->st));
  c->num_local += total;
  return push_count(c);
}

// BCinflow.f90:2-476
int picard_gpu_bc_inflow(picard_ctx* c, int32_t iteration) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  long long total = c->inflow.cells * c->inflow.per_cell;
  PICARD_TRY(ensure_capacity(c, total));
  if (c->layout == PICARD_LAYOUT_F64)
    PICARD_CUDA(launch_inflow_f64(c->K, c->inflow, iteration, c->f64, c->num_local, c->st));
  else
    PICARD_CUDA(launch_inflow_c32(c->K, c->inflow, iteration, c->c32, c->num_local, c->st));
  c->num_local += total;
  return push_count(c);
}

// AdvancePosition.f90:4-19
int picard_gpu_advance_position(picard_ctx* c, double dt) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  if (c->layout == PICARD_LAYOUT_F64)
    PICARD_CUDA(launch_advance_position_f64(c->K, c->f64, c->num_local, dt, c->st));
  else
    PICARD_CUDA(launch_advance_position_c32(c->K, c->c32, c->num_local, dt, c->st));
  return PICARD_OK;
}

// ParticlesProduce.f90:1-113
int picard_gpu_particles_produce(picard_ctx* c, int32_t iteration) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  if (!has_neutral_source(c->K)) return PICARD_OK;
  const int cells = c->prm.nx * c->prm.ny * c->prm.nz;
  PICARD_CUDA(launch_produce_count(c->K, iteration, c->cell_counts, c->st));
  int* total = c->cell_offsets + cells;
  PICARD_CUDA(launch_scan_int(c->cell_counts, c->cell_offsets, cells, total, c->cell_offsets + cells + 2, c->st));
  PICARD_CUDA(cudaMemcpyAsync(c->h_pinned_i + 3, total, sizeof(int), cudaMemcpyDeviceToHost, c->st));
  PICARD_CUDA(cudaStreamSynchronize(c->st));
  c->stats.d2h_bytes += sizeof(int);
  long long add = c->h_pinned_i[3];
  if (add == 0) return PICARD_OK;
  PICARD_TRY(ensure_capacity(c, add));
  if (c->layout == PICARD_LAYOUT_F64)
    PICARD_CUDA(launch_produce_emit_f64(c->K, iteration, c->cell_offsets, c->f64, c->d_count,
                                        c->capacity, c->d_err, c->st));
  else
    PICARD_CUDA(launch_produce_emit_c32(c->K, iteration, c->cell_offsets, c->c32, c->d_count,
                                        c->capacity, c->d_err, c->st));
  PICARD_TRY(count_issue(c));
  return count_collect(c);
}

// BCoutflow.f90:5-87, in place and in the reference's order (outflow.cuh)
//
// In two stages around a read of the survivor count n' and of m, the survivors of the
// window [n', n): its chains are followed one by one, or resolved by pointer jumping
// (outflow.cuh; scratch of one int per window position, allocated on first use).  The
// jumping launches some ten kernels, which a call that the host waits for pays in
// full: about 100 us up to windows of 2 x 10^5.  The walk takes longer with the window
// and, at equal windows, with the survivors its chains pass.  us of the call, walk and
// jumping: few survivors, W 42 k, m 50 76 / 94; 85 k, 112 91 / 103; 131 k, 30 98 / 97; 209 k,
// 53 155 / 116; 526 k, 138 242 / 145; many, W 16 k, m 400 164 / 98; 55 k, 1,340 190 / 102; 170 k,
// 4,290 186 / 109; 738 k, 18.8 k (the reference's default parameters) 283 / 162.
int picard_gpu_bc_outflow(picard_ctx* c) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  const long long n = c->num_local;
  OutflowSplit sp{1, 0, c->d_info, nullptr};
  PICARD_CUDA(launch_outflow_split(c, n, &sp));
  PICARD_CUDA(cudaMemcpyAsync(c->h_pinned_i + 6, c->d_info, sizeof(int), cudaMemcpyDeviceToHost, c->st));
  PICARD_TRY(sync_count(c));
  c->stats.d2h_bytes += sizeof(int);
  const long long np = c->num_local, window = n - np, m = c->h_pinned_i[6];
  sp.stage = 2;
  sp.np = np;
  if (window >= 4 * m && (window >= (1LL << 17) || (window >= (1LL << 14) && 128 * m >= window))) {
    if (c->jump_cap < window) {
      const long long cap = std::min<long long>(c->capacity, std::max<long long>(window, 2 * c->jump_cap));
      if (c->jump) {
        release(c, c->jump);
        c->jump = nullptr;
        c->jump_cap = 0;
      }
      PICARD_TRY(dalloc(c, c->jump, (size_t)cap));
      c->jump_cap = cap;
    }
    sp.nxt = c->jump;
  }
  PICARD_CUDA(launch_outflow_split(c, n, &sp));
  return check_dev_err(c);
}

// ParticlesTransfer.f90:2-614 (one rank: periodic wrap, ibid. 494-519)
int picard_gpu_particles_transfer(picard_ctx* c) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  if (c->layout == PICARD_LAYOUT_F64)
    PICARD_CUDA(launch_transfer_f64(c->K, c->f64, c->num_local, c->st));
  else
    PICARD_CUDA(launch_transfer_c32(c->K, c->c32, c->num_local, c->st));
  return PICARD_OK;
}

static int deposit(picard_ctx* c, bool with_flux) {
  const long long nn = c->K.nodes;
  const int S = c->prm.species;
  PICARD_CUDA(launch_zero(c->Nacc, (long long)nn * S, c->st));
  unsigned long long* Facc = nullptr;
  if (with_flux) {
    if (!c->Facc) PICARD_TRY(dalloc(c, c->Facc, (size_t)3 * S * nn));
    if (!c->F) PICARD_TRY(dalloc(c, c->F, (size_t)3 * S * nn));
    Facc = c->Facc;
    PICARD_CUDA(cudaMemsetAsync(Facc, 0, sizeof(unsigned long long) * nn * S * 3, c->st));
  }
  if (c->layout == PICARD_LAYOUT_F64)
    PICARD_CUDA(launch_deposit_f64(c->K, c->f64, c->num_local, c->Nacc, Facc, c->st));
  else
    PICARD_CUDA(launch_deposit_c32(c->K, c->c32, c->num_local, c->Nacc, Facc, c->st));
  PICARD_CUDA(launch_finish_deposit(c->K, c->Nacc, c->N, c->C, c->st));
  if (with_flux) PICARD_CUDA(launch_finish_flux(c->K, Facc, c->F, c->st));
  return PICARD_OK;
}

// ParticlesGridify.f90:1-296
int picard_gpu_particles_gridify(picard_ctx* c) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  return deposit(c, false);
}

// ParticlesGridifyAll.f90:1-455
int picard_gpu_particles_gridify_all(picard_ctx* c) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  return deposit(c, true);
}

static int set_option(picard_ctx* c, int32_t option, int32_t value) {
  if (option == PICARD_OPT_BCPOT_TENSOR) {
    if (value < PICARD_BCPOT_DIRECT || value > PICARD_BCPOT_FFT)
      return fail(PICARD_ERR_BAD_ARG, "BCPOT_TENSOR must be 0 (direct), 1 (tensor cores) or 2 (FFT)");
    if (value == PICARD_BCPOT_FFT && !bcpot_fft_supported(c->K))
      return fail(PICARD_ERR_BAD_ARG, "FFT BCpotentials: a face is longer than its shared-memory FFT");
    c->bcpot_tensor = value;
    return PICARD_OK;
  }
  if (option == PICARD_OPT_SWEEP_CTAS) {
    if (value < -1) return fail(PICARD_ERR_BAD_ARG, "SWEEP_CTAS must be -1, 0 or a CTA count");
    if (value == 0) {
      c->G.ctas = -1;  // forget the cached shape of this context
      return tune_sweep(c, true);
    }
    c->G.ctas = value < 0 ? 0 : value;
    return PICARD_OK;
  }
  if (option == PICARD_OPT_SWEEP_PDL) {
    c->G.pdl = value != 0;
    return PICARD_OK;
  }
  if (option == PICARD_OPT_SWEEP_RESIDENT) {
    if (value < 0 || value > kResidentShapes) return fail(PICARD_ERR_BAD_ARG, "SWEEP_RESIDENT must be 0..5");
    return set_resident(c, value);
  }
  if (option == PICARD_OPT_SWEEP_PAIRS) {
    c->G.pairs = value != 0;
    if (!c->G.pairs) c->G.fused2 = 0;
    return PICARD_OK;
  }
  if (option == PICARD_OPT_SWEEP_FUSED) {
    if (value && (!c->G.tma || c->G.zc > 8)) return fail(PICARD_ERR_STATE, "two-sweep launches need the TMA sweep with zc <= 8");
    c->G.fused2 = value != 0;
    if (c->G.fused2) c->G.pairs = 1;
    return PICARD_OK;
  }
  if (option == PICARD_OPT_SWEEP_STAGES) {
    if (value != 1 && value != 2) return fail(PICARD_ERR_BAD_ARG, "SWEEP_STAGES must be 1 or 2");
    c->G.stages = value;
    return PICARD_OK;
  }
  if (option == PICARD_OPT_SWEEP_R_GLOBAL) {
    c->G.rglobal = value != 0;
    if (c->G.rglobal) c->G.pairs = 1, c->G.fused2 = 0;
    return PICARD_OK;
  }
  if (option == PICARD_OPT_SWEEP_CLUSTER) {
    if (value != 0 && value != 1) return fail(PICARD_ERR_BAD_ARG, "SWEEP_CLUSTER must be 0 or 1");
    return set_cluster(c, value);
  }
  if (option == PICARD_OPT_SORT_EVERY) {
    if (value < 0) return fail(PICARD_ERR_BAD_ARG, "SORT_EVERY must be >= 0");
    c->sort_every = value;
    return PICARD_OK;
  }
  if (option == PICARD_OPT_WAIT_TEST) {
    if (value != 0 && value != 1) return fail(PICARD_ERR_BAD_ARG, "WAIT_TEST must be 0 or 1");
    c->wait_test = value;
    return PICARD_OK;
  }
  return fail(PICARD_ERR_BAD_ARG, "unknown option");
}

int picard_gpu_set_option(picard_ctx* c, int32_t option, int32_t value) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  PICARD_TRY(set_option(c, option, value));
  // a sweep shape asked for by hand replaces the cluster that the tuner may have
  // picked (SWEEP_CTAS 0 has just asked the tuner)
  const bool shape = (option >= PICARD_OPT_SWEEP_CTAS && option <= PICARD_OPT_SWEEP_FUSED) ||
                     option == PICARD_OPT_SWEEP_R_GLOBAL;
  if (shape && !(option == PICARD_OPT_SWEEP_CTAS && value == 0)) c->cluster32 = ClusterPlan();
  return PICARD_OK;
}

int picard_gpu_get_option(picard_ctx* c, int32_t option, int32_t* value) {
  if (!c || !value) return fail(PICARD_ERR_BAD_ARG, "NULL argument");
  switch (option) {
    case PICARD_OPT_BCPOT_TENSOR: *value = c->bcpot_tensor; return PICARD_OK;
    case PICARD_OPT_SWEEP_CTAS: *value = c->G.ctas; return PICARD_OK;
    case PICARD_OPT_SWEEP_PDL: *value = c->G.pdl; return PICARD_OK;
    case PICARD_OPT_SWEEP_STAGES: *value = c->G.stages; return PICARD_OK;
    case PICARD_OPT_SWEEP_PAIRS: *value = c->G.pairs; return PICARD_OK;
    case PICARD_OPT_SWEEP_FUSED: *value = c->G.fused2; return PICARD_OK;
    case PICARD_OPT_SWEEP_RESIDENT: *value = resident_option_value(c); return PICARD_OK;
    case PICARD_OPT_WAIT_TEST: *value = c->wait_test; return PICARD_OK;
    case PICARD_OPT_SWEEP_R_GLOBAL: *value = c->G.rglobal; return PICARD_OK;
    case PICARD_OPT_SORT_EVERY: *value = c->sort_every; return PICARD_OK;
    case PICARD_OPT_SWEEP_CLUSTER: *value = c->cluster32.ctas != 0; return PICARD_OK;
  }
  return fail(PICARD_ERR_BAD_ARG, "unknown option");
}

// BCpotentials.f90:1-145
int picard_gpu_bc_potentials(picard_ctx* c) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  PICARD_TRY(bc_potentials_async(c));
  return c->bcpot_tensor == PICARD_BCPOT_TENSOR ? check_dev_err_timeout(c) : PICARD_OK;
}

// CalcEfield.f90:3-232
int picard_gpu_calc_efield(picard_ctx* c) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  PICARD_CUDA(launch_efield(c->K, c->U, c->E, c->E32, c->st));
  return PICARD_OK;
}

// BCfields.f90:3-94: on one rank the open-face ghost layers of E are zero
// already (picard_gpu_calc_efield writes them); this re-zeroes them so the
// routine also holds after picard_gpu_set_field.
int picard_gpu_bc_fields(picard_ctx* c) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  PICARD_CUDA(launch_bc_fields(c->K, c->E, c->E32, c->st));
  return PICARD_OK;
}

static int advance_velocity(picard_ctx* c, double dt, double deltat, int mode) {
  if (!c) return fail(PICARD_ERR_BAD_ARG, "ctx is NULL");
  if (!(dt != 0.0)) return fail(PICARD_ERR_BAD_ARG, "dt must be nonzero");
  if (c->layout == PICARD_LAYOUT_F64)
    PICARD_CUDA(launch_advance_velocity_f64(c->K, c->f64, c->num_local, c->E, dt, deltat, mode, c->st));
  else
    PICARD_CUDA(launch_advance_velocity_c32(c->K, c->c32, c->num_local, c->E32, dt, deltat, mode, c->st));
  return PICARD_OK;
}

// AdvanceVelocity.f90:6-125
int picard_gpu_advance_velocity(picard_ctx* c, double dt) { return advance_velocity(c, dt, 0.0, 0); }
// AdvanceVelocity.f90:128-236
int picard_gpu_advance_velocity_exp(picard_ctx* c, double deltat, double dt) {
  return advance_velocity(c, dt, deltat, 1);
}
// AdvanceVelocity.f90:239-347
int picard_gpu_advance_velocity_imp(picard_ctx* c, double deltat, double dt) {
  return advance_velocity(c, dt, deltat, 2);
}

// picard.f90:651-665
int picard_gpu_energy(picard_ctx* c, double out[3], int32_t* num) {
  if (!c || !out) return fail(PICARD_ERR_BAD_ARG, "NULL argument");
  ReduceBuf rb{c->red_partial, c->red_result, c->red_blocks};
  if (c->layout == PICARD_LAYOUT_F64)
    PICARD_CUDA(launch_energy_particles_f64(c->K, c->f64, c->num_local, rb, c->st));
  else
    PICARD_CUDA(launch_energy_particles_c32(c->K, c->c32, c->num_local, rb, c->st));
  ReduceBuf rf{c->red_partial, c->red_result + 1, c->red_blocks};
  PICARD_CUDA(launch_energy_field(c->K, c->E, rf.partial, rf.result, c->st));
  PICARD_CUDA(cudaMemcpyAsync(c->h_pinned, c->red_result, 2 * sizeof(double), cudaMemcpyDeviceToHost, c->st));
  PICARD_CUDA(cudaStreamSynchronize(c->st));
  c->stats.d2h_bytes += 2 * sizeof(double);
  out[0] = c->h_pinned[0];
  out[1] = c->h_pinned[1];
  // B is uniform (updateBfield is not implemented in the reference)
  double b2 = 0.0;
  for (int c3 = 0; c3 < 3; ++c3) b2 += c->prm.B0[c3] * c->prm.B0[c3];
  double nodes = (double)c->prm.nx * c->prm.ny * c->prm.nz;
  out[2] = nodes * b2 * 0.5 / kMu0 * c->K.dV;
  if (num) *num = int32_t(c->num_local);
  return PICARD_OK;
}

}  // extern "C"
