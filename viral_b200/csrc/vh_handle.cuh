// The handle behind the C ABI and the launch sequence of one TVDRK2 step,
// shared by the translation units that drive the step (the entry points of
// include/vh.h and the discrete adjoint).
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <string>
#include <type_traits>
#include <vector>

#include "vh.h"
#include "vh_aux.cuh"
#include "vh_hostcopy.cuh"
#include "vh_nvtx.h"

using namespace vh;

struct vh_handle {
  vh_config cfg{};
  DevCfg C{};
  cudaStream_t stream = nullptr;
  bool mixed = false;
  size_t esz = 8;            // bytes per state element
  void* state = nullptr;     // 18 canonical fields + B(9) + v1t(4) + res(9) + du(12)
  double* stage = nullptr;   // 18*n doubles: host<->device staging for the mixed path / du16 scratch
  double* eos_d = nullptr;
  float* eos_f = nullptr;
  unsigned int* status = nullptr;
  unsigned long long* iters = nullptr;
  unsigned long long* red = nullptr;  // reduction slots
  double* part = nullptr;              // conservation partial sums
  int part_blocks = 0;
  DevPtrs<double> pd{};
  DevPtrs<float> pf{};
  std::vector<double> eos_host;  // 4 x eos_n
  double tau = 0;
  bool have_state = false;
  // step kernels launched with programmatic dependent launch (VH_PDL=0 in
  // the environment at vh_create turns it off, e.g. under a profiler that
  // replays kernels one by one)
  bool pdl = true;
  SweepPlan plan{};         // the flux sweeps' tiles
  TileMaps tmap;            // tensor maps of the state for their TMA staging
  bool tma = false;         // the maps were made (else the sweeps load through the cache)
  bool tma_wanted = true;  // VH_TMA=0 in the environment at vh_create: cached loads
  // discrete-adjoint workspace (kept between calls) and the device
  // milliseconds of the last call's phases
  void* adj_buf = nullptr;
  size_t adj_bytes = 0;
  double adj_ms[4] = {0, 0, 0, 0};
  // the slice vh_freezeout_step saw last: T and u^mu (5 x n doubles) at
  // fo_tau; forgotten whenever the state is set from outside
  double* fo_prev = nullptr;
  double fo_tau = 0;
  bool fo_have = false;
  // canonical-layout transfer buffer between host arrays and the padded
  // device arrays (allocated on first use)
  double* xfer = nullptr;
  size_t xfer_bytes = 0;
  HostCopy to_host;  // large results into pageable memory
  std::string err;
};

#define VH_CUDA(h, call)                                                                        \
  do {                                                                                          \
    cudaError_t _e = (call);                                                                    \
    if (_e != cudaSuccess) {                                                                    \
      (h)->err = std::string(#call) + ": " + cudaGetErrorString(_e);                            \
      return VH_E_CUDA;                                                                         \
    }                                                                                           \
  } while (0)

static inline int fail(vh_handle* h, int code, const std::string& msg) {
  if (h) h->err = msg;
  return code;
}

template <class R>
static void set_ptrs(DevPtrs<R>& P, void* base, void* res1, long long n, unsigned int* status,
                     unsigned long long* iters) {
  P.base0 = static_cast<R*>(base);
  P.base1 = static_cast<R*>(base) + 18 * n;
  P.stride = n;
  P.res1 = static_cast<R*>(res1);
  P.status = status;
  P.iters = iters;
}
static constexpr int kStateArrays = 52;

static inline unsigned grid1(long long n, int b) { return (unsigned)((n + b - 1) / b); }

template <class R>
static auto sweep_kernel(const vh_handle* h, bool tma) {
  const bool mm = h->C.recon != 0;
  return tma ? (mm ? k_dir<R, true, true> : k_dir<R, false, true>) : (mm ? k_dir<R, true, false> : k_dir<R, false, false>);
}

// The flux sweeps of a stage along directions d0..d1-1, one launch.
template <class R>
static int launch_dirs(vh_handle* h, const DevPtrs<R>& P, int d0, int d1, int use_b, double tau) {
  const DevCfg& C = h->C;
  const SweepPlan& p = h->plan;
  int first = 0, n = 0;
  for (int d = 0; d < d1; d++) (d < d0 ? first : n) += p.blocks(d);
  // one divergence array for all directions (P.res1 null): the cached kernels
  // (a plan's tile stays below the 48 KB that need no attribute)
  auto kern = sweep_kernel<R>(h, h->tma && P.res1);
  VH_CUDA(h, launch_step_kernel(h->pdl, kern, dim3(n), dim3(kSweepThreads), sweep_smem<R>(p, C.bi ? 2 : 3), h->stream,
                                C, P, use_b, (R)tau, p, first, h->tmap));
  return VH_OK;
}

// The tensor maps of the state: a 4D tensor (x over the padded row pitch,
// y, z, array) of the 52 arrays, one box shape per sweep direction and
// array count (SweepLay).  cuTensorMapEncodeTiled comes from the driver
// through the runtime's entry-point query.
template <class R, int DIR>
static int encode_dir_maps(vh_handle* h, PFN_cuTensorMapEncodeTiled_v12000 enc) {
  const DevCfg& C = h->C;
  const SweepLay<R, DIR> L(h->plan.n[DIR]);
  const cuuint64_t dims[4] = {(cuuint64_t)C.px, (cuuint64_t)C.gy, (cuuint64_t)C.gz, (cuuint64_t)kStateArrays};
  const cuuint64_t strides[3] = {(cuuint64_t)C.px * sizeof(R), (cuuint64_t)C.px * C.gy * sizeof(R),
                                 (cuuint64_t)C.n * sizeof(R)};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  for (int q = 0; q < 2; q++) {
    const cuuint32_t box[4] = {(cuuint32_t)(DIR == 0 ? L.ld : kSweepLines),
                               (cuuint32_t)(DIR == 0 ? kSweepLines : DIR == 1 ? L.na : 1),
                               (cuuint32_t)(DIR == 2 ? L.na : 1), q ? 9u : 5u};
    const CUresult r = enc(&h->tmap.m[DIR][q], sizeof(R) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64,
                           4, h->state, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return VH_E_CUDA;
  }
  return VH_OK;
}

// Sets h->tma when every map of the grid's directions was made; a grid the
// encoder refuses (none is known) steps with the sweeps loading through the
// cache instead, the same arithmetic.
template <class R>
static void encode_maps(vh_handle* h) {
  h->tma = false;
  if (!h->tma_wanted) return;
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn ||
      q != cudaDriverEntryPointSuccess) {
    cudaGetLastError();
    return;
  }
  auto enc = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  if (encode_dir_maps<R, 0>(h, enc) || encode_dir_maps<R, 1>(h, enc)) return;
  if (!h->C.bi && encode_dir_maps<R, 2>(h, enc)) return;
  h->tma = true;
}

template <class R>
static int set_smem_attrs(vh_handle* h) {
  h->plan = sweep_plan<R>(h->C);
  encode_maps<R>(h);
  // for the kernel the steps will launch alone: this loads it
  VH_CUDA(h, set_sweep_smem(sweep_kernel<R>(h, h->tma)));
  return VH_OK;
}

// the flux-divergence part of a stage: every direction into its divergence
// and du, in one launch
template <class R>
static int stage_rhs(vh_handle* h, const DevPtrs<R>& P, int use_b, double tau) {
  const int dirs = h->C.bi ? 2 : 3;
  if (P.res1) return launch_dirs<R>(h, P, 0, dirs, use_b, tau);
  for (int d = 0; d < dirs; d++)
    if (int r = launch_dirs<R>(h, P, d, d + 1, use_b, tau)) return r;
  return VH_OK;
}

// the update part of a stage (sources, RK, root-find, ghosts): k_update,
// one thread per interior cell
template <class R, int STAGE>
static int stage_update(vh_handle* h, const DevPtrs<R>& P, double tau, double ts) {
  const DevCfg& C = h->C;
  const long long nint = (long long)C.nx * C.ny * (C.kr - C.kl);
  VH_CUDA(h, launch_step_kernel(h->pdl, k_update<R, STAGE>, dim3(grid1(nint, kUpdThreads)), dim3(kUpdThreads), 0, h->stream, C, P,
                                tau, ts));
  return VH_OK;
}

template <class R>
static int step_once(vh_handle* h, const DevPtrs<R>& P) {
  VhNvtxRange range("TVDRK2 step");
  const double tau = h->tau, ts = h->cfg.dtau;
  int r;
  if ((r = stage_rhs<R>(h, P, 0, tau))) return r;
  if ((r = stage_update<R, 1>(h, P, tau, ts))) return r;
  if ((r = stage_rhs<R>(h, P, 1, tau + ts))) return r;
  if ((r = stage_update<R, 2>(h, P, tau, ts))) return r;
  h->tau = tau + ts;
  return VH_OK;
}


// Arrays of the C ABI (host or device memory) hold nfields fields of
// gx*gy*gz cells each, rows of gx cells; the handle's device arrays hold
// rows of px cells.  When the two differ, a kernel moves the rows between
// the layouts on the device: from (to) the caller's array itself when it is
// device memory, else through one contiguous copy to (from) the handle's
// transfer buffer, so that host data crosses the bus in a single copy.
static inline long long canon_cells(const DevCfg& C) { return (long long)C.gx * C.gy * C.gz; }

// Rows of gx canonical doubles <-> rows of px elements R of the handle's
// arrays, converted on the way: field blockIdx.y, four cells a thread (their
// loads in flight together), the row from a 32-bit division.  Bound by DRAM.
// Against an element a thread with 64-bit divisions, and in the mixed mode a
// conversion pass of its own, a state set and read back (161x161x41, 18
// fields) takes 0.09 ms less in FP64 (0.20 before) and 0.25 ms less in the
// mixed mode (0.059 ms a direction now).
template <class R, bool IN>
static __global__ void __launch_bounds__(256) k_repitch(std::conditional_t<IN, const double, double>* canon,
                                                         std::conditional_t<IN, R, const R>* dev, unsigned nc,
                                                         long long n, unsigned gx, unsigned px) {
  canon += (long long)blockIdx.y * nc;
  dev += (long long)blockIdx.y * n;
  const unsigned t0 = blockIdx.x * 1024 + threadIdx.x;
  R v[4];
  unsigned at[4];
#pragma unroll
  for (int m = 0; m < 4; m++) {
    const unsigned t = t0 + m * 256, row = t / gx;
    at[m] = row * px + (t - row * gx);
    if (t < nc) v[m] = IN ? (R)canon[t] : (R)dev[at[m]];
  }
#pragma unroll
  for (int m = 0; m < 4; m++) {
    const unsigned t = t0 + m * 256;
    if (t >= nc) continue;
    if constexpr (IN) dev[at[m]] = v[m];
    else canon[t] = (double)v[m];
  }
}

static inline bool device_accessible(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

// the transfer buffer, nfields canonical fields (allocated on first use)
// (in the mixed mode the staging buffer, which a float array's transfer does
// not use otherwise)
static int xfer_buffer(vh_handle* h, int nfields, bool staging, double** out) {
  if (staging) {
    *out = h->stage;
    return VH_OK;
  }
  const size_t need = sizeof(double) * (size_t)nfields * (size_t)canon_cells(h->C);
  if (h->xfer_bytes < need) {
    VH_CUDA(h, cudaStreamSynchronize(h->stream));
    cudaFree(h->xfer);
    h->xfer = nullptr;
    h->xfer_bytes = 0;
    VH_CUDA(h, cudaMalloc(&h->xfer, need));
    h->xfer_bytes = need;
  }
  *out = h->xfer;
  return VH_OK;
}

// canonical doubles (host or device) into a handle's array, and back
template <class R>
static int pitched_in(vh_handle* h, R* dev_padded, const double* canon, int nfields) {
  const DevCfg& C = h->C;
  const long long nc = canon_cells(C), total = nfields * nc;
  if (sizeof(R) == 8 && C.px == C.gx) {
    VH_CUDA(h, cudaMemcpyAsync(dev_padded, canon, sizeof(double) * total, cudaMemcpyDefault, h->stream));
    return VH_OK;
  }
  const double* src = canon;
  if (!device_accessible(canon)) {
    double* x = nullptr;
    if (int r = xfer_buffer(h, nfields, sizeof(R) == 4, &x)) return r;
    VH_CUDA(h, cudaMemcpyAsync(x, canon, sizeof(double) * total, cudaMemcpyHostToDevice, h->stream));
    src = x;
  }
  k_repitch<R, true><<<dim3(grid1(nc, 1024), nfields), 256, 0, h->stream>>>(src, dev_padded, (unsigned)nc, C.n,
                                                                            (unsigned)C.gx, (unsigned)C.px);
  VH_CUDA(h, cudaGetLastError());
  return VH_OK;
}
template <class R>
static int pitched_out(vh_handle* h, double* canon, const R* dev_padded, int nfields) {
  const DevCfg& C = h->C;
  const long long nc = canon_cells(C), total = nfields * nc;
  if (sizeof(R) == 8 && C.px == C.gx) {
    VH_CUDA(h, h->to_host.copy(canon, dev_padded, sizeof(double) * total, h->stream));
    return VH_OK;
  }
  const bool dev = device_accessible(canon);
  double* x = canon;
  if (!dev)
    if (int r = xfer_buffer(h, nfields, sizeof(R) == 4, &x)) return r;
  k_repitch<R, false><<<dim3(grid1(nc, 1024), nfields), 256, 0, h->stream>>>(x, dev_padded, (unsigned)nc, C.n,
                                                                             (unsigned)C.gx, (unsigned)C.px);
  VH_CUDA(h, cudaGetLastError());
  if (!dev) VH_CUDA(h, h->to_host.copy(canon, x, sizeof(double) * total, h->stream));
  return VH_OK;
}

static inline int read_status(vh_handle* h) {
  unsigned int st = 0;
  VH_CUDA(h, cudaMemcpyAsync(&st, h->status, sizeof(st), cudaMemcpyDeviceToHost, h->stream));
  VH_CUDA(h, cudaStreamSynchronize(h->stream));
  if (st & ST_ROOT) return fail(h, VH_E_ROOTFIND, "root-find failed in at least one cell");
  if (st & ST_NEGE) return fail(h, VH_E_NEG_ENERGY, "non-positive energy density after the root-find");
  if (st & ST_CAUSAL) return fail(h, VH_E_CAUSALITY, "superluminal velocity after the root-find");
  if (st & ST_TMA) return fail(h, VH_E_CUDA, "a flux-sweep tile copy (TMA) did not complete");
  return VH_OK;
}
