// Kernels of one RK stage of the viscous KT step and its helpers.
//
// A stage is two launches:
//   k_dir       the flux sweeps of every direction (vh_sweep.cuh), each
//               direction's flux differences into its own set of nine
//               arrays, so that the directions need no order among them
//               (NEWEST5/hydroKT.h:16-491, NEWEST5/Source.h:3-101).
//   k_update    one thread per interior cell: the sum of the directions'
//               flux differences, sources, RK2 combination,
//               FP64 root-find, and the ghost copy of boundary cells
//               (NEWEST5/Source.h:165-433, time.h:1-387, multiroot.h:331-493,
//               boundary.h:1-276).
#pragma once

#include "vh_sweep.cuh"

namespace vh {

// Programmatic dependent launch: the step's kernels are launched so that the
// next one may start while this one's last blocks still run.  Every block
// first waits until the previous kernel in the stream has completed and its
// writes are visible (a no-op under an ordinary launch), then lets the next
// kernel be launched.
__device__ __forceinline__ void pdl_wait_then_release() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// A step kernel launched with programmatic stream serialization (when pdl):
// it may begin while the kernel before it in the stream finishes its last
// blocks; the kernel itself waits for that kernel's completion before
// reading anything (pdl_wait_then_release), so the overlap covers launch and
// block set-up.
template <class K, class... Args>
static cudaError_t launch_step_kernel(bool pdl, K kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                      Args... args) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = grid;
  lc.blockDim = block;
  lc.dynamicSmemBytes = smem;
  lc.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = at;
  lc.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&lc, kernel, args...);
}

// The tensor maps of the state: per direction, arrays 0..4 (e, u^mu) and one
// conserved set (9 arrays); used by the TMA-staged sweeps alone.
struct alignas(64) TileMaps {
  CUtensorMap m[3][2];
};

// Blocks of 96 threads per SM the sweeps are compiled for: 5 in FP64 (124
// registers; at 6 blocks and 96 registers, with spills, the 161x161x41 step
// takes 7 % longer), 9 in FP32 (72).
template <class R>
struct DirOcc {
  static constexpr int MIN_BLOCKS = sizeof(R) == 8 ? 5 : 9;
};

// The sweeps of a stage: blocks first_block.. of the plan, which runs
// through the directions' tiles one after the other (a launch of one
// direction's blocks alone is that direction's sweep).  With a divergence set
// per direction the directions need no order, so a stage is one launch: no
// drained tail between directions, and half the launches of a small grid's
// step.  Adding up one set instead, a launch per direction in order, costs
// the sweeps more than the update saves (161x161x41 FP64 step 1.57 ms against
// 1.31, boost-invariant 129x129 0.083 against 0.058).  TMA: the tiles are
// staged by box copies from the handle's padded state, else by loads through
// the cache (the same arithmetic).
template <class R, bool MM, bool TMA>
__global__ void __launch_bounds__(kSweepThreads, DirOcc<R>::MIN_BLOCKS)
    k_dir(const __grid_constant__ DevCfg C, const __grid_constant__ DevPtrs<R> P, int use_b, R tau,
          const __grid_constant__ SweepPlan plan, int first_block, const __grid_constant__ TileMaps maps) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  R* sm = reinterpret_cast<R*>(smem_raw);
  pdl_wait_then_release();
  if (*P.status) return;
  int b = blockIdx.x + first_block, d = 0;
  while (d < 2 && b >= plan.blocks(d)) b -= plan.blocks(d++);
  const int bx = b % plan.along[d], r = b / plan.along[d], by = r % plan.across[d], bz = r / plan.across[d];
  if (d == 0)
    sweep_tile<R, 0, MM, TMA>(C, P, use_b, tau, (R)(1.0 / C.dx), plan.n[0], bx, by, bz, sm, &maps.m[0][0], &maps.m[0][1]);
  else if (d == 1)
    sweep_tile<R, 1, MM, TMA>(C, P, use_b, tau, (R)(1.0 / C.dy), plan.n[1], bx, by, bz, sm, &maps.m[1][0], &maps.m[1][1]);
  else
    sweep_tile<R, 2, MM, TMA>(C, P, use_b, tau, (R)(1.0 / C.dz), plan.n[2], bx, by, bz, sm, &maps.m[2][0], &maps.m[2][1]);
}

// Shared memory a sweep kernel may be launched with: the longest tile's, the
// same for every grid, since the attribute belongs to the function and not to
// a handle.
template <class K>
static cudaError_t set_sweep_smem(K kernel) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)(SweepLay<double, 0>(kSweepMaxN).size * sizeof(double)));
}

// Copy one cell's fields into a ghost cell (NEWEST5/boundary.h).
template <class R>
__device__ inline void ghost_put(const DevPtrs<R>& P, int set_b, long long dst, R e, const R* u, const R* pu,
                                 const R* q9, bool skip_u12) {
  P.e()[dst] = e;
  P.u(0)[dst] = u[0];
  if (!skip_u12) { P.u(1)[dst] = u[1]; P.u(2)[dst] = u[2]; }
  P.u(3)[dst] = u[3];
#pragma unroll
  for (int l = 0; l < 4; l++) P.pu(l)[dst] = pu[l];
#pragma unroll
  for (int l = 0; l < 9; l++) P.S(set_b, l)[dst] = q9[l];
}

// The update of one interior cell, in two parts: rk_cell (du_tau, sources,
// the RK combination, prevu) and root_cell (the root-find and the ghost
// copy).  STAGE 1 reads set A and writes set B and v1t; STAGE 2 reads A (its
// own cell), B and v1t and writes A.
struct CellAt {
  int i, j, k;
  long long c;
};
__device__ __forceinline__ CellAt cell_at(const DevCfg& C, long long t) {
  // 32-bit division: a handle's arrays would not fit the GPU at 2^31 cells
  const unsigned row = (unsigned)t / (unsigned)C.nx, k = row / (unsigned)C.ny;
  CellAt x;
  x.i = C.il + (int)((unsigned)t - row * (unsigned)C.nx);
  x.j = C.jl + (int)(row - k * (unsigned)C.ny);
  x.k = C.kl + (int)k;
  x.c = cix(C, x.i, x.j, x.k);
  return x;
}

// What the RK combination reads besides the sources' inputs (the flux
// divergence of every direction; at stage 2 also set A and v1t) is copied
// into shared memory at the start, asynchronously and without registers, and
// read after the sources: the copies' latency, of memory mostly, hides behind
// the sources' arithmetic.  Slot q of a thread is at pre[q * blockDim.x].
constexpr int kPreSlots = 40;  // 27 divergences, 9 of set A, 4 of v1t
template <class R>
__device__ __forceinline__ void cp_async(R* dst, const R* src) {
  if constexpr (sizeof(R) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// Sources and RK combination of cell x: stores the new conserved set (q9,
// also returned) and, at stage 1, v1t and prevu; returns e, u and prevu for
// the root-find.  pre: the thread's slots, spaced by ps.
template <class R, int STAGE>
__device__ __forceinline__ void rk_cell(const DevCfg& C, const DevPtrs<R>& P, double tau_n, double ts, const CellAt& x,
                                        R& e_out, R* u_out, R* pu_out, R* q9, R* pre, int ps) {
  {
    const int k = x.k;
    const long long c = x.c;
    const int nd = P.res1 ? (C.bi ? 2 : 3) : 1;  // sets of flux divergences
    for (int d = 0; d < nd; d++) {
      const R* r = P.resd(d) + c;
#pragma unroll
      for (int l = 0; l < 9; l++) cp_async<R>(pre + (d * 9 + l) * ps, r + (long long)l * P.stride);
    }
    R* const preA = pre + nd * 9 * ps;
    if (STAGE == 2) {
#pragma unroll
      for (int l = 0; l < 9; l++) cp_async<R>(preA + l * ps, P.A(l) + c);
#pragma unroll
      for (int l = 0; l < 4; l++) cp_async<R>(preA + (9 + l) * ps, P.v1t(l) + c);
    }
    auto div = [&](int l) {
      R v = pre[l * ps];
      for (int d = 1; d < nd; d++) v += pre[(d * 9 + l) * ps];
      return v;
    };
    const double tau1 = tau_n + ts;
    const R tau_s = (R)(STAGE == 1 ? tau_n : tau1);  // time of the sources
    const bool cart = C.cart;

    R u[4], pu[4], p[5], e = P.e()[c];
#pragma unroll
    for (int l = 0; l < 4; l++) { u[l] = P.u(l)[c]; pu[l] = P.pu(l)[c]; }
    const int cur_b = STAGE == 1 ? 0 : 1;  // conserved set read
    R Tc[4];
#pragma unroll
    for (int l = 0; l < 4; l++) Tc[l] = P.S(cur_b, l)[c];
#pragma unroll
    for (int l = 0; l < 5; l++) p[l] = P.S(cur_b, 4 + l)[c];

    // velocity gradients
    R du[4][4];
#pragma unroll
    for (int l = 0; l < 4; l++) {
      du[l][0] = (u[l] - pu[l]) * (R)(1.0 / ts);
      du[l][1] = P.du(l * 3 + 0)[c];
      du[l][2] = P.du(l * 3 + 1)[c];
      du[l][3] = C.bi ? (R)0 : P.du(l * 3 + 2)[c];
    }
    // sources (NEWEST5/Source.h:165-191 geometric, 311-433 shear)
    R src[9];
    {
      R Pp, cs2, Te;
      eos_all<R>(C, e, Pp, cs2, Te);
      if (cart) {
        src[0] = src[1] = src[2] = src[3] = 0;
      } else {
        const R t2 = tau_s * tau_s;
        PiDep<R> d = pi_dep<R>(u[0], u[1], u[2], u[3], p, t2);
        const R ep = e + Pp;
        src[0] = -Pp - t2 * (d.ee + ep * u[3] * u[3]);
        src[1] = 0;
        src[2] = 0;
        src[3] = -(R)2 * (d.te + ep * u[0] * u[3]);
      }
      R s5[5];
      is_source_PT<R>(C, tau_s, e, Pp, Te, u, p, du, s5);
      // TXYZ5/Source.h:268-270: the Cartesian 3+1D shear source skips the
      // last three interior z layers
      if (cart && !C.bi && (k - C.kl) >= C.nz - NG) s5[0] = s5[1] = s5[2] = s5[3] = s5[4] = 0;
#pragma unroll
      for (int q = 0; q < 5; q++) src[4 + q] = s5[q];
    }
    // RK combination (NEWEST5/time.h:2-140)
    asm volatile("cp.async.wait_all;" ::: "memory");  // the thread's own copies
    R Vn[9];
    const int out_b = STAGE == 1 ? 1 : 0;  // conserved set written
    if (STAGE == 1) {
#pragma unroll
      for (int l = 0; l < 9; l++) {
        const R L0 = div(l) + src[l];
        const R v0 = l < 4 ? (cart ? Tc[l] : (R)tau_n * Tc[l]) : p[l - 4];
        Vn[l] = v0 + (R)ts * L0;
      }
#pragma unroll
      for (int l = 0; l < 4; l++) P.v1t(l)[c] = Vn[l];
    } else {
#pragma unroll
      for (int l = 0; l < 9; l++) {
        const R L1 = div(l) + src[l], va = preA[l * ps];
        const R v0 = l < 4 && !cart ? (R)tau_n * va : va;
        const R v1 = l < 4 ? preA[(9 + l) * ps] : p[l - 4];
        Vn[l] = (R)0.5 * v0 + (R)0.5 * v1 + (R)0.5 * (R)ts * L1;
      }
    }
#pragma unroll
    for (int l = 0; l < 4; l++) q9[l] = cart ? Vn[l] : Vn[l] * (R)(1.0 / tau1);
#pragma unroll
    for (int l = 0; l < 5; l++) q9[4 + l] = Vn[4 + l];
#pragma unroll
    for (int l = 0; l < 9; l++) P.S(out_b, l)[c] = q9[l];
    // the root-find's first start: e scaled by the change of T^{tau tau}
    // and, at stage 1, the velocity extrapolated linearly from prevu (the
    // root is the same; root_cell falls back to the stage's primitives)
    const R rt = q9[0] / Tc[0];
    e_out = (rt > (R)0.5 && rt < (R)2) ? e * rt : e;
    u_out[0] = u[0];
#pragma unroll
    for (int l = 1; l < 4; l++) u_out[l] = STAGE == 1 ? (R)2 * u[l] - pu[l] : u[l];
    // previous velocity (NEWEST5/time.h:166, stage 1 only)
    if (STAGE == 1) {
#pragma unroll
      for (int l = 0; l < 4; l++) { pu[l] = u[l]; P.pu(l)[c] = u[l]; }
    }
#pragma unroll
    for (int l = 0; l < 4; l++) pu_out[l] = pu[l];
  }
}

// Root-find (FP64) of cell x from its new conserved set q9 with (e, u) as the
// guess, then the ghost copy; returns the Newton iterations and, at stage 2,
// the new temperature in GeV in *t_gev.
template <class R, int STAGE>
__device__ __forceinline__ unsigned root_cell(const DevCfg& C, const DevPtrs<R>& P, double tau_n, double ts,
                                              const CellAt& at, R e, R* u, const R* pu, const R* q9, double* t_gev) {
  unsigned my_it = 0;
  {
    const int i = at.i, j = at.j, k = at.k;
    const long long c = at.c;
    const double tau1 = tau_n + ts;
    const bool cart = C.cart;
    const int out_b = STAGE == 1 ? 1 : 0;  // conserved set written
    // root-find (FP64) with the current primitives as the guess
    double Tt[4], pd[5], x[4] = {(double)e, (double)u[1], (double)u[2], (double)u[3]};
#pragma unroll
    for (int l = 0; l < 4; l++) Tt[l] = (double)q9[l];
#pragma unroll
    for (int l = 0; l < 5; l++) pd[l] = (double)q9[4 + l];
    // stopping (con2prim): FP64 steps below 1e-13, or an undamped one below
    // 1e-8, taken without the confirming evaluation; the mixed mode stores
    // the result in FP32, so a Newton step below 3e-4 ends it (the error it
    // leaves, of the order of its square, is below FP32 rounding)
    const double rtol = sizeof(R) == 4 ? 1e-10 : 1e-13, qtol = sizeof(R) == 4 ? 1e-6 : 1e-8;
    const double qskip = sizeof(R) == 4 ? 3e-4 : 1e-8, fskip = sizeof(R) == 4 ? 3e-3 : 1e-6;
    int it = -1;
    // a second attempt starts from the stage's primitives, still in memory
    // (near-vacuum cells, where the extrapolated start can lead Newton
    // astray); one loop keeps a single copy of the solver in the kernel
#pragma unroll 1
    for (int attempt = 0; attempt < 2 && it < 0; attempt++) {
      if (attempt) {
        x[0] = (double)P.e()[c];
#pragma unroll
        for (int l = 1; l < 4; l++) x[l] = (double)P.u(l)[c];
      }
      it = con2prim(C, Tt, pd, tau1, x, rtol, qtol, qskip, fskip);
    }
    if (it < 0) {
      atomicOr(P.status, ST_ROOT);
    } else {
      my_it = (unsigned)it;
      const double tt = cart ? 1.0 : tau1;
      const double u0 = sqrt(1 + x[1] * x[1] + x[2] * x[2] + x[3] * x[3] * tt * tt);
      const double vx = x[1] / u0, vy = x[2] / u0, ve = x[3] / u0;
      if (sqrt(vx * vx + vy * vy + tt * tt * ve * ve) >= 1) atomicOr(P.status, ST_CAUSAL);
      if (x[0] <= 0) atomicOr(P.status, ST_NEGE);
      e = (R)x[0];
      u[0] = (R)u0; u[1] = (R)x[1]; u[2] = (R)x[2]; u[3] = (R)x[3];
      P.e()[c] = e;
#pragma unroll
      for (int l = 0; l < 4; l++) P.u(l)[c] = u[l];
    }
    // ghost copy of boundary cells: faces only, corners untouched
    // (NEWEST5/boundary.h:1-276); Gubser test mirrors u^x,u^y.  A boundary
    // cell reads back the conserved set and prevu it stored above, so that
    // they need not stay in registers through the root-find.
    const bool mir = C.mirror;
    const bool edge = i == C.il || i == C.ir - 1 || j == C.jl || j == C.jr - 1 || (!C.bi && (k == C.kl || k == C.kr - 1));
    const bool near = mir && (i - C.il < NG || C.ir - 1 - i < NG || j - C.jl < NG || C.jr - 1 - j < NG);
    if (!edge && !near) {
      if (STAGE == 2 && t_gev) *t_gev = C.hbarc * (double)eos_T<R>(C, e);
      return my_it;
    }
    R qb[9], pb[4];
    if (edge) {
#pragma unroll
      for (int l = 0; l < 9; l++) qb[l] = P.S(out_b, l)[c];
#pragma unroll
      for (int l = 0; l < 4; l++) pb[l] = P.pu(l)[c];
    }
    q9 = qb;
    pu = pb;
    if (i == C.il)
      for (int m = 0; m < NG; m++) ghost_put<R>(P, out_b, cix(C, m, j, k), e, u, pu, q9, mir);
    if (i == C.ir - 1)
      for (int m = 0; m < NG; m++) ghost_put<R>(P, out_b, cix(C, C.ir + m, j, k), e, u, pu, q9, mir);
    if (j == C.jl)
      for (int m = 0; m < NG; m++) ghost_put<R>(P, out_b, cix(C, i, m, k), e, u, pu, q9, mir);
    if (j == C.jr - 1)
      for (int m = 0; m < NG; m++) ghost_put<R>(P, out_b, cix(C, i, C.jr + m, k), e, u, pu, q9, mir);
    if (!C.bi) {
      if (k == C.kl)
        for (int m = 0; m < NG; m++) ghost_put<R>(P, out_b, cix(C, i, j, m), e, u, pu, q9, false);
      if (k == C.kr - 1)
        for (int m = 0; m < NG; m++) ghost_put<R>(P, out_b, cix(C, i, j, C.kr + m), e, u, pu, q9, false);
    }
    if (mir) {
      // ghost m <- cell il + 2 - m on the left, ghost ir + m <- ir - 1 - m on the right
      const int dl = i - C.il, dr = C.ir - 1 - i;
      if (dl < NG) { long long g = cix(C, C.il - 1 - dl, j, k); P.u(1)[g] = u[1]; P.u(2)[g] = u[2]; }
      if (dr < NG) { long long g = cix(C, C.ir + dr, j, k); P.u(1)[g] = u[1]; P.u(2)[g] = u[2]; }
      const int el = j - C.jl, er = C.jr - 1 - j;
      if (el < NG) { long long g = cix(C, i, C.jl - 1 - el, k); P.u(1)[g] = u[1]; P.u(2)[g] = u[2]; }
      if (er < NG) { long long g = cix(C, i, C.jr + er, k); P.u(1)[g] = u[1]; P.u(2)[g] = u[2]; }
    }
    if (STAGE == 2 && t_gev) *t_gev = C.hbarc * (double)eos_T<R>(C, e);
  }
  return my_it;
}

// One interior cell t (0 <= t < nx*ny*nz) of the update, both parts.
template <class R, int STAGE>
__device__ __forceinline__ unsigned update_cell(const DevCfg& C, const DevPtrs<R>& P, double tau_n, double ts,
                                                long long t, double* t_gev, R* pre, int ps) {
  const CellAt x = cell_at(C, t);
  R e, u[4], pu[4], q9[9];
  rk_cell<R, STAGE>(C, P, tau_n, ts, x, e, u, pu, q9, pre, ps);
  return root_cell<R, STAGE>(C, P, tau_n, ts, x, e, u, pu, q9, t_gev);
}

// One thread per interior cell.  Bound by the latency of its loads and of the
// Newton chain, with DRAM at half its rate (79 words a cell at
// stage 1 and 84 at stage 2 in 3+1D).  Blocks per SM: FP64 4 (128 registers), mixed 5 (96); measured on the
// 161x161x41 event, ms per stage-1 launch: FP64 0.220 / 0.213 / 0.305 at 3 / 4 /
// 5 blocks (spills), mixed 0.155 / 0.146 / 0.145 at 4 / 5 / 6.  Divisions and
// roots by the hardware's seeds and one step (rcp, root_rsqrt), elimination
// without row exchanges and the asynchronous prefetch brought it from 0.273 /
// 0.193 (and 0.211 / 0.138 before the directions had a divergence set each).
constexpr int kUpdThreads = 128;
template <class R>
struct UpdOcc {
  static constexpr int MIN_BLOCKS = sizeof(R) == 8 ? 4 : 5;
};
template <class R, int STAGE>
__global__ void __launch_bounds__(kUpdThreads, UpdOcc<R>::MIN_BLOCKS) k_update(const __grid_constant__ DevCfg C, const __grid_constant__ DevPtrs<R> P, double tau_n,
                                                                                        double ts) {
  pdl_wait_then_release();
  if (*P.status) return;
  const long long nint = (long long)C.nx * C.ny * (C.kr - C.kl);
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  __shared__ R pre[kPreSlots * kUpdThreads];
  unsigned long long my_it =
      t < nint ? update_cell<R, STAGE>(C, P, tau_n, ts, t, nullptr, pre + threadIdx.x, kUpdThreads) : 0u;
  // one atomic per warp for the iteration counter
  for (int o = 16; o > 0; o >>= 1) my_it += __shfl_down_sync(0xffffffffu, my_it, o);
  if ((threadIdx.x & 31) == 0 && my_it) atomicAdd(P.iters, my_it);
}

}  // namespace vh
