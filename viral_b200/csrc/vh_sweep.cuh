// The flux sweep along one direction: KT flux divergence of the nine evolved
// quantities and the WENO velocity derivative, tile by tile
// (NEWEST5/hydroKT.h:16-491, NEWEST5/Source.h:3-101).
//
// A tile is 8 lines of N cells along the direction, with 3 more cells at
// either end, in shared memory.  96 threads share it as 8 lines x 12 tasks:
// tasks 0..8 own a conserved quantity each (its flux F^l and its variable
// V^l), tasks 9 and 10 two components of u^mu each.  A thread walks along its
// line cell by cell and keeps the stencil in registers, so that every
// difference, smoothness term and face correction of a line is formed once;
// a lane per cell would form the stencil's differences three to five times
// over or pass them by shuffle, and waste 6 of 32 lanes on the halo.
//
// Bound: latency and FP64 (FMA in FP32) issue, about half of the FP64 pipe's
// cycles used at 3 to 4 warps per scheduler; DRAM at a third of its rate.  On
// the 161x161x41 event the three sweeps of a stage take 0.43 ms in FP64 and
// 0.23 ms in FP32 launched one by one, where a lane per cell (five stencil
// values and shuffles) took 0.61 and 0.35.  One quantity per thread instead
// of two (twice the warps at half the registers) was measured 15 % slower:
// twice the address, loop and shuffle instructions per FP64 instruction.
#pragma once

#include <cuda.h>

#include "vh_device.cuh"

namespace vh {

constexpr int kSweepLines = 8;     // lines of a tile
constexpr int kSweepThreads = 96;  // 8 lines x 12 tasks (11 used)
constexpr int kSweepMaxN = 58;     // longest tile a plan may hold

// Shared-memory layout of a tile of N cells: slots of `cells` elements each,
// 0..4 e and u^mu, then (from off9, a 128-byte boundary) the nine arrays of
// the conserved set, then (from offf) F^0..F^3 and the faces' signal speed.
// Position a of line c sits at c * ld + a * st of its slot.  Across x the
// lines are 8 neighbouring x (ld 1, st 8); along x a line is a row (st 1),
// its length rounded up to an odd number of 16-byte units: whole units as the
// tile copies need it, an odd number so that the 8 lines' cells of one
// position lie in different banks (measured at a length of 128 bytes: the
// FP32 x sweep takes three times as long).
template <class R, int DIR>
struct SweepLay {
  static constexpr int XA = 16 / (int)sizeof(R);  // elements in 16 bytes
  int na, ld, st, cells, off9, offf, size;
  __host__ __device__ explicit SweepLay(int N) {
    na = N + 2 * NG;
    ld = DIR == 0 ? ((na + XA - 1) / XA | 1) * XA : 1;
    st = DIR == 0 ? 1 : kSweepLines;
    cells = kSweepLines * (DIR == 0 ? ld : na);
    const int b128 = 128 / (int)sizeof(R);
    off9 = (5 * cells + b128 - 1) / b128 * b128;
    offf = off9 + 9 * cells;
    size = offf + 5 * cells;
  }
};

// How a stage's tiles are cut: tile length, tiles along, line groups across
// and third-axis extent per direction; the blocks of one launch run through
// the directions one after the other.
struct SweepPlan {
  int n[3], along[3], across[3], third[3];
  __host__ __device__ int blocks(int d) const { return along[d] * across[d] * third[d]; }
};

// ------------------------------------------------- pairs of quantities
// The WENO arithmetic below runs on one quantity (double, float), on two
// doubles, or on two floats in a 64-bit register pair (sm_100's f32x2
// add/mul/fma: one instruction for two lanes, each rounded as the scalar
// operation would).
struct F2 {
  unsigned long long v;
};
struct D2 {
  double a, b;
};
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2u(F2 x, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}
__device__ __forceinline__ F2 v_add(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 v_sub(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 v_mul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 v_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ D2 v_add(D2 x, D2 y) { return {x.a + y.a, x.b + y.b}; }
__device__ __forceinline__ D2 v_sub(D2 x, D2 y) { return {x.a - y.a, x.b - y.b}; }
__device__ __forceinline__ D2 v_mul(D2 x, D2 y) { return {x.a * y.a, x.b * y.b}; }
__device__ __forceinline__ D2 v_fma(D2 x, D2 y, D2 z) { return {fma(x.a, y.a, z.a), fma(x.b, y.b, z.b)}; }
template <class T>
__device__ __forceinline__ T v_add(T x, T y) { return x + y; }
template <class T>
__device__ __forceinline__ T v_sub(T x, T y) { return x - y; }
template <class T>
__device__ __forceinline__ T v_mul(T x, T y) { return x * y; }
template <class T>
__device__ __forceinline__ T v_fma(T x, T y, T z) { return fma(x, y, z); }
// a constant in every lane
template <class V>
__device__ __forceinline__ V v_c(double s) { return (V)s; }
template <>
__device__ __forceinline__ F2 v_c<F2>(double s) { return f2((float)s, (float)s); }
template <>
__device__ __forceinline__ D2 v_c<D2>(double s) { return {s, s}; }

template <class R>
struct PairOf;
template <>
struct PairOf<float> { using V = F2; };
template <>
struct PairOf<double> { using V = D2; };
__device__ __forceinline__ F2 v_pair(float a, float b) { return f2(a, b); }
__device__ __forceinline__ D2 v_pair(double a, double b) { return {a, b}; }
__device__ __forceinline__ void v_split(F2 x, float& a, float& b) { f2u(x, a, b); }
__device__ __forceinline__ void v_split(D2 x, double& a, double& b) { a = x.a; b = x.b; }

// ------------------------------------------------------------------ WENO5
// The face values of a stencil (vh_device.cuh, weno_lr) in difference form.
// With the first differences dm = q_c - q_{c-1}, dp = q_{c+1} - q_c and the
// second differences Dm, D, Dp centred on c-1, c, c+1 the three candidates
// at the right face are q_c + dp/2 - {Dp, D, 3D - 2 Dm}/6, so
//   L = q_c + dp/2 - NL / (6 SL),   R = q_c - dm/2 - NR / (6 SR)
// with the weighted sums below, and mirrored at the left face.  The
// smoothness indicators of NEWEST5/utils.h:102-160 become
//   b0 = (13/12) Dp^2 + (dp - Dp/2)^2,  b1 = (13/12) D^2 + ((dm + dp)/2)^2,
//   b2 = (13/12) Dm^2 + (dm + Dm/2)^2,
// whose first terms (with the weights' eps) are the neighbours' tp, t, tm.
// The weights (0.3, 0.6, 0.1) / (eps + b)^2 are taken over their common
// denominator and times 10, as in weno_lr.  27 operations for both faces of
// a quantity, and 4 per cell for its differences and its t, against 53 for
// the stencil from its five values; the central part q_c + dp/2 cancels in
// V_R - V_L, which is formed from the corrections alone.
template <class V>
struct Face {
  V nl, sl, nr, sr;
};
template <class V>
__device__ __forceinline__ V weno_t(V D) {
  return v_fma(v_mul(v_c<V>(13. / 12.), D), D, v_c<V>(1e-6));
}
template <class V>
__device__ __forceinline__ Face<V> weno_face(V dm, V dp, V Dm, V D, V Dp, V tm, V t, V tp) {
  const V g0 = v_fma(v_c<V>(-0.5), Dp, dp), g1 = v_add(dm, dp), g2 = v_fma(v_c<V>(0.5), Dm, dm);
  const V e0 = v_fma(g0, g0, tp), e1 = v_fma(v_mul(v_c<V>(0.25), g1), g1, t), e2 = v_fma(g2, g2, tm);
  const V E0 = v_mul(e0, e0), E1 = v_mul(e1, e1), E2 = v_mul(e2, e2);
  const V A = v_mul(E1, E2), B = v_mul(v_c<V>(6.), v_mul(E0, E2)), Cc = v_mul(E0, E1);
  const V S = v_add(v_add(A, Cc), B), Z = v_mul(B, D);
  const V X = v_mul(A, Dp), Y = v_mul(Cc, Dm);
  Face<V> f;
  f.sl = v_fma(v_c<V>(2.), A, S);
  f.sr = v_fma(v_c<V>(2.), Cc, S);
  f.nl = v_fma(v_c<V>(-2.), Y, v_fma(v_c<V>(3.), v_fma(Cc, D, X), Z));
  f.nr = v_fma(v_c<V>(-2.), X, v_fma(v_c<V>(3.), v_fma(A, D, Y), Z));
  return f;
}

// ------------------------------------------------------- one cell's terms
// F^0..F^3 along DIR (the fluxes of tau T^{tau mu}) and the velocity v that
// carries pi (F^{4+l} = pi^l v) and is the signal speed: u^i / u^tau, times
// tau along eta (NEWEST5/hydroKT.h:16-83, 161-245).
template <class R, int DIR>
__device__ __forceinline__ void cell_flux(const DevCfg& C, R tau, R e, const R* u, const R* p, R* F, R& v) {
  const bool cart = C.cart;
  const R t2 = cart ? (R)1 : tau * tau;
  const R tf = cart ? (R)1 : tau;
  const R P = eos_P<R>(C, e);
  const R ep = e + P;
  const R u0 = u[0], u1 = u[1], u2 = u[2], u3 = u[3];
  const PiDep<R> d = pi_dep<R>(u0, u1, u2, u3, p, t2);
  const R iu0 = rcp<R>(u0);
  if (DIR == 0) {
    F[0] = tf * (d.tx + u1 * u0 * ep);
    F[1] = tf * (p[0] + P + u1 * u1 * ep);
    F[2] = tf * (p[2] + u1 * u2 * ep);
    F[3] = tf * (p[3] + u1 * u3 * ep);
    v = u1 * iu0;
  } else if (DIR == 1) {
    F[0] = tf * (d.ty + u2 * u0 * ep);
    F[1] = tf * (p[2] + u2 * u1 * ep);
    F[2] = tf * (p[1] + P + u2 * u2 * ep);
    F[3] = tf * (p[4] + u2 * u3 * ep);
    v = u2 * iu0;
  } else {
    F[0] = tf * (d.te + u3 * u0 * ep);
    F[1] = tf * (p[3] + u3 * u1 * ep);
    F[2] = tf * (p[4] + u3 * u2 * ep);
    F[3] = cart ? (d.ee + P + u3 * u3 * ep) : tf * (d.ee + P * rcp<R>(t2) + u3 * u3 * ep);
    // the eta flux of pi and its speed carry a factor tau (NEWEST5/hydroKT.h:76-81)
    v = cart ? u3 * iu0 : tau * u3 * iu0;
  }
}

// ------------------------------------------------------------ TMA staging
// The state is one 4D tensor (x over the padded row pitch, y, z, array): the
// 52 arrays back to back.  A tile is two box copies: arrays 0..4 (e, u^mu)
// and the nine arrays of the conserved set it reads (set A: pi 5..9 then
// T^{tau mu} 10..13; set B: T^{tau mu} 18..21 then pi 22..26).  Along x a
// tile starts at a multiple of its length, which the plan keeps a multiple of
// 16 bytes; across x at a multiple of 8 cells of the padded row.  Cells
// outside the tensor are filled with zeros by the copy and never used.
__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// bounded wait for phase 0 of the barrier; false if it did not complete
__device__ __forceinline__ bool mbar_wait0(unsigned long long* bar, int max_polls) {
  for (int k = 0; k < max_polls; k++) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(0u)
        : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int x, int y, int z, int f,
                                            unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
      "[%6];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(f), "r"(smem_u32(bar))
      : "memory");
}
// the tile's two copies by TMA; false when they did not arrive, and then the
// whole block leaves with the step flagged
template <class R, int DIR>
__device__ __forceinline__ bool tile_by_tma(const DevPtrs<R>& P, const SweepLay<R, DIR>& L, int use_b, int x0, int y0,
                                            int z0, R* sm, const CUtensorMap* map5, const CUtensorMap* map9) {
  __shared__ __align__(8) unsigned long long bar;
  const int tid = threadIdx.x;
  // a box lands only on a 128-byte boundary of shared memory (the same
  // address in every thread: the block leaves as a whole)
  if (smem_u32(sm) & 127u) {
    if (tid == 0) atomicOr(P.status, ST_TMA);
    return false;
  }
  if (tid == 0) mbar_init(&bar, 1);
  __syncthreads();
  if (tid == 0) {
    mbar_expect_tx(&bar, (unsigned)(14 * L.cells * sizeof(R)));
    tma_load_4d(sm, map5, x0, y0, z0, 0, &bar);
    tma_load_4d(sm + L.off9, map9, x0, y0, z0, use_b ? 18 : 5, &bar);
  }
  // every thread waits for the copies (bounded); the block leaves as a
  // whole if any of them gave up, after a second bounded wait for the
  // copies still in flight
  const bool got = mbar_wait0(&bar, 1 << 22);
  if (!__syncthreads_and(got)) {
    if (tid == 0) atomicOr(P.status, ST_TMA);
    mbar_wait0(&bar, 1 << 22);
    return false;
  }
  return true;
}

// --------------------------------------------------------------- the walks
// Both walk cells 2 .. nout + 3 of a line (the first and the last supply the
// outer faces) and keep two differences, two second differences and their t
// of the stencil in registers.  Cell a of the walk completes the face left of
// a and with it cell a - 1, whose divergence (or velocity derivative, formed
// one cell earlier) it stores.  so, sp, sa: the slots of T^{tau tau},
// pi^{xx} and the faces' speed; cell0: global index of the line's position 0.
// One position past the needed ones is loaded and not used; the slot behind
// (the last one holds the speed) keeps that inside the tile.

// A thread owns two quantities, F^l and V^l (tasks 0..8) or two components of
// u^mu (9, 10).
template <class R, int DIR, bool TMA>
__device__ __forceinline__ void walk(const DevPtrs<R>& P, const SweepLay<R, DIR>& L, R* sm, int so, int sp, int sa,
                                     int tid, int nout, R inv_h, bool ok, long long cell0, long long stride) {
  using V = typename PairOf<R>::V;
  constexpr int ST = DIR == 0 ? 1 : kSweepLines;
  const int c = tid % kSweepLines, task = tid / kSweepLines;
  const bool flux = task < 9;
  if (task >= 11 || !ok) return;
  // slots of the thread's two quantities: V^l and F^l (from pi^l and the
  // speed for l >= 4), or two velocities: (u^tau, u^x), (u^eta, u^y)
  const int vslot = task < 4 ? so + task * L.cells : sp + (task - 4) * L.cells;
  const int qb = flux ? vslot : (task == 9 ? 2 : 3) * L.cells;
  const int qa = flux ? (task < 4 ? L.offf + task * L.cells : 0) : (task == 9 ? 1 : 4) * L.cells;
  const bool carried = flux && task >= 4;
  // one divergence array for all directions: y and eta add to it (TMA-staged
  // sweeps always have a set per direction)
  const bool acc = !TMA && DIR != 0 && flux && !P.res1;
  R* const line = sm + c * L.ld;
  const R *pa = line + qa, *pb = line + qb, *pm = line + sa + ST;
  auto load = [&]() {
    const R y = *pb, x = *pa;
    pa += ST;
    pb += ST;
    return v_pair(carried ? x * y : x, y);
  };
  // the results of cell a - 1: into the tile along x, else to memory
  R *oa, *ob;
  if constexpr (DIR == 0) {
    oa = line + (flux ? vslot : qa) + 1;
    ob = line + qb + 1;
  } else {
    oa = (flux ? P.resd(DIR) + (long long)task * P.stride : P.du((task == 9 ? 0 : 9) + DIR)) + cell0 + stride;
    ob = P.du((task == 9 ? 3 : 6) + DIR) + cell0 + stride;
  }
  const R kdiv = (R)-0.5 * inv_h, sixth = (R)(1. / 6.);
  const V q0 = load(), q1 = load();
  V qc = load(), qp = load(), qn = load();  // cells a, a + 1, a + 2
  V dm = v_sub(qc, q1), dp = v_sub(qp, qc);
  V Dm = v_sub(dm, v_sub(q1, q0)), D = v_sub(dp, dm);
  V tm = weno_t<V>(Dm), t = weno_t<V>(D);
  // the left neighbour's right-face sums (FP32: nl holds the quotients nl/sl)
  V nlp = v_c<V>(0.), slp = v_c<V>(1.);
  R fm = 0, hprev = 0;  // F of the left neighbour; flux at the face before (or its derivative)
  R xprev = 0;
  // the value to add to is loaded a cell ahead
  R acc0 = 0;
  if (acc) acc0 = oa[2 * stride];
  // the window moves on by renaming registers, not by copies (its period is 3)
  constexpr int kUnr = sizeof(R) == 8 ? 3 : 6;
#pragma unroll kUnr
  for (int a = 2; a < nout + 4; a++) {
    const V qnn = load();
    const V dn = v_sub(qn, qp), Dp = v_sub(dn, dp), tp = weno_t<V>(Dp);
    R fc, vc;
    v_split(qc, fc, vc);
    const Face<V> f = weno_face<V>(dm, dp, Dm, D, Dp, tm, t, tp);
    const R am = *pm;  // of the face left of cell a (a = 2: not used)
    pm += ST;
    if (flux) {
      R h, acc1 = acc0;
      if (!TMA && DIR != 0 && acc && a > 3 && a < nout + 3) acc1 = oa[stride];
      // 2 H = F_L + F_R - a (V_R - V_L)
      R n0, n1, m0, m1, r0, r1, corr;
      v_split(nlp, n0, n1);
      v_split(f.nr, m0, m1);
      v_split(f.sr, r0, r1);
      if constexpr (sizeof(R) == 8) {
        // one reciprocal for the face's four quotients.  A sum lies between
        // 1e-23 (the weights' eps alone) and 1.3e7 |q|^8: up to |q| = 1e8 the
        // products of four and of their numerators are inside double range
        R s0, s1;
        v_split(slp, s0, s1);
        const R nf = fma(n0, r0, m0 * s0), nv = am * fma(n1, r1, -(m1 * s1)), df = s0 * r0, dv = s1 * r1;
        corr = fma(nf, dv, nv * df) * fast_rcp(df * dv);
        nlp = f.nl;
        slp = f.sl;
      } else {
        R x0, x1;
        corr = fma(am, fma(-m1, fast_rcp(r1), n1), fma(m0, fast_rcp(r0), n0));
        v_split(f.sl, x0, x1);
        nlp = v_mul(f.nl, v_pair(fast_rcp(x0), fast_rcp(x1)));
      }
      h = fma(-sixth, corr, fm + fc);
      const R r = kdiv * (h - hprev);
      if (a > 3) {
        *oa = !TMA && DIR != 0 ? acc0 + r : r;
        acc0 = acc1;
      }
      hprev = h;
      fm = fc;
    } else {
      if (a > 3) {
        *oa = hprev;
        *ob = xprev;
      }
      // (L - R) / h of the cell's own stencil (genWENOder)
      R n0, n1, s0, s1, m0, m1, r0, r1, g0, g1;
      v_split(f.nl, n0, n1);
      v_split(f.sl, s0, s1);
      v_split(f.nr, m0, m1);
      v_split(f.sr, r0, r1);
      v_split(v_add(dm, dp), g0, g1);
      R x0, x1;
      if constexpr (sizeof(R) == 8) {
        const R df = s0 * r0, dv = s1 * r1, inv = fast_rcp(df * dv);
        x0 = fma(n0, r0, -(m0 * s0)) * (dv * inv);
        x1 = fma(n1, r1, -(m1 * s1)) * (df * inv);
      } else {
        x0 = n0 * fast_rcp(s0) - m0 * fast_rcp(r0);
        x1 = n1 * fast_rcp(s1) - m1 * fast_rcp(r1);
      }
      hprev = inv_h * fma(-sixth, x0, (R)0.5 * g0);
      xprev = inv_h * fma(-sixth, x1, (R)0.5 * g1);
    }
    oa += DIR == 0 ? 1 : stride;
    ob += DIR == 0 ? 1 : stride;
    qc = qp;
    qp = qn;
    qn = qnn;
    dm = dp;
    dp = dn;
    Dm = D;
    D = Dp;
    tm = t;
    t = tp;
  }
}

// Generalized minmod: a thread owns F^l and V^l (tasks 0..8) and keeps their
// slopes, s = mm3(theta dm, (dm + dp)/2, theta dp), with
// 2 H = F + F' + (s - s')/2 - a (V' - V - (s + s')/2).
template <class R, int DIR, bool TMA>
__device__ __forceinline__ void walk_minmod(const DevCfg& C, const DevPtrs<R>& P, const SweepLay<R, DIR>& L, R* sm,
                                            int so, int sp, int sa, int tid, int nout, R inv_h, bool ok,
                                            long long cell0, long long stride) {
  constexpr int ST = DIR == 0 ? 1 : kSweepLines;
  const int c = tid % kSweepLines, task = tid / kSweepLines;
  if (task >= 9 || !ok) return;
  const int vslot = task < 4 ? so + task * L.cells : sp + (task - 4) * L.cells;
  const bool carried = task >= 4;
  const bool acc = !TMA && DIR != 0 && !P.res1;
  R* const line = sm + c * L.ld + ST;
  const R *pa = line + (task < 4 ? L.offf + task * L.cells : 0), *pb = line + vslot, *pm = line + sa;
  R* o = DIR == 0 ? line + vslot : P.resd(DIR) + (long long)task * P.stride + cell0 + stride;
  const R kdiv = (R)-0.5 * inv_h, th = (R)C.mm_theta;
  R f0, v0, f1, v1, f2, v2;  // cells a - 1, a, a + 1
  auto load = [&](R& f, R& v) {
    v = *pb;
    f = carried ? *pa * v : *pa;
    pa += ST;
    pb += ST;
  };
  load(f0, v0);
  load(f1, v1);
  R sf = 0, sv = 0, hprev = 0;  // slopes of the left neighbour; flux at the face before
#pragma unroll 3
  for (int a = 2; a < nout + 4; a++) {
    load(f2, v2);
    const R df = f1 - f0, ef = f2 - f1, dv = v1 - v0, ev = v2 - v1;
    const R tf = mm3<R>(th * df, (R)0.5 * (df + ef), th * ef), tv = mm3<R>(th * dv, (R)0.5 * (dv + ev), th * ev);
    const R h = (f0 + f1) + (R)0.5 * (sf - tf) - *pm * (dv - (R)0.5 * (sv + tv));
    pm += ST;
    if (a > 3) {
      const R r = kdiv * (h - hprev);
      *o = acc ? *o + r : r;
    }
    o += DIR == 0 ? 1 : stride;
    hprev = h;
    sf = tf;
    sv = tv;
    f0 = f1;
    v0 = v1;
    f1 = f2;
    v1 = v2;
  }
}

// The velocity derivatives of the minmod sweep's cells, (L - R) / h of the
// WENO5 stencil (genWENOder), a cell a thread: in the walk they would be two
// tasks of three times the others' length.
template <class R, int DIR, class Ok, class Base>
__device__ __forceinline__ void cell_derivatives(const DevPtrs<R>& P, const SweepLay<R, DIR>& L, const R* sm, int tid,
                                                 int nout, R inv_h, Ok&& line_ok, Base&& cell_of) {
  using V = typename PairOf<R>::V;
  constexpr int ST = DIR == 0 ? 1 : kSweepLines;
  const int lanes = DIR == 0 ? 32 : kSweepLines;  // along x a warp takes a line
  for (int q = tid / lanes; q < (DIR == 0 ? kSweepLines : nout); q += kSweepThreads / lanes)
    for (int r = tid % lanes; r < (DIR == 0 ? nout : kSweepLines); r += lanes) {
      const int c = DIR == 0 ? q : r, a = NG + (DIR == 0 ? r : q);
      if (!line_ok(c)) continue;
      const R* s = sm + c * L.ld + a * ST;
      const long long g = cell_of(c, a);
#pragma unroll
      for (int l = 0; l < 4; l += 2) {
        V x[5], d[4], D[3], t[3];
#pragma unroll
        for (int m = 0; m < 5; m++) x[m] = v_pair(s[(1 + l) * L.cells + (m - 2) * ST], s[(2 + l) * L.cells + (m - 2) * ST]);
#pragma unroll
        for (int m = 0; m < 4; m++) d[m] = v_sub(x[m + 1], x[m]);
#pragma unroll
        for (int m = 0; m < 3; m++) {
          D[m] = v_sub(d[m + 1], d[m]);
          t[m] = weno_t<V>(D[m]);
        }
        const Face<V> f = weno_face<V>(d[1], d[2], D[0], D[1], D[2], t[0], t[1], t[2]);
        R n[2], sl[2], m0[2], sr[2], gsum[2];
        v_split(f.nl, n[0], n[1]);
        v_split(f.sl, sl[0], sl[1]);
        v_split(f.nr, m0[0], m0[1]);
        v_split(f.sr, sr[0], sr[1]);
        v_split(v_add(d[1], d[2]), gsum[0], gsum[1]);
#pragma unroll
        for (int k = 0; k < 2; k++)
          P.du((l + k) * 3 + DIR)[g] =
              inv_h * fma((R)(-1. / 6.), n[k] * fast_rcp(sl[k]) - m0[k] * fast_rcp(sr[k]), (R)0.5 * gsum[k]);
      }
    }
}

// --------------------------------------------------------------- the tile
// Tile bx along the direction (N cells from lo + bx N), line group by across
// it, bz the third axis (interior index).  MM: generalized-minmod face
// states (the velocity derivative stays WENO5, as in the reference).
template <class R, int DIR, bool MM, bool TMA>
__device__ __forceinline__ void sweep_tile(const DevCfg& C, const DevPtrs<R>& P, int use_b, R tau, R inv_h, int N,
                                           int bx, int by, int bz, R* sm, const CUtensorMap* map5 = nullptr,
                                           const CUtensorMap* map9 = nullptr) {
  constexpr int T = kSweepThreads;
  const SweepLay<R, DIR> L(N);
  const int tid = threadIdx.x;
  const int lo = DIR == 0 ? C.il : (DIR == 1 ? C.jl : C.kl), hi = DIR == 0 ? C.ir : (DIR == 1 ? C.jr : C.kr);
  const int a0 = lo - NG + bx * N;  // global along index of position 0
  const int nout = min(N, hi - (a0 + NG));
  const int npos = nout + 2 * NG;   // positions the outputs need; all inside the grid
  const long long stride = DIR == 0 ? 1 : (DIR == 1 ? (long long)C.px : (long long)C.px * C.gy);
  // the first cell of line c's cross section.  Across x the tiles start at
  // x = xt0 + 8 by: on a handle's padded rows xt0 = 0, so that a tile's x
  // segment sits on whole 32-byte sectors (the lines in the ghost cells are
  // idle); on unpadded rows xt0 = il.
  const int i0 = DIR == 0 ? 0 : C.xt0 + by * kSweepLines;
  const int j0 = DIR == 0 ? C.jl + by * kSweepLines : (DIR == 1 ? 0 : C.jl + bz);
  const int k0 = DIR == 2 ? 0 : C.kl + bz;
  auto line_ok = [&](int c) { return DIR == 0 ? j0 + c < C.jr : (i0 + c >= C.il && i0 + c < C.ir); };
  auto line_base = [&](int c) { return DIR == 0 ? cix(C, 0, j0 + c, k0) : cix(C, i0 + c, j0, k0); };

  // ---- the tile: e, u^mu, T^{tau mu}, pi
  if constexpr (TMA) {
    if (!tile_by_tma<R, DIR>(P, L, use_b, DIR == 0 ? a0 : i0, DIR == 1 ? a0 : j0, DIR == 2 ? a0 : k0, sm, map5, map9))
      return;
  } else {
    // 14 loads a cell through the cache: rows of x first
    const int lanes = DIR == 0 ? 32 : kSweepLines;
    for (int q = tid / lanes; q < (DIR == 0 ? kSweepLines : npos); q += T / lanes)
      for (int r = tid % lanes; r < (DIR == 0 ? npos : kSweepLines); r += lanes) {
        const int c = DIR == 0 ? q : r, a = DIR == 0 ? r : q;
        R* s = sm + c * L.ld + a * L.st;
        const bool ok = line_ok(c);
        const long long g = line_base(c) + (long long)(a0 + a) * stride;
#pragma unroll
        for (int l = 0; l < 5; l++) s[l * L.cells] = ok ? P.base0[(long long)l * P.stride + g] : (R)0;
        const R* set = use_b ? P.base1 : P.base0 + 5 * P.stride;
#pragma unroll
        for (int l = 0; l < 9; l++) s[L.off9 + l * L.cells] = ok ? set[(long long)l * P.stride + g] : (R)0;
      }
    __syncthreads();
  }

  // ---- fluxes, tau T^{tau mu} and speed of every cell, in place
  const int so = L.off9 + (use_b ? 0 : 5 * L.cells);  // slot of T^{tau tau}
  const int sp = L.off9 + (use_b ? 4 * L.cells : 0);  // slot of pi^{xx}
  const int sa = L.offf + 4 * L.cells;                // slot of the faces' speed
  for (int t = tid; t < kSweepLines * npos; t += T) {
    R* s = sm + (t % kSweepLines) * L.ld + (t / kSweepLines) * L.st;
    R u[4], p[5], F[4], v;
#pragma unroll
    for (int l = 0; l < 4; l++) u[l] = s[(1 + l) * L.cells];
#pragma unroll
    for (int l = 0; l < 5; l++) p[l] = s[sp + l * L.cells];
    cell_flux<R, DIR>(C, tau, s[0], u, p, F, v);
    s[0] = v;
#pragma unroll
    for (int l = 0; l < 4; l++) s[L.offf + l * L.cells] = F[l];
    if (!C.cart) {
#pragma unroll
      for (int l = 0; l < 4; l++) s[so + l * L.cells] *= tau;
    }
  }
  __syncthreads();

  // ---- the faces' maximal signal speed; face f is the one right of
  // position f.  Speeds are zero in ghost cells, and the face left of the
  // first interior cell takes no dissipation: its max speed sits in a ghost
  // cell the reference never fills (NEWEST5/hydroKT.h:265-314 vs 435-440).
  for (int t = tid; t < kSweepLines * (nout + 1); t += T) {
    const int f = 2 + t / kSweepLines, g = a0 + f;
    R* s = sm + (t % kSweepLines) * L.ld + f * L.st;
    R q[6];
#pragma unroll
    for (int m = 0; m < 6; m++) q[m] = (g - 2 + m >= lo && g - 2 + m < hi) ? s[(m - 2) * L.st] : (R)0;
    R amax = 0;
    if (g + 1 != lo) {
      R l, r;
      if constexpr (MM) {
        l = mm_left<R>((R)C.mm_theta, q[1], q[2], q[3]);
        r = mm_right<R>((R)C.mm_theta, q[2], q[3], q[4]);
      } else {
        R d[5], D[4], w[4];
#pragma unroll
        for (int m = 0; m < 5; m++) d[m] = q[m + 1] - q[m];
#pragma unroll
        for (int m = 0; m < 4; m++) {
          D[m] = d[m + 1] - d[m];
          w[m] = weno_t<R>(D[m]);
        }
        const Face<R> a = weno_face<R>(d[1], d[2], D[0], D[1], D[2], w[0], w[1], w[2]);
        const Face<R> b = weno_face<R>(d[2], d[3], D[1], D[2], D[3], w[1], w[2], w[3]);
        const R half = (R)0.5 * d[2], sixth = (R)(1. / 6.);
        l = q[2] + half - sixth * (a.nl * fast_rcp(a.sl));
        r = q[3] - half - sixth * (b.nr * fast_rcp(b.sr));
      }
      amax = fmax(fabs(l), fabs(r));
    }
    s[sa] = amax;
  }
  __syncthreads();

  // ---- the walk along the lines
  const bool ok = line_ok(tid % kSweepLines);
  const long long cell0 = line_base(tid % kSweepLines) + (long long)a0 * stride;
  if constexpr (MM) {
    cell_derivatives<R, DIR>(P, L, sm, tid, nout, inv_h, line_ok,
                             [&](int c, int a) { return line_base(c) + (long long)(a0 + a) * stride; });
    walk_minmod<R, DIR, TMA>(C, P, L, sm, so, sp, sa, tid, nout, inv_h, ok, cell0, stride);
  } else {
    walk<R, DIR, TMA>(P, L, sm, so, sp, sa, tid, nout, inv_h, ok, cell0, stride);
  }
  if constexpr (DIR == 0) {
    // a warp's lanes walked along rows a pitch apart: the results, left in
    // the tile, go out row by row
    __syncthreads();
    for (int cc = tid / 32; cc < kSweepLines; cc += T / 32) {
      if (!line_ok(cc)) continue;
      const R* s = sm + cc * L.ld;
      R* const r0 = P.resd(0) + line_base(cc) + a0;
      R* const d0 = P.du(0) + line_base(cc) + a0;
      for (int a = NG + tid % 32; a < NG + nout; a += 32) {
#pragma unroll
        for (int q = 0; q < 9; q++) r0[(long long)q * P.stride + a] = s[(q < 4 ? so + q * L.cells : sp + (q - 4) * L.cells) + a];
        if (!MM) {
#pragma unroll
          for (int q = 0; q < 4; q++) d0[(long long)(q * 3) * P.stride + a] = s[(1 + q) * L.cells + a];
        }
      }
    }
  }
}

// ------------------------------------------------------------- host side
// The tiles of a grid: as long as 24 cells (FP64) or 30 (FP32), which leaves
// 5 and 9 blocks on an SM, and equally long along a line (161 cells: 7 tiles
// of 23 or 24).  Measured on the 161x161x41 event, ms per step at 24 / 28 / 30
// cells: FP64 1.293 / 1.383 / 1.381, FP32 0.808 / 0.802 / 0.802.  Grids with
// fewer than two such tiles per SM take up to 16 cells, more blocks of less
// latency (129x129: 0.0543 ms per step at 16, 0.0568 at 24, 0.0556 at 8).
// Where the directions are launched one by one (together false: the
// allocation-free step's largest grids, up to 61,680 cells with ghosts) a
// launch has a third or half of the tiles, and 12 cells are best: 240x240 at
// 8 / 12 / 16 / 24 cells 102 / 88 / 91 / 104 us a step, 34x34x32 121 / 111 /
// 116 / 125.
template <class R>
static SweepPlan sweep_plan(const DevCfg& C, bool together = true) {
  SweepPlan p{};
  const int len[3] = {C.nx, C.ny, C.kr - C.kl}, dirs = C.bi ? 2 : 3;
  const int longest = together ? (sizeof(R) == 8 ? 24 : 30) : 12;
  for (int most : {longest, longest < 16 ? longest : 16}) {
    int tiles = 0;
    for (int d = 0; d < dirs; d++) {
      const int k = (len[d] + most - 1) / most;
      int n = (len[d] + k - 1) / k;
      // along x a tile starts at a multiple of 16 bytes; across x an odd
      // number of positions keeps neighbouring slots in different banks
      if (d == 0 && k > 1) n = (n + SweepLay<R, 0>::XA - 1) / SweepLay<R, 0>::XA * SweepLay<R, 0>::XA;
      if (d > 0) n |= 1;
      p.n[d] = n;
      p.along[d] = (len[d] + n - 1) / n;
      p.across[d] = d == 0 ? (C.ny + kSweepLines - 1) / kSweepLines : (C.ir - C.xt0 + kSweepLines - 1) / kSweepLines;
      p.third[d] = d == 2 ? C.ny : len[2];
      tiles += p.blocks(d);
    }
    if (tiles >= 2 * 148) break;
  }
  return p;
}

// shared memory of a launch over the first `dirs` directions
template <class R>
static size_t sweep_smem(const SweepPlan& p, int dirs) {
  int m = 0;
  const int s[3] = {SweepLay<R, 0>(p.n[0]).size, SweepLay<R, 1>(p.n[1]).size, SweepLay<R, 2>(p.n[2]).size};
  for (int d = 0; d < dirs; d++) m = s[d] > m ? s[d] : m;
  return (size_t)m * sizeof(R);
}

}  // namespace vh
