// Isothermal freeze-out hypersurface and Cooper-Frye spectra on the GPU,
// from device arrays: the per-simplex arithmetic of vh_freezeout.cuh, in two
// passes so that the elements land in the host entry points' order (cube
// order, x fastest): a count pass from the signs of T - T_fo alone, which also
// lists the cut cubes, an exclusive scan of the counts, and an emit pass, a
// group of lanes per cut cube and a lane per simplex, that writes the cube's
// elements from its offset.  The list's order varies from run to run, the
// elements' places do not.  The spectra are sums over the elements per
// momentum bin in a fixed order (deterministic).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <vector>

#include <cub/device/device_scan.cuh>

#include "vh.h"
#include "vh_freezeout.cuh"
#include "vh_nvtx.h"

namespace {

constexpr int kThreads = 256;

// counts[c]: elements of cube c; list[0 .. *ncut): the cubes with any
template <int D>
__global__ void __launch_bounds__(kThreads) k_fo_count(vh_fo::Geo g, const double* __restrict__ t0,
                                                        const double* __restrict__ t1, long long ncubes,
                                                        long long* __restrict__ counts, int* __restrict__ list,
                                                        int* __restrict__ ncut) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long n = 0;
  if (c < ncubes) {
    int i, j, k;
    vh_fo::cube_ijk(g, c, &i, &j, &k);
    counts[c] = n = vh_fo::count<D>(g, i, j, k, t0, t1);
  }
  const unsigned cut = __ballot_sync(0xffffffffu, n != 0);
  if (cut == 0) return;
  const int lane = threadIdx.x & 31;
  int at = 0;
  if (lane == 0) at = atomicAdd(ncut, __popc(cut));
  at = __shfl_sync(0xffffffffu, at, 0);
  if (n) list[at + __popc(cut & ((1u << lane) - 1))] = (int)c;
}

// a cube's corners, read where a simplex needs them
template <int D>
struct CornersAt {
  const vh_fo::Geo& g;
  const double *t0, *t1, *u0, *u1;
  int i, j, k;
  double lo[D], hi[D];
  __device__ __forceinline__ double x(int v, int q) const { return ((v >> q) & 1) ? hi[q] : lo[q]; }
  __device__ __forceinline__ double f(int v) const {
    return ((v & 1) ? t1 : t0)[vh_fo::corner_cell<D>(g, i, j, k, v)] - g.t_fo;
  }
  __device__ __forceinline__ double u(int v, int q) const {
    return ((v & 1) ? u1 : u0)[q * g.n + vh_fo::corner_cell<D>(g, i, j, k, v)];
  }
};

// A cut cube takes a whole warp in 3+1D (24 simplices) and 8 lanes in 2+1D
// (6).  A thread per cube had left one or two lanes of a warp at work, each
// on 24 simplices in turn from its own stack (121x121x31, 0.8 M elements:
// 0.92 ms; now 0.15).
template <int D>
__global__ void __launch_bounds__(kThreads) k_fo_emit(vh_fo::Geo g, const double* __restrict__ t0,
                                                       const double* __restrict__ t1, const double* __restrict__ u0,
                                                       const double* __restrict__ u1, const int* __restrict__ list,
                                                       const int* __restrict__ ncut,
                                                       const long long* __restrict__ offs, double* __restrict__ out,
                                                       long long cap) {
  constexpr int G = D == 3 ? 8 : 32, S = D == 3 ? 6 : 24, MANY = D == 3 ? 2 : 3;
  const int lane = threadIdx.x & 31, sx = lane % G, first = lane - sx;
  int v[5];
  vh_fo::kuhn_simplex(sx < S ? sx : 0, D, v);
  const int n = *ncut;
  const long long groups = (long long)gridDim.x * (kThreads / G);
  for (long long at = (long long)blockIdx.x * (kThreads / G) + threadIdx.x / G;; at += groups) {
    // the warp's groups step together: their lanes meet in the ballots
    if (!__any_sync(0xffffffffu, at < n)) break;
    const bool live = at < n && sx < S;
    const long long c = at < n ? list[at] : 0;
    CornersAt<D> K{g, t0, t1, u0, u1, 0, 0, 0, {}, {}};
    vh_fo::cube_ijk(g, c, &K.i, &K.j, &K.k);
    K.lo[0] = g.tau0;
    K.hi[0] = g.tau1;
    K.lo[1] = g.x0 + (K.i - vh_fo::kG) * g.dx;
    K.hi[1] = g.x0 + (K.i + 1 - vh_fo::kG) * g.dx;
    K.lo[2] = g.y0 + (K.j - vh_fo::kG) * g.dy;
    K.hi[2] = g.y0 + (K.j + 1 - vh_fo::kG) * g.dy;
    if (D == 4) {
      K.lo[D - 1] = g.z0 + (K.k - vh_fo::kG) * g.dz;
      K.hi[D - 1] = g.z0 + (K.k + 1 - vh_fo::kG) * g.dz;
    }
    int nh = 0;
    if (live)
      for (int q = 0; q <= D; q++) nh += K.f(v[q]) > 0;
    const int nc = D + 1 - nh;
    const bool cut = live && nh && nc, lone = cut && (nh == 1 || nc == 1);
    // the elements of the cube's simplices before this one
    const unsigned before = ((1u << lane) - 1) & ~((1u << first) - 1);
    const unsigned one = __ballot_sync(0xffffffffu, lone) & before, many = __ballot_sync(0xffffffffu, cut && !lone) & before;
    if (cut) {
      vh_fo::Sink s{out, offs[c] + __popc(one) + MANY * __popc(many), cap};  // writes below cap only
      if constexpr (D == 3)
        vh_fo::simplex2(K, v, s);
      else
        vh_fo::simplex3(K, v, s);
    }
  }
}

// ---- spectra
// A block sums a share of the elements for kBins momentum bins at once, 128
// elements at a time: the block copies their rows into shared memory, a thread
// forms what depends on its element alone (in 3+1D cosh and sinh of y - eta;
// in 2+1D the Bessel functions, which depend on the bin through m_T only),
// then each warp takes kWarpBins bins, held in registers, through all 128.
// 0.8 M elements and 8 x 16 bins: 0.33 ms, bound by the FP64 exponentials.  An
// element a thread with all 16 bins held 128 registers with spills and read its
// row 96 bytes from the next lane's, 0.79 ms; one block per bin before that,
// forming the element's part anew for each, 4.06 ms.  4 blocks per SM (102
// registers): with 5, 6 and 8 the call takes 0.93, 0.82 and 0.86 ms against 0.76.
// bins: m_T, p_x, p_y, kBins a tile, zeros where a tile has fewer; part: a
// partial sum per bin and share of the elements.
constexpr int kBins = 16, kCfThreads = 128, kCfWarps = kCfThreads / 32, kWarpBins = kBins / kCfWarps;
template <int D>
__global__ void __launch_bounds__(kCfThreads, 4) k_cooper_frye(const double* __restrict__ el, long long count,
                                                             const double* __restrict__ bins, double y, double t_fo,
                                                             double* __restrict__ part) {
  // a row's words; an odd pitch keeps lanes an element apart on their own banks
  constexpr int W = D == 3 ? vh_fo::kW2 : vh_fo::kW3, P = W | 1;
  __shared__ double row[kCfThreads * P], term[6][kCfThreads];
  const int tid = threadIdx.x, lane = tid & 31;
  const double* mine = bins + ((long long)blockIdx.x * kBins + tid / 32 * kWarpBins) * 3;
  double mt[kWarpBins], px[kWarpBins], py[kWarpBins], acc[kWarpBins];
#pragma unroll
  for (int b = 0; b < kWarpBins; b++) {
    mt[b] = D == 3 ? 1.0 : mine[3 * b];  // 2+1D: within the element's part
    px[b] = mine[3 * b + 1];
    py[b] = mine[3 * b + 2];
    acc[b] = 0;
  }
  const double it = 1.0 / t_fo, mt_tile = bins[(long long)blockIdx.x * kBins * 3];
  for (long long e0 = (long long)blockIdx.y * kCfThreads; e0 < count; e0 += (long long)gridDim.y * kCfThreads) {
    const int live = (int)(count - e0 < kCfThreads ? count - e0 : kCfThreads);
    // row was last read before the previous turn's second barrier
    for (int w = tid; w < live * W; w += kCfThreads) row[w / W * P + w % W] = el[e0 * W + w];
    __syncthreads();
    // the term of a bin: (m_T A + p_x B + p_y C) exp(p_x V + p_y Y - m_T U)
    double A = 0, B = 0, C = 0, U = 0, V = 0, Y = 0;
    if (tid < live) {
      const double* q = row + tid * P;
      if constexpr (D == 4) {
        const double tau = q[0], ch = cosh(y - q[3]), sh = sinh(y - q[3]);
        A = ch * q[4] + sh / tau * q[7], B = q[5], C = q[6];
        U = (ch * q[8] - tau * sh * q[11]) * it, V = q[9] * it, Y = q[10] * it;
      } else {
        double k0e, k1e;
        U = mt_tile * q[6] * it;
        vh_fo::bessel_k01e(U, &k0e, &k1e);
        A = 2 * mt_tile * k1e * q[3], B = 2 * k0e * q[4], C = 2 * k0e * q[5], V = q[7] * it, Y = q[8] * it;
      }
    }
    term[0][tid] = A, term[1][tid] = B, term[2][tid] = C;
    term[3][tid] = U, term[4][tid] = V, term[5][tid] = Y;
    __syncthreads();
#pragma unroll 1
    for (int i = lane; i < live; i += 32) {
      const double a = term[0][i], b1 = term[1][i], c = term[2][i], u = term[3][i], v = term[4][i], yy = term[5][i];
#pragma unroll
      for (int b = 0; b < kWarpBins; b++)
        acc[b] += (mt[b] * a + px[b] * b1 + py[b] * c) * exp(px[b] * v + py[b] * yy - mt[b] * u);
    }
  }
#pragma unroll
  for (int b = 0; b < kWarpBins; b++) {
    for (int o = 16; o > 0; o >>= 1) acc[b] += __shfl_down_sync(0xffffffffu, acc[b], o);
    if (lane == 0)
      part[((long long)blockIdx.x * kBins + tid / 32 * kWarpBins + b) * gridDim.y + blockIdx.y] = acc[b];
  }
}
// The same for tiles of one bin, a thread an element with all of the bin's
// term: in 2+1D with a single azimuth nothing of an element is shared between
// bins, and the Bessel functions, which bound it, want the warps that an
// accumulator and no staging leave room for.  0.8 M elements and 400 x 1 bins:
// 54.3 ms as tiles of 16, 46.0 with the missing bins left out of them, 34.9 so,
// and 37.8 a bin a block over all elements (with two azimuths 69.8 a bin a
// block, 54.3 as tiles).
__global__ void __launch_bounds__(kThreads) k_cooper_frye_one(const double* __restrict__ el, long long count,
                                                              const double* __restrict__ bins, double t_fo,
                                                              double* __restrict__ part) {
  __shared__ double red[kThreads / 32];
  const int tid = threadIdx.x;
  const double* m = bins + (long long)blockIdx.x * 3;
  const double mt = m[0], px = m[1], py = m[2];
  double s = 0;
  for (long long e = (long long)blockIdx.y * kThreads + tid; e < count; e += (long long)gridDim.y * kThreads)
    s += vh_fo::cf2_term(el + vh_fo::kW2 * e, mt, px, py, t_fo);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (tid % 32 == 0) red[tid / 32] = s;
  __syncthreads();
  if (tid) return;
  for (int w = 1; w < kThreads / 32; w++) s += red[w];
  part[(long long)blockIdx.x * gridDim.y + blockIdx.y] = s;
}
// the shares' sums, one warp per slot; slot q of tile t is the bin
// first_bin(t) + q of the spectrum
struct CfTiles {
  int nphi, width, per_row;  // per_row: tiles of a p_T (2+1D), 0: tiles run on over the bins (3+1D)
  long long nb;
  __host__ __device__ long long first(long long t) const {
    return per_row ? t / per_row * nphi + t % per_row * width : t * width;
  }
  __host__ __device__ long long end(long long t) const {
    const long long f = first(t) + width, m = per_row ? (t / per_row + 1) * nphi : nb;
    return f < m ? f : m;
  }
};
__global__ void k_cf_final(const double* __restrict__ part, int shares, CfTiles tl, long long tile0, int tiles,
                           double pref, double* __restrict__ out) {
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 32;
  const int lane = threadIdx.x & 31;
  if (w >= (long long)tiles * tl.width) return;
  const long long t = tile0 + w / tl.width, bin = tl.first(t) + w % tl.width;
  if (bin >= tl.end(t)) return;
  double s = 0;
  for (int k = lane; k < shares; k += 32) s += part[w * shares + k];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) out[bin] = pref * s;
}

inline unsigned blocks(long long n) { return (unsigned)((n + kThreads - 1) / kThreads); }

// the surface between two device slices; scratch from the stream's pool
template <int D>
int surface(const vh_fo::Geo& g, const double* t0, const double* t1, const double* u0, const double* u1, double* out,
            long long cap, long long* count, cudaStream_t st) {
  const long long nc = vh_fo::cubes(g, D);
  if (nc > INT_MAX) return VH_E_ARG;  // one scan of int-counted items
  VhNvtxRange range("freeze-out surface");
  size_t scan_bytes = 0;
  const long long* scan_in = nullptr;
  long long* scan_out = nullptr;
  if (cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, scan_in, scan_out, (int)nc, st) != cudaSuccess)
    return VH_E_CUDA;
  const size_t words = 2 * (size_t)nc;  // counts, offsets
  const size_t ints = (size_t)nc + 1;   // cut cubes and their number
  char* buf = nullptr;
  if (cudaMallocAsync((void**)&buf, words * sizeof(long long) + ints * sizeof(int) + scan_bytes + 512, st) !=
      cudaSuccess) {
    cudaGetLastError();
    return VH_E_NOMEM;
  }
  long long* counts = reinterpret_cast<long long*>(buf);
  long long* offs = counts + nc;
  scan_in = counts;
  scan_out = offs;
  int* list = reinterpret_cast<int*>(offs + nc);
  int* ncut = list + nc;
  void* scan_tmp = buf + ((words * sizeof(long long) + ints * sizeof(int) + 255) / 256) * 256;
  int rc = VH_OK;
  long long tail[2] = {0, 0};
  if (cudaMemsetAsync(ncut, 0, sizeof(int), st) != cudaSuccess) rc = VH_E_CUDA;
  k_fo_count<D><<<blocks(nc), kThreads, 0, st>>>(g, t0, t1, nc, counts, list, ncut);
  if (cudaGetLastError() != cudaSuccess ||
      cub::DeviceScan::ExclusiveSum(scan_tmp, scan_bytes, scan_in, scan_out, (int)nc, st) != cudaSuccess ||
      cudaMemcpyAsync(&tail[0], offs + nc - 1, sizeof(long long), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaMemcpyAsync(&tail[1], counts + nc - 1, sizeof(long long), cudaMemcpyDeviceToHost, st) != cudaSuccess)
    rc = VH_E_CUDA;
  if (rc == VH_OK && cap > 0) {
    // as many warps as an SM holds, each taking cut cubes in turn
    const unsigned most = 148 * 8, need = blocks(nc * (D == 3 ? 8 : 32));
    k_fo_emit<D><<<need < most ? need : most, kThreads, 0, st>>>(g, t0, t1, u0, u1, list, ncut, offs, out, cap);
    if (cudaGetLastError() != cudaSuccess) rc = VH_E_CUDA;
  }
  if (cudaFreeAsync(buf, st) != cudaSuccess && rc == VH_OK) rc = VH_E_CUDA;
  if (cudaStreamSynchronize(st) != cudaSuccess && rc == VH_OK) rc = VH_E_CUDA;
  if (rc != VH_OK) return rc;
  *count = tail[0] + tail[1];
  return *count > cap ? VH_E_ARG : VH_OK;
}

// the spectrum of count device elements at the host's momentum bins
template <int D>
int spectrum(const double* el, long long count, double t_fo, double mass, double degeneracy, double y,
             const double* pt, int npt, const double* phi, int nphi, double* out, cudaStream_t st) {
  const long long nb = (long long)npt * nphi;
  if (nb > INT_MAX) return VH_E_ARG;
  VhNvtxRange range("Cooper-Frye spectrum");
  // bins in tiles of kBins, in 2+1D the azimuths of one p_T (the Bessel
  // functions depend on p_T alone), of 1 where that is one; in 3+1D any.  A
  // launch holds 1024 x kBins bins at most, which bounds the scratch
  const bool one = D == 3 && nphi == 1;
  const int width = one ? 1 : kBins;
  const long long most_tiles = 1024 * kBins / width;
  const CfTiles tl{nphi, width, D == 3 ? (nphi + width - 1) / width : 0, nb};
  const long long tiles = D == 3 ? (long long)npt * tl.per_row : (nb + width - 1) / width;
  const int chunk = (int)(tiles < most_tiles ? tiles : most_tiles);
  // shares of the elements: about four blocks per SM over the launch's tiles
  // (eight of single bins)
  const int threads = one ? kThreads : kCfThreads;
  const long long most = (count + threads - 1) / threads;
  auto shares_of = [&](long long n) {
    const long long k = ((one ? 8 : 4) * 148 + n - 1) / n;
    return k > most ? (most < 1 ? 1 : most) : k;
  };
  const long long last = tiles % chunk;  // tiles of a shorter last launch
  const long long parts = std::max(chunk * shares_of(chunk), last ? last * shares_of(last) : 0);
  std::vector<double> bins(3 * width * (size_t)chunk);  // of one launch
  const size_t w_bins = 3 * width * (size_t)chunk, w_part = (size_t)(width * parts);
  double* dbuf = nullptr;
  if (cudaMallocAsync((void**)&dbuf, (w_bins + w_part + (size_t)nb) * sizeof(double), st) != cudaSuccess) {
    cudaGetLastError();
    return VH_E_NOMEM;
  }
  double *part = dbuf + w_bins, *dout = part + w_part;
  const double pref = degeneracy / (8 * M_PI * M_PI * M_PI);
  int rc = VH_OK;
  for (long long t0 = 0; t0 < tiles && rc == VH_OK; t0 += chunk) {
    const int n = (int)(tiles - t0 < chunk ? tiles - t0 : chunk);
    std::fill(bins.begin(), bins.end(), 0.0);
    for (long long t = t0; t < t0 + n; t++)
      for (long long i = tl.first(t); i < tl.end(t); i++) {
        double* q = &bins[3 * (size_t)((t - t0) * width + i - tl.first(t))];
        const double p = pt[i / nphi], f = phi[i % nphi];
        q[0] = std::sqrt(mass * mass + p * p);
        q[1] = p * std::cos(f);
        q[2] = p * std::sin(f);
      }
    // (from pageable memory: staged when the call returns)
    if (cudaMemcpyAsync(dbuf, bins.data(), 3 * width * (size_t)n * sizeof(double),
                        cudaMemcpyHostToDevice, st) != cudaSuccess) {
      rc = VH_E_CUDA;
      break;
    }
    const int shares = (int)shares_of(n);
    const dim3 grid((unsigned)n, (unsigned)shares);
    if (one) k_cooper_frye_one<<<grid, kThreads, 0, st>>>(el, count, dbuf, t_fo, part);
    else k_cooper_frye<D><<<grid, kCfThreads, 0, st>>>(el, count, dbuf, y, t_fo, part);
    k_cf_final<<<(unsigned)(((long long)n * width * 32 + 255) / 256), 256, 0, st>>>(part, shares, tl, t0, n, pref, dout);
    if (cudaGetLastError() != cudaSuccess) rc = VH_E_CUDA;
  }
  if (rc == VH_OK &&
      cudaMemcpyAsync(out, dout, (size_t)nb * sizeof(double), cudaMemcpyDeviceToHost, st) != cudaSuccess)
    rc = VH_E_CUDA;
  if (cudaFreeAsync(dbuf, st) != cudaSuccess && rc == VH_OK) rc = VH_E_CUDA;
  if (cudaStreamSynchronize(st) != cudaSuccess && rc == VH_OK) rc = VH_E_CUDA;
  return rc;
}

}  // namespace

extern "C" int vh_freezeout_2d_device(int nx, int ny, double dx, double dy, double tau0, double tau1, const double* t0,
                                      const double* t1, const double* u0, const double* u1, double t_fo, double* out,
                                      long long cap, long long* count, void* stream) {
  if (nx < 2 || ny < 2 || !(dx > 0) || !(dy > 0) || !(tau1 > tau0) || !t0 || !t1 || !u0 || !u1 || !count ||
      (cap > 0 && !out) || cap < 0)
    return VH_E_ARG;
  const vh_fo::Geo g = vh_fo::make_geo(nx, ny, 1, dx, dy, 0.0, tau0, tau1, t_fo, true);
  return surface<3>(g, t0, t1, u0, u1, out, cap, count, static_cast<cudaStream_t>(stream));
}

extern "C" int vh_freezeout_3d_device(int nx, int ny, int nz, double dx, double dy, double dz, double tau0,
                                      double tau1, const double* t0, const double* t1, const double* u0,
                                      const double* u1, double t_fo, double* out, long long cap, long long* count,
                                      void* stream) {
  if (nx < 2 || ny < 2 || nz < 2 || !(dx > 0) || !(dy > 0) || !(dz > 0) || !(tau1 > tau0) || !t0 || !t1 || !u0 ||
      !u1 || !count || (cap > 0 && !out) || cap < 0)
    return VH_E_ARG;
  const vh_fo::Geo g = vh_fo::make_geo(nx, ny, nz, dx, dy, dz, tau0, tau1, t_fo, false);
  return surface<4>(g, t0, t1, u0, u1, out, cap, count, static_cast<cudaStream_t>(stream));
}

extern "C" int vh_cooper_frye_2d_device(const double* elements, long long count, double t_fo, double mass,
                                        double degeneracy, const double* pt, int npt, const double* phi, int nphi,
                                        double* out, void* stream) {
  if ((count > 0 && !elements) || count < 0 || !(t_fo > 0) || !(mass >= 0) || !pt || !phi || npt < 1 || nphi < 1 ||
      !out || !vh_fo::bins_ok(mass, pt, npt, phi, nphi, false))
    return VH_E_ARG;
  return spectrum<3>(elements, count, t_fo, mass, degeneracy, 0.0, pt, npt, phi, nphi, out,
                     static_cast<cudaStream_t>(stream));
}

extern "C" int vh_cooper_frye_3d_device(const double* elements, long long count, double t_fo, double mass,
                                        double degeneracy, double y, const double* pt, int npt, const double* phi,
                                        int nphi, double* out, void* stream) {
  if ((count > 0 && !elements) || count < 0 || !(t_fo > 0) || !(mass >= 0) || !std::isfinite(y) || !pt || !phi ||
      npt < 1 || nphi < 1 || !out || !vh_fo::bins_ok(mass, pt, npt, phi, nphi, true))
    return VH_E_ARG;
  return spectrum<4>(elements, count, t_fo, mass, degeneracy, y, pt, npt, phi, nphi, out,
                     static_cast<cudaStream_t>(stream));
}
