// Single-particle accumulator: the delayed NFFT of sign * M(tau_i - tau_j) onto a padded time
// grid per (b_i, b_j, r_i - r_j) label, and its transform to Matsubara frequencies.
//
// Replaces Dnfft1DGpu (dnfft_1d_gpu.hpp:38-276) whose accumulateOnDeviceKernel
// (dnfft_1d_kernels.cu:56-138) gives every (i, j, tap) a thread that recomputes its pair's grid
// position, and whose finalize copies f(tau) to the host for FFTW.  Here:
//   * a lane computes one pair's label, grid position and weight, then the warp writes the 16-tap
//     cubic convolutions (dnfft_1d.hpp:353-399, nfft_atomic_convolution.hpp:20-35) of its 32 pairs
//     two at a time, each as one 128-byte row of FP64 reductions;
//   * finalize folds the halos (dnfft_1d.hpp:401-418) and evaluates the transform only at the
//     Matsubara indices (the values transformFTauToFW, dnfft_1d.hpp:427-489, picks from its FFT),
//     divides by the window's phi(w_n) and by n, and scales by 1/Nc
//     (sp_accumulator.hpp:205-220) -- all on the device.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/dcaacc.h"
#include "common.cuh"
#include "sp_accumulator.hpp"

namespace dcaacc {

namespace {

constexpr int kOversampling = 8;
constexpr int kWindowSampling = 32;

struct NfftGrid {
  int n_padded, n, nb, nc, n_labels;
  double T0, Delta, one_div_Delta, t0_window, delta, one_div_delta, one_div_two_beta;
};

// The two spin sectors of one measurement (by value) and their vertices: tau, row orbitals
// b + nb r (right band / site), column orbitals (left band / site), packed by sector.
struct SpMeasurement {
  SpSector sector[2];
  const double* tau;
  const int* orb_r;
  const int* orb_c;
};

// Pairs (i, j) in M's memory order, 32 to a warp step: a lane reads one M element (coalesced) and
// computes its pair's label, grid position and interpolation argument; the warp then walks the 32
// pairs two at a time, lane (l & 15) of a half-warp adding tap (l & 15) + 1 to the pair's 16
// consecutive grid points with one FP64 reduction to L2 (2 x 128 contiguous bytes per warp
// instruction; no result is read back, so nothing waits on it).
//
// Bound by those reductions and the coefficient reads (L1 resident, 32 KB).  Work is split over
// pairs, not labels: a CTA per (label, spin) with the label's row in shared memory, the earlier
// form, fills 32 of the 148 SMs on a 4x4 cluster and serialises on shared-memory FP64 atomics
// (compare-and-swap loops).
// One measurement, 4x4 cluster, n 50..400: 212 -> 10 us; 6x6, n 300..1000, with squares: 657 -> 64 us.
template <bool SQR, typename Index>
__device__ inline void spAccumulateSector(const NfftGrid& g, const SpMeasurement& m, int spin, long first, long step,
                                          const int* __restrict__ r_sub, const double* __restrict__ coeff,
                                          double factor, double* __restrict__ f_tau, double* __restrict__ f_tau_sqr) {
  const SpSector sd = m.sector[spin];
  const int lane = threadIdx.x % 32;
  const Index n = sd.n, pairs = n * n;
  const double* tv = m.tau + sd.vtx_off;
  const int* orb_r = m.orb_r + sd.vtx_off;
  const int* orb_c = m.orb_c + sd.vtx_off;
  for (long grp = first; grp * 32 < static_cast<long>(pairs); grp += step) {
    const Index p = static_cast<Index>(grp) * 32 + lane;
    double f = 0, d = 0, mv = 0;
    int row = -1, t0 = 0, tab = 0;  // row < 0: nothing to add
    if (p < pairs) {
      const int j = static_cast<int>(p / n), i = static_cast<int>(p % n);
      // convoluteToFTauFineCubicInterpolation (dnfft_1d.hpp:353-399), FP64.
      const double t_val = (tv[i] - tv[j]) * g.one_div_two_beta;
      const int tau_0 = static_cast<int>((t_val - g.T0) * g.one_div_Delta);
      const double t0_val_lb = g.T0 + tau_0 * g.Delta;
      const int tau_1 = static_cast<int>((t0_val_lb - t_val - g.t0_window) * g.one_div_delta);
      const double t1_val_lb = g.t0_window + tau_1 * g.delta;
      d = t0_val_lb - t_val - t1_val_lb;
      const int dti = tau_1 - kOversampling * kWindowSampling;
      const int jw = dti % kWindowSampling;
      const int iw = (dti - jw) / kWindowSampling;
      mv = sd.M[i + static_cast<long>(sd.ldm) * j];
      f = factor * mv;
      t0 = tau_0 - kOversampling;
      tab = 4 * (iw + 4 * kOversampling * jw);
      // Out of the table only for |t_val| > 1/2, which the host rejects.
      if (jw >= 0 && iw >= -1 && iw + 2 * kOversampling < 4 * kOversampling) {
        // label = b_i + nb (b_j + nb dr), dr = index of r_i - r_j (sp_accumulator.hpp:185-191).
        const int oi = orb_r[i], oj = orb_c[j];
        const int r_i = oi / g.nb, r_j = oj / g.nb;
        row = oi - g.nb * r_i + g.nb * (oj - g.nb * r_j + g.nb * r_sub[r_j + g.nc * r_i]) + spin * g.n_labels;
      }
    }
    const int tap = (lane & 15) + 1;
#pragma unroll 4
    for (int s = 0; s < 16; ++s) {
      const int src = 2 * s + (lane >> 4);
      const double fs = __shfl_sync(0xffffffffu, f, src), ds = __shfl_sync(0xffffffffu, d, src);
      const int rs = __shfl_sync(0xffffffffu, row, src), ts = __shfl_sync(0xffffffffu, t0, src) + tap;
      const int cs = __shfl_sync(0xffffffffu, tab, src);
      double ms = 0;
      if constexpr (SQR)
        ms = __shfl_sync(0xffffffffu, mv, src);
      if (rs < 0 || ts < 0 || ts >= g.n_padded)
        continue;
      const double2* cf = reinterpret_cast<const double2*>(coeff + cs + 4 * tap);
      const double2 c01 = __ldg(cf), c23 = __ldg(cf + 1);
      const double d2 = ds * ds;
      const double w = c01.x + c01.y * ds + c23.x * d2 + c23.y * d2 * ds;
      const long o = static_cast<long>(rs) * g.n_padded + ts;
      atomicAdd(f_tau + o, fs * w);
      if constexpr (SQR)
        atomicAdd(f_tau_sqr + o, fs * ms * w);
    }
  }
}

template <bool SQR>
__global__ void __launch_bounds__(256)
spAccumulateKernel(const NfftGrid g, const SpMeasurement m, const int* __restrict__ r_sub,
                   const double* __restrict__ coeff, double factor, double* __restrict__ f_tau,
                   double* __restrict__ f_tau_sqr) {
  const long warp = (static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x) / 32;
  const long warps = static_cast<long>(gridDim.x) * blockDim.x / 32;
  for (int spin = 0; spin < 2; ++spin) {
    // The second sector's steps continue where the first sector's round ends, so that the warps
    // left over there start on it.
    const long n = m.sector[spin].n;
    const long skip = spin ? ((static_cast<long>(m.sector[0].n) * m.sector[0].n + 31) / 32) % warps : 0;
    const long first = (warp + warps - skip) % warps;
    if (n <= 65535)  // 32-bit pair indices
      spAccumulateSector<SQR, unsigned>(g, m, spin, first, warps, r_sub, coeff, factor, f_tau, f_tau_sqr);
    else
      spAccumulateSector<SQR, unsigned long long>(g, m, spin, first, warps, r_sub, coeff, factor, f_tau, f_tau_sqr);
  }
}

// f(w) = -(1/n) sum_x f(x) e^{2 pi i x nu / n} / phi(w) / Nc of the folded f, nu = 2 l + 1, and its
// conjugate at -nu.  n = 8 N (N = n_sp), so with x = a + N b
//   sum_x f(x) e^{2 pi i x nu / n} = sum_{a < N} W^{nu a} g_c(a),   W = e^{2 pi i / n},
//   g_c(a) = sum_{b < 8} f(a + N b) e^{2 pi i (2 c + 1) b / 8},     c = l mod 4:
// N terms per frequency instead of 8 N.  CTA = (label, spin, kFinL frequencies); a warp sums
// kFinU frequencies of one class c with lanes over a: nu is odd, so the lanes' table reads W^{nu a}
// fall in distinct banks.
//
// Latency and shared-memory bound.  One CTA per (label, spin) over all 8 N terms with a thread per
// frequency, the earlier form, took 1,142 us on a 4x4 cluster with N = 512; this one 20 us.
constexpr int kFinThreads = 256, kFinU = 2;
constexpr int kFinL = kFinThreads / 32 * kFinU;  // frequencies per CTA and pass
constexpr int kFinPasses = 4;                    // passes per CTA

__global__ void __launch_bounds__(kFinThreads)
spFinalizeKernel(const NfftGrid g, const double* __restrict__ f_tau, const double* __restrict__ inv_phi,
                 const double2* __restrict__ roots, int n_sp, double2* __restrict__ out) {
  extern __shared__ __align__(16) double fin_smem[];
  double2* tw = reinterpret_cast<double2*>(fin_smem);  // [8 N] W^m
  double2* gc = tw + g.n;                              // [4][N]
  const int label = blockIdx.x, spin = blockIdx.y;
  const int pad = (g.n_padded - g.n) / 2;
  const double* f = f_tau + (static_cast<long>(spin) * g.n_labels + label) * g.n_padded;
  for (int m = threadIdx.x; m < g.n; m += blockDim.x)
    tw[m] = roots[m];
  for (int a = threadIdx.x; a < n_sp; a += blockDim.x) {
    double v[8];
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      // foldTimeDomainBack: halo t < pad lands on t + n, halo t >= n_padded - pad on t - n.
      const int t = pad + a + n_sp * b;
      v[b] = f[t];
      if (t >= g.n && t - g.n < pad)
        v[b] += f[t - g.n];
      if (t + g.n >= g.n_padded - pad && t + g.n < g.n_padded)
        v[b] += f[t + g.n];
    }
    constexpr double h = 0.70710678118654752440;
    constexpr double cs[8] = {1, h, 0, -h, -1, -h, 0, h}, sn[8] = {0, h, 1, h, 0, -h, -1, -h};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      double re = 0, im = 0;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        re = fma(v[b], cs[((2 * c + 1) * b) & 7], re);
        im = fma(v[b], sn[((2 * c + 1) * b) & 7], im);
      }
      gc[c * n_sp + a] = make_double2(re, im);
    }
  }
  __syncthreads();
  const int b1 = label % g.nb, b2 = (label / g.nb) % g.nb, r = label / (g.nb * g.nb);
  const int nb = g.nb;
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  for (int pass = 0; pass < kFinPasses; ++pass) {
    // Frequencies l0 + 4 u: warps 0..3 (and 4..7, 4 kFinU further) take the four classes.
    const int l0 = (blockIdx.z * kFinPasses + pass) * kFinL + (warp / 4) * 4 * kFinU + warp % 4;
    if (l0 >= n_sp)
      break;
    double re[kFinU], im[kFinU];
    int m[kFinU], step[kFinU];
#pragma unroll
    for (int u = 0; u < kFinU; ++u) {
      const long nu = 2 * (l0 + 4 * u) + 1;
      re[u] = im[u] = 0;
      m[u] = static_cast<int>(nu * lane % g.n);
      step[u] = static_cast<int>(nu * 32 % g.n);
    }
    const double2* gl = gc + (l0 & 3) * n_sp;
    for (int a = lane; a < n_sp; a += 32) {
      const double2 x = gl[a];
#pragma unroll
      for (int u = 0; u < kFinU; ++u) {
        const double2 e = tw[m[u]];
        re[u] = fma(x.x, e.x, re[u]);
        re[u] = fma(-x.y, e.y, re[u]);
        im[u] = fma(x.x, e.y, im[u]);
        im[u] = fma(x.y, e.x, im[u]);
        m[u] += step[u];
        if (m[u] >= g.n)
          m[u] -= g.n;
      }
    }
#pragma unroll
    for (int u = 0; u < kFinU; ++u) {
#pragma unroll
      for (int s = 16; s; s /= 2) {
        re[u] += __shfl_xor_sync(0xffffffffu, re[u], s);
        im[u] += __shfl_xor_sync(0xffffffffu, im[u], s);
      }
      const int l = l0 + 4 * u;
      if (l < n_sp && lane < 2) {
        const int w = lane ? n_sp - 1 - l : n_sp + l;
        const double scale = -inv_phi[w] / (double(g.n) * g.nc);
        // (b1, s, b2, s, r, w)
        const long o = b1 + nb * (spin + 2 * (b2 + nb * (spin + 2 * (r + static_cast<long>(g.nc) * w))));
        out[o] = make_double2(re[u] * scale, (lane ? -im[u] : im[u]) * scale);
      }
    }
  }
}

__global__ void addKernel(double* __restrict__ dst, const double* __restrict__ src, size_t n) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    dst[i] += src[i];
}

// Kaiser-Bessel window, restated from kaiser_bessel_function.cpp:28-116 (n = padded size,
// m = oversampling, sigma = 2); host only, used to build the cubic table and phi(w_n).
struct KaiserBessel {
  int n, m;
  double sigma;
  double b() const {
    return M_PI * (2. - 1. / sigma);
  }
  double renorm() const {
    return 1. / (M_PI * m) * std::sinh(M_PI * m * (2. * sigma - 1.) / sigma);
  }
  double phi_t(double x) const {
    double r = 0;
    const double val = double(m) * m - double(n) * n * x * x;
    if (val > 1.e-12)
      r = 1. / M_PI * std::sinh(b() * std::sqrt(val)) / std::sqrt(val);
    if (val < -1.e-12)
      r = 1. / M_PI * std::sin(b() * std::sqrt(-val)) / std::sqrt(-val);
    if (val >= -1.e-12 && val < 1.e-12)
      r = b() / M_PI;
    return r / renorm();
  }
  double d_phi_t(double x) const {
    double r = 0;
    const double val = double(m) * m - double(n) * n * x * x;
    if (val > 1.e-12)
      r = 1. / M_PI * (double(n) * n * x) *
          ((-b() * std::cosh(b() * std::sqrt(val))) / val + std::sinh(b() * std::sqrt(val)) / std::pow(val, 1.5));
    if (val < -1.e-12)
      r = 1. / M_PI * (double(n) * n * x) *
          ((b() * std::cos(b() * std::sqrt(-val))) / (-val) - std::sin(b() * std::sqrt(-val)) / std::pow(-val, 1.5));
    if (val >= -1.e-12 && val < 1.e-12)
      return 0;
    return r / renorm();
  }
  static double besselI0(double x) {
    double result = 0., gamma = 1, y = 1.;
    const double sq = x * x / 4.;
    for (int l = 0; l < 100000; l++) {
      const double term = y / gamma;
      if (std::abs(term) < 1.e-16)
        break;
      result += term;
      gamma *= ((l + 1) * (l + 1));
      y *= sq;
    }
    return result;
  }
  double phi_wn(int wn) const {
    if (std::pow(wn, 2) < std::pow(n * (1. - 1. / (2. * sigma)), 2))
      return 1. / double(n) *
             besselI0(m * std::sqrt(std::pow(b(), 2) - std::pow((2. * M_PI * double(wn) / double(n)), 2))) /
             renorm();
    throw Error(DCAACC_INVALID_ARG, "Matsubara index outside the window's support");
  }
};

}  // namespace

struct SpAccumulator::Impl {
  NfftGrid g{};
  int n_sp = 0, max_order = 0;
  double beta = 0;
  bool sqr = false;
  bool stamping = false;
  int device = 0, n_sm = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  DevBuf<double> coeff, inv_phi, f_tau, f_tau_sqr, f_tau_single, M_d;
  DevBuf<int> r_sub_d;
  DevBuf<double2> out_d, roots;
  // A measurement's vertices, packed (tau, row orbitals, column orbitals) so that one copy uploads
  // them; the device set is reused in stream order.
  PinBuf<double> vtx_h;
  DevBuf<double> vtx_d;
  cudaEvent_t uploaded = nullptr;  // the last measurement's inputs, host M included, have been copied
  std::vector<double2> mrw, mrw_sqr;
  bool ready = false, finalized = false;
  uint64_t launches = 0;
};

SpAccumulator::SpAccumulator(const dcaacc_sp_config& c) : d_(new Impl) {
  auto& d = *d_;
  if (c.n_bands < 1 || c.n_sites < 1 || c.n_sp_freq < 1 || c.max_order < 1)
    throw Error(DCAACC_INVALID_ARG, "band, site, frequency counts and max_order must be positive");
  if (!(c.beta > 0) || !c.r_sub)
    throw Error(DCAACC_INVALID_ARG, "beta must be positive and r_sub non-null");
  const int nb = c.n_bands, nc = c.n_sites;
  d.n_sp = c.n_sp_freq;
  d.beta = c.beta;
  d.sqr = c.accumulate_m_sqr != 0;
  d.stamping = c.stamping != 0;
  d.max_order = c.max_order;
  // The index of r_i - r_j for every pair of sites; each difference once per r_j.
  const std::vector<int> r_sub(c.r_sub, c.r_sub + nc * nc);
  std::vector<char> seen(nc * nc, 0);
  for (int rj = 0; rj < nc; ++rj)
    for (int ri = 0; ri < nc; ++ri) {
      const int dr = r_sub[rj + nc * ri];
      if (dr < 0 || dr >= nc)
        throw Error(DCAACC_INVALID_ARG, "r_sub entry out of range");
      seen[rj + nc * dr] = 1;
    }
  for (char v : seen)
    if (!v)
      throw Error(DCAACC_INVALID_ARG, "r_sub is not a group subtraction table");

  // nfft_time_domain (nfft_time_domain.hpp:112-176) with MAX_FREQUENCY = n_sp.
  auto& g = d.g;
  g.nb = nb;
  g.nc = nc;
  g.n_labels = nb * nb * nc;
  g.Delta = 1. / double(kOversampling * d.n_sp);
  g.delta = 1. / double(kOversampling * d.n_sp * kWindowSampling);
  g.one_div_Delta = 1. / g.Delta;
  g.one_div_delta = 1. / g.delta;
  g.n = kOversampling * d.n_sp;
  g.n_padded = g.n + 2 * kOversampling;
  g.T0 = -0.5 - kOversampling * g.Delta;
  g.t0_window = -2. / double(d.n_sp);
  g.one_div_two_beta = 1. / (2. * c.beta);

  // Cubic interpolation table of the window (dnfft_1d.hpp:198-250), layout (4, 4*os, ws).
  const KaiserBessel kb{g.n_padded, kOversampling, 2.0};
  const int n_os = 4 * kOversampling;
  std::vector<double> cf(4 * n_os * kWindowSampling);
  auto fine_tau = [&](int idx) { return g.t0_window + idx * g.delta; };
  const double dl = fine_tau(1) - fine_tau(0);
  for (int i = 0; i < n_os; ++i)
    for (int j = 0; j < kWindowSampling; ++j) {
      const double tau = fine_tau(j + i * kWindowSampling);
      const double f0 = kb.phi_t(tau), f1 = kb.phi_t(tau + dl);
      const double df0 = kb.d_phi_t(tau), df1 = kb.d_phi_t(tau + dl);
      double* p = &cf[4 * (i + n_os * j)];
      p[0] = f0;
      p[1] = df0;
      p[2] = -(3. * f0 - 3. * f1 + 2. * df0 * dl + df1 * dl) / std::pow(dl, 2);
      p[3] = -(-2. * f0 + 2. * f1 - 1. * df0 * dl - df1 * dl) / std::pow(dl, 3);
    }
  std::vector<double> ip(2 * d.n_sp);
  for (int w = 0; w < 2 * d.n_sp; ++w) {
    const int nu = w >= d.n_sp ? 2 * (w - d.n_sp) + 1 : -(2 * (d.n_sp - 1 - w) + 1);
    ip[w] = 1.0 / kb.phi_wn(nu);
  }

  DCAACC_CUDA_CHECK(cudaGetDevice(&d.device));
  DCAACC_CUDA_CHECK(cudaDeviceGetAttribute(&d.n_sm, cudaDevAttrMultiProcessorCount, d.device));
  DCAACC_CUDA_CHECK(cudaStreamCreateWithFlags(&d.stream, cudaStreamNonBlocking));
  d.own_stream = true;
  DCAACC_CUDA_CHECK(cudaEventCreateWithFlags(&d.uploaded, cudaEventDisableTiming));
  d.coeff.alloc(cf.size());
  DCAACC_CUDA_CHECK(cudaMemcpy(d.coeff.get(), cf.data(), d.coeff.bytes(), cudaMemcpyHostToDevice));
  d.inv_phi.alloc(ip.size());
  DCAACC_CUDA_CHECK(cudaMemcpy(d.inv_phi.get(), ip.data(), d.inv_phi.bytes(), cudaMemcpyHostToDevice));
  d.r_sub_d.alloc(r_sub.size());
  DCAACC_CUDA_CHECK(cudaMemcpy(d.r_sub_d.get(), r_sub.data(), d.r_sub_d.bytes(), cudaMemcpyHostToDevice));
  std::vector<double2> roots(g.n);
  for (int m = 0; m < g.n; ++m) {
    const long double x = 2 * 3.14159265358979323846264338327950288L * m / g.n;
    roots[m] = make_double2(double(std::cos(x)), double(std::sin(x)));
  }
  d.roots.alloc(roots.size());
  DCAACC_CUDA_CHECK(cudaMemcpy(d.roots.get(), roots.data(), d.roots.bytes(), cudaMemcpyHostToDevice));
  const size_t ft = 2 * size_t(g.n_labels) * g.n_padded;
  d.f_tau.alloc(ft);
  if (d.sqr)
    d.f_tau_sqr.alloc(ft);
  if (d.stamping)
    d.f_tau_single.alloc(ft);
  const size_t nv = 2 * size_t(d.max_order);
  d.M_d.alloc(2 * size_t(d.max_order) * d.max_order);
  d.out_d.alloc(size_t(2 * nb) * (2 * nb) * nc * 2 * d.n_sp);
  d.vtx_d.alloc(2 * nv);  // per vertex one double and two ints
  d.vtx_h.alloc(2 * nv);
  DCAACC_CUDA_CHECK(cudaEventRecord(d.uploaded, d.stream));
  if (sizeof(double) * 2 * g.n_padded > 200 * 1024 || sizeof(double) * 3 * g.n > 200 * 1024)
    throw Error(DCAACC_INVALID_ARG, "n_sp_freq too large for the shared-memory NFFT rows");
}

SpAccumulator::~SpAccumulator() {
  if (d_->stream)
    cudaStreamSynchronize(d_->stream);
  if (d_->uploaded)
    cudaEventDestroy(d_->uploaded);
  if (d_->own_stream && d_->stream)
    cudaStreamDestroy(d_->stream);
}

void SpAccumulator::reset() {
  auto& d = *d_;
  DCAACC_CUDA_CHECK(cudaMemsetAsync(d.f_tau.get(), 0, d.f_tau.bytes(), d.stream));
  if (d.sqr)
    DCAACC_CUDA_CHECK(cudaMemsetAsync(d.f_tau_sqr.get(), 0, d.f_tau_sqr.bytes(), d.stream));
  if (d.stamping)
    DCAACC_CUDA_CHECK(cudaMemsetAsync(d.f_tau_single.get(), 0, d.f_tau_single.bytes(), d.stream));
  d.ready = true;
  d.finalized = false;
}

void SpAccumulator::accumulate(const dcaacc_sector* sec, double factor) {
  auto& d = *d_;
  auto& g = d.g;
  if (!d.ready)
    throw Error(DCAACC_NOT_READY, "The accumulator was not initialized.");
  if (d.finalized)
    throw Error(DCAACC_NOT_READY, "The accumulator is already finalized.");
  if (!sec)
    throw Error(DCAACC_INVALID_ARG, "null sectors");
  // One measurement's uploads in flight: the inputs of a call may be reused once the next one has returned.  The
  // uploads are behind the kernel of the measurement before theirs alone, so the GPU is not idle meanwhile.
  DCAACC_CUDA_CHECK(cudaEventSynchronize(d.uploaded));
  for (int s = 0; s < 2; ++s) {
    const auto& x = sec[s];
    if (x.n < 0 || x.n > d.max_order)
      throw Error(DCAACC_INVALID_ARG, "expansion order outside [0, max_order]");
    if (x.n && (!x.tau || !x.left_band || !x.right_band || !x.left_site || !x.right_site || !x.M ||
                x.ldm < x.n))
      throw Error(DCAACC_INVALID_ARG, "invalid sector");
    for (int i = 0; i < x.n; ++i) {
      if (x.left_band[i] < 0 || x.left_band[i] >= g.nb || x.right_band[i] < 0 || x.right_band[i] >= g.nb ||
          x.left_site[i] < 0 || x.left_site[i] >= g.nc || x.right_site[i] < 0 || x.right_site[i] >= g.nc)
        throw Error(DCAACC_INVALID_ARG, "vertex band or site out of range");
      if (!(x.tau[i] >= 0.0 && x.tau[i] <= d.beta))
        throw Error(DCAACC_INVALID_ARG, "vertex time outside [0, beta]");
    }
  }
  const int vtx = sec[0].n + sec[1].n;
  if (vtx == 0) {
    if (d.stamping)  // an empty measurement: its own f(tau) is zero
      DCAACC_CUDA_CHECK(cudaMemsetAsync(d.f_tau_single.get(), 0, d.f_tau_single.bytes(), d.stream));
    return;
  }
  double* tau = d.vtx_h.get();
  int* orb_r = reinterpret_cast<int*>(tau + vtx);
  int* orb_c = orb_r + vtx;
  SpMeasurement m{};
  m.tau = d.vtx_d.get();
  m.orb_r = reinterpret_cast<const int*>(m.tau + vtx);
  m.orb_c = m.orb_r + vtx;
  int off = 0;
  long groups = 0;
  for (int s = 0; s < 2; ++s) {
    const auto& x = sec[s];
    std::copy_n(x.tau, x.n, tau + off);
    // Rows: right band / site; columns: left band / site (sp_accumulator.hpp:181-187).
    for (int v = 0; v < x.n; ++v) {
      orb_r[off + v] = x.right_band[v] + g.nb * x.right_site[v];
      orb_c[off + v] = x.left_band[v] + g.nb * x.left_site[v];
    }
    SpSector& sd = m.sector[s];
    sd.n = x.n;
    sd.vtx_off = off;
    sd.M = x.M;
    sd.ldm = std::max(x.ldm, 1);
    if (x.n && !x.m_on_device) {
      double* dst = d.M_d.get() + size_t(s) * d.max_order * d.max_order;
      DCAACC_CUDA_CHECK(cudaMemcpy2DAsync(dst, sizeof(double) * x.n, x.M, sizeof(double) * x.ldm,
                                          sizeof(double) * x.n, x.n, cudaMemcpyHostToDevice, d.stream));
      sd.M = dst;
      sd.ldm = x.n;
    }
    off += x.n;
    groups += (long(x.n) * x.n + 31) / 32;
  }
  DCAACC_CUDA_CHECK(cudaMemcpyAsync(d.vtx_d.get(), tau, (sizeof(double) + 2 * sizeof(int)) * vtx,
                                    cudaMemcpyHostToDevice, d.stream));
  DCAACC_CUDA_CHECK(cudaEventRecord(d.uploaded, d.stream));
  // With stamping the measurement goes to its own f(tau) first, which is then added to the sum.
  double* target = d.f_tau.get();
  if (d.stamping) {
    target = d.f_tau_single.get();
    DCAACC_CUDA_CHECK(cudaMemsetAsync(target, 0, d.f_tau_single.bytes(), d.stream));
  }
  // Eight warps a CTA, eight CTAs to an SM at most: the reductions need many warps in flight.
  const unsigned blocks = static_cast<unsigned>(std::max(1L, std::min((groups + 7) / 8, long(d.n_sm) * 8)));
  if (d.sqr)
    spAccumulateKernel<true><<<blocks, 256, 0, d.stream>>>(g, m, d.r_sub_d.get(), d.coeff.get(), factor, target,
                                                           d.f_tau_sqr.get());
  else
    spAccumulateKernel<false><<<blocks, 256, 0, d.stream>>>(g, m, d.r_sub_d.get(), d.coeff.get(), factor, target,
                                                            nullptr);
  DCAACC_LAUNCH_CHECK();
  ++d.launches;
  if (d.stamping) {
    addKernel<<<d.n_sm * 4, 256, 0, d.stream>>>(d.f_tau.get(), target, d.f_tau.size());
    DCAACC_LAUNCH_CHECK();
    ++d.launches;
  }
}

void SpAccumulator::finalize() {
  auto& d = *d_;
  if (d.finalized)
    return;
  finalizeInto(d.f_tau.get(), d.mrw);
  if (d.sqr)
    finalizeInto(d.f_tau_sqr.get(), d.mrw_sqr);
  DCAACC_CUDA_CHECK(cudaStreamSynchronize(d.stream));
  d.finalized = true;
}

// Fold, DFT and window division of one f(tau) set into host memory (enqueued on the stream).
void SpAccumulator::finalizeInto(const double* f_tau, std::vector<double2>& host) {
  auto& d = *d_;
  auto& g = d.g;
  const size_t smem = sizeof(double2) * (g.n + 4 * size_t(d.n_sp));
  DCAACC_CUDA_CHECK(cudaFuncSetAttribute(spFinalizeKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  DCAACC_CUDA_CHECK(cudaMemsetAsync(d.out_d.get(), 0, d.out_d.bytes(), d.stream));
  const int splits = ceil_div(d.n_sp, kFinL * kFinPasses);
  spFinalizeKernel<<<dim3(g.n_labels, 2, splits), kFinThreads, smem, d.stream>>>(g, f_tau, d.inv_phi.get(),
                                                                                 d.roots.get(), d.n_sp, d.out_d.get());
  DCAACC_LAUNCH_CHECK();
  ++d.launches;
  host.resize(d.out_d.size());
  DCAACC_CUDA_CHECK(cudaMemcpyAsync(host.data(), d.out_d.get(), d.out_d.bytes(), cudaMemcpyDeviceToHost, d.stream));
}

void SpAccumulator::singleMeasurementMrw(double* out, size_t count) {
  auto& d = *d_;
  if (!d.stamping)
    throw Error(DCAACC_NOT_READY, "single-measurement functions need stamping");
  if (count != d.out_d.size())
    throw Error(DCAACC_INVALID_ARG, "output size does not match");
  std::vector<double2> host;
  finalizeInto(d.f_tau_single.get(), host);
  DCAACC_CUDA_CHECK(cudaStreamSynchronize(d.stream));
  std::memcpy(out, host.data(), 16 * count);
}

void SpAccumulator::singleMeasurementFtau(double* out, size_t count) {
  auto& d = *d_;
  if (!d.stamping)
    throw Error(DCAACC_NOT_READY, "single-measurement functions need stamping");
  if (count != d.f_tau_single.size())
    throw Error(DCAACC_INVALID_ARG, "output size does not match");
  DCAACC_CUDA_CHECK(cudaMemcpyAsync(out, d.f_tau_single.get(), d.f_tau_single.bytes(), cudaMemcpyDeviceToHost,
                                    d.stream));
  DCAACC_CUDA_CHECK(cudaStreamSynchronize(d.stream));
}

void SpAccumulator::clearSingleMeasurement() {
  auto& d = *d_;
  if (!d.stamping)
    throw Error(DCAACC_NOT_READY, "single-measurement functions need stamping");
  DCAACC_CUDA_CHECK(cudaMemsetAsync(d.f_tau_single.get(), 0, d.f_tau_single.bytes(), d.stream));
}

size_t SpAccumulator::fTauSize() const {
  return d_->f_tau.size();
}

void SpAccumulator::get(bool sqr, double* out, size_t count) const {
  auto& d = *d_;
  if (!d.finalized)
    throw Error(DCAACC_NOT_READY, "The accumulator was not finalized.");
  if (sqr && !d.sqr)
    throw Error(DCAACC_NOT_READY, "M squared was not accumulated.");
  const auto& v = sqr ? d.mrw_sqr : d.mrw;
  if (count != v.size())
    throw Error(DCAACC_INVALID_ARG, "output size does not match");
  std::memcpy(out, v.data(), 16 * count);
}

void SpAccumulator::sumTo(SpAccumulator& other) const {
  auto& d = *d_;
  auto& o = *other.d_;
  if (o.g.n_padded != d.g.n_padded || o.g.n_labels != d.g.n_labels || o.sqr != d.sqr)
    throw Error(DCAACC_INVALID_ARG, "accumulators have different shapes");
  DCAACC_CUDA_CHECK(cudaStreamSynchronize(d.stream));
  const int blocks = 148 * 4;
  addKernel<<<blocks, 256, 0, o.stream>>>(o.f_tau.get(), d.f_tau.get(), d.f_tau.size());
  DCAACC_LAUNCH_CHECK();
  ++o.launches;
  if (d.sqr) {
    addKernel<<<blocks, 256, 0, o.stream>>>(o.f_tau_sqr.get(), d.f_tau_sqr.get(), d.f_tau_sqr.size());
    DCAACC_LAUNCH_CHECK();
    ++o.launches;
  }
  DCAACC_CUDA_CHECK(cudaStreamSynchronize(o.stream));
}

void SpAccumulator::setStream(cudaStream_t s) {
  auto& d = *d_;
  DCAACC_CUDA_CHECK(cudaStreamSynchronize(d.stream));
  if (d.own_stream)
    DCAACC_CUDA_CHECK(cudaStreamDestroy(d.stream));
  d.own_stream = false;
  d.stream = s;
}

void SpAccumulator::synchronize() {
  DCAACC_CUDA_CHECK(cudaStreamSynchronize(d_->stream));
}

size_t SpAccumulator::deviceFingerprint() const {
  auto& d = *d_;
  return d.coeff.bytes() + d.inv_phi.bytes() + d.f_tau.bytes() + d.f_tau_sqr.bytes() + d.f_tau_single.bytes() +
         d.M_d.bytes() + d.r_sub_d.bytes() + d.vtx_d.bytes() + d.out_d.bytes() + d.roots.bytes();
}

uint64_t SpAccumulator::kernelLaunches() const {
  return d_->launches;
}

size_t SpAccumulator::outputSize() const {
  return d_->out_d.size();
}

}  // namespace dcaacc
