// Two-particle front-end: M(tau, tau') -> G(k1, w1; k2, w2) for every sector of a batch.
//
// Replaces the reference's CachedNdft<GPU>::execute (cached_ndft_gpu.hpp:131-252: sortM,
// computeT, two MAGMA vbatched GEMMs, rearrange), SpaceTransform2DGpu::execute
// (space_transform_2D_gpu.hpp:116-171: two MAGMA batched GEMMs + phaseFactorsAndRearrange) and
// computeGSingleband / computeGMultiband (tp_accumulator_kernels.cu:73-217) with three kernels:
//
//   twiddle_kernel      T(w, v) = exp(i w tau_v) over the extended frequency mesh, in both the
//                       row-sorted and column-sorted vertex orders.
//   row_transform       X'(b1 k1 w1, j) = -1/Nc sum_b G0(b1, b; k1, w1) sum_{r1} e^{i k1 (r1 + a_b)}
//                       sum_{i in orbital (b,r1)} T(w1, i) M(i, j)
//   col_transform       G(b1 k1, w1; b2 k2 w2) = sum_b [ sum_{r2} e^{-i k2 (r2 + a_b)}
//                       sum_{j in orbital (b,r2)} X'(b1 k1 w1, j) conj(T(w2, j)) ] G0(b, b2; k2, w2)
//                       + beta G0(k1,w1) delta_{k1k2} delta_{w1w2}, in frequency-block layout.
//
// Both exploit the orbital structure (each vertex belongs to one orbital, so the inner sums run
// over that orbital's vertices only, as the reference's per-orbital-pair products do) and both are
// the same two small products per CTA: the sums of a 16 x WT tile for every orbital (phase 1), then
// the cluster transform of those sums from shared memory (phase 2), so M, X' and G each cross
// global memory once per tile column.
//
// Phase 1: the orbitals are handed to the warps one by one (a shared counter).  A warp holds the
// whole 16 x WT tile, 2 x WT/4 sums a lane, and streams its orbital's vertices through a ring of
// its own in shared memory, one asynchronous 16-byte copy per lane and vertex; per vertex a lane
// reads 2 + WT/4 elements for 2 WT/4 complex multiply-adds.  Phase 2: 4 x 2 sums a lane over the
// sites, or on a 4 x 4 grid axis by axis (AxisTransform: 384 multiply-adds instead of 1,024, which were more than
// phase 1's), one (row, frequency) pair a thread.  Bound by the FP64 pipe and by latencies: a measurement is one
// partial wave of CTAs, four times as long as its FP64 operations.  The earlier kernels gave a thread one sum, that
// is two shared-memory reads per multiply-add, and a whole CTA one orbital at a time.  One measurement, 4x4,
// Nw = 64, n 100..300: row step 42 -> 17 us, 14.5 axis by axis; column step 151 -> 41, 29 axis by axis.  An FFT (14 and
// 27.5 us) would take momenta such as 2 pi m / 4 + 8 ulps for exact quarters: G off by 2e-15 instead of 8e-16.
//
// Half G (dims.half_g; mirror-symmetric inputs, a G4 kernel that reads mirrored blocks): the rows with
// w1 >= NwExt / 2 alone, in both steps: 29 -> 17 and 14.5 -> 13 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "async_copy.cuh"
#include "common.cuh"
#include "tp_frontend.hpp"

namespace dcaacc {

namespace {

// Matsubara frequency of extended index w: +-pi (2l+1) / beta, ordered as the reference's
// vertex_frequency_domain<EXTENDED> (vertex_frequency_domain.hpp EXTENDED initialize).
__device__ inline double extFrequency(int w, int nw_ext, double beta) {
  const int half = nw_ext / 2;
  if (w >= half)
    return M_PI / beta * (1 + 2 * (w - half));
  return -M_PI / beta * (1 + 2 * (half - 1 - w));
}

__global__ void twiddleKernel(const SectorDesc* __restrict__ sectors,
                              const double* __restrict__ tau,     // packed, original vertex order
                              const int* __restrict__ perm,       // packed, sorted -> original
                              double2* __restrict__ T,            // packed sorted x NwExt
                              int nw_ext, double beta) {
  const SectorDesc sd = sectors[blockIdx.y];
  const int ii = blockIdx.x;
  if (ii >= sd.n)
    return;
  const int v = perm[sd.vtx_off + ii];
  const double t = tau[sd.vtx_off + v];
  for (int w = threadIdx.x; w < nw_ext; w += blockDim.x) {
    // x = tau * w as in CachedNdft<CPU>::computeT (cached_ndft_cpu.hpp:151-156).
    const double x = t * extFrequency(w, nw_ext, beta);
    double s, c;
    sincos(x, &s, &c);
    T[static_cast<long>(sd.vtx_off + ii) * nw_ext + w] = make_double2(c, s);
  }
}

constexpr int kTileR = 16;  // rows of G (column step) or columns of M (row step) of a CTA's tile
constexpr int kRing = 8;    // vertices in flight per warp

template <int BYTES>
__device__ inline void cpAsync(void* dst, const void* src) {
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smemAddr(dst)), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smemAddr(dst)), "l"(src), "n"(BYTES) : "memory");
}
__device__ inline void cpAsyncCommit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ inline void cpAsyncWait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// z[m] := sum_a p[m][a] z[a] (SIGN < 0: with conjugated phases), the four z S apart; p[m][0] = 1.
template <int SIGN, int S>
__device__ inline void axisSums(double2* z, const double2 (&p)[4][4]) {
  const double2 in[4] = {z[0], z[S], z[2 * S], z[3 * S]};
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    double2 s = in[0];
#pragma unroll
    for (int a = 1; a < 4; ++a) {
      if (SIGN < 0)
        cfmac(s, in[a], p[m][a]);
      else
        cfma(s, in[a], p[m][a]);
    }
    z[m * S] = s;
  }
}

// Shared memory of a tile kernel: the orbitals' sums Z[o][w][16], the warps' rings (16 bytes per
// lane and slot), the phases F[b][r][k] (k padded with zeros), the orbital starts and the
// counter that hands them out.
template <int WT, int L>
struct Tile {
  static constexpr int kPairs = kTileR * WT;
  static constexpr int kSums = kPairs + (L ? 1 : 0);  // stride of an orbital's sums (L: lanes along k, distinct banks)
  static constexpr int kThreads = kPairs;
  static constexpr int kWarps = kThreads / 32;
  static_assert(kTileR + WT <= 32, "one copy per lane and vertex");
  unsigned char* ring;
  double2 *Z, *F;
  int *start, *next;

  // Phase 2 reads whole groups of momenta: 16 of one band, 8 otherwise.
  __host__ __device__ static int kPad(const TpDims& d) {
    return d.nb == 1 ? (d.nc + 15) / 16 * 16 : (d.nc + 7) / 8 * 8;
  }
  __host__ __device__ static int factors(const TpDims& d) {
    return L ? WT * L * L : d.nb * d.nc * kPad(d);
  }
  __host__ __device__ static size_t bytes(const TpDims& d) {
    return size_t(kWarps) * kRing * 512 + sizeof(double2) * (size_t(d.n_orb) * kSums + factors(d)) +
           sizeof(int) * (d.n_orb + 2);
  }
  // Lays the memory out and fills the phases (L: factor(w, k), in slot order), the starts and the counter.
  template <typename Factor>
  __device__ Tile(unsigned char* raw, const TpDims& d, const double2* __restrict__ Fb,
                  const int* __restrict__ orb_start, const AxisTransform& axes, Factor factor) {
    ring = raw;
    Z = reinterpret_cast<double2*>(raw + kWarps * kRing * 512);
    F = Z + d.n_orb * kSums;
    start = reinterpret_cast<int*>(F + factors(d));
    next = start + d.n_orb + 1;
    if constexpr (L > 0) {
      for (int i = threadIdx.x; i < WT * L * L; i += kThreads)
        F[i] = factor(i / (L * L), static_cast<int>(axes.kmap[i % (L * L)]));
    }
    else {
      const int kp = kPad(d);
      for (int i = threadIdx.x; i < d.nb * d.nc * kp; i += kThreads) {
        const int k = i % kp, r = (i / kp) % d.nc, b = i / (kp * d.nc);
        F[i] = k < d.nc ? Fb[(b * d.nc + k) * d.nc + r] : mk(0., 0.);
      }
    }
    for (int i = threadIdx.x; i <= d.n_orb; i += kThreads)
      start[i] = orb_start[i];
    if (threadIdx.x == 0)
      *next = 0;
    __syncthreads();
  }

  // Phase 1: hands the orbitals to the warps.  issue(v, slot) starts this lane's copy of vertex v into
  // a ring slot, use(slot) adds a landed slot, done(o) stores orbital o's sums and clears them.
  template <typename Issue, typename Use, typename Done>
  __device__ void orbitals(int n_orb, Issue issue, Use use, Done done) {
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    unsigned char* mine = ring + warp * kRing * 512;
    for (;;) {
      int o = 0;
      if (lane == 0)
        o = atomicAdd(next, 1);
      o = __shfl_sync(0xffffffffu, o, 0);
      if (o >= n_orb)
        break;
      const int v0 = start[o], v1 = start[o + 1];
      __syncwarp();  // every lane is done with the previous orbital's slots
#pragma unroll
      for (int p = 0; p < kRing - 1; ++p) {
        if (v0 + p < v1)
          issue(v0 + p, mine + p * 512);
        cpAsyncCommit();
      }
      int slot = 0;
      for (int v = v0; v < v1; ++v) {
        cpAsyncWait<kRing - 2>();
        __syncwarp();  // vertex v has landed for every lane, and every lane is done with vertex v - 1
        if (v + kRing - 1 < v1)
          issue(v + kRing - 1, mine + (slot == 0 ? kRing - 1 : slot - 1) * 512);
        cpAsyncCommit();
        use(mine + slot * 512);
        slot = slot == kRing - 1 ? 0 : slot + 1;
      }
      done(o);
    }
    cpAsyncWait<0>();
    __syncthreads();
  }

  // Phase 2 of one line of the tile (16 rows of frequency wl) and band b: acc[i][c] = sum_r
  // Z(b, r; wl, tr + 4 i) F(b, k0 + kl + 8 c; r), F conjugated when CONJ (tr = lane / 8, kl = lane % 8).
  template <bool CONJ, int KC>
  __device__ void clusterSum(double2 (&acc)[4][KC], const TpDims& d, int nb, int b, int wl, int k0) const {
    const int lane = threadIdx.x % 32, kp = kPad(d);
    const double2* z = Z + b * kSums + wl * kTileR + lane / 8;
    const double2* f = F + b * d.nc * kp + k0 + lane % 8;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < KC; ++c)
        acc[i][c] = mk(double(0), double(0));
#pragma unroll 2
    for (int r = 0; r < d.nc; ++r, z += nb * kSums, f += kp) {
      double2 zv[4], fv[KC];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        zv[i] = z[4 * i];
#pragma unroll
      for (int c = 0; c < KC; ++c)
        fv[c] = f[8 * c];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < KC; ++c) {
          if constexpr (CONJ)
            cfmac(acc[i][c], zv[i], fv[c]);
          else
            cfma(acc[i][c], zv[i], fv[c]);
        }
    }
  }

  // Phase 2 axis by axis (L = 4), for the 32 pairs of this warp from line wl on (two lines): the sums of site
  // (a, b) become factor times the transform e^{SIGN i k r}, element k in place of orbital k.
  template <int SIGN>
  __device__ void axisLines(const AxisTransform& axes, int wl) const {
    const int lane = threadIdx.x % 32;
    double2* p = Z + wl * kTileR + lane;
    double2 z[16];
#pragma unroll
    for (int g = 0; g < 16; ++g)
      z[g] = p[axes.rmap[g] * kSums];
#pragma unroll
    for (int b = 0; b < 4; ++b)
      axisSums<SIGN, 1>(z + 4 * b, axes.x);
#pragma unroll
    for (int m = 0; m < 4; ++m)
      axisSums<SIGN, 4>(z + m, axes.y);
    const double2* f = F + (wl + lane / kTileR) * 16;
#pragma unroll
    for (int g = 0; g < 16; ++g)
      p[axes.kmap[g] * kSums] = cmul(f[g], z[g]);
    __syncwarp();
  }
};

// Momenta of one phase 2 task: 16 of one band, or 8 with all the bands.
template <int NB>
constexpr int kTaskK = NB == 1 ? 16 : 8;

// Row transform.  grid (ceil(n_max / 16), ceil(frequencies / WT), n_sectors).  NB: bands (1, 2 or 3), 0 for
// any number.
template <int WT, int L, int NB>
__global__ void __launch_bounds__(kTileR* WT, WT == 16 ? 2 : 4)
rowTransformKernel(const TpDims dims, const SectorDesc* __restrict__ sectors,
                   const int* __restrict__ perm_r, const int* __restrict__ perm_c,
                   const int* __restrict__ row_start, const double2* __restrict__ Tr,
                   const double2* __restrict__ Fb,  // (r, k, b): e^{i k (r + a_b)}
                   const double2* __restrict__ G0,  // (b1, b2, k, w, s)
                   const __grid_constant__ AxisTransform axes, double2* __restrict__ Xp) {
  using T = Tile<WT, L>;
  const SectorDesc sd = sectors[blockIdx.z];
  // Half G: the frequencies from NwExt / 2 on.
  const int n = sd.n, j0 = blockIdx.x * kTileR, w0 = (dims.half_g ? dims.nw_ext / 2 : 0) + blockIdx.y * WT;
  if (j0 >= n)
    return;
  const int nw_ext = dims.nw_ext, R = dims.R, nb = NB ? NB : dims.nb, nc = dims.nc;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const double2* g0s = G0 + static_cast<long>(sd.spin) * nw_ext * nc * nb * nb;
  const double norm = -1.0 / nc;
  T tile(smem_raw, dims, Fb, row_start + sd.orb_off, axes, [&](int w, int k) {
    const double2 g = cmul(g0s[k + nc * min(w0 + w, nw_ext - 1)], Fb[k * nc + axes.r0]);
    return mk(norm * g.x, norm * g.y);
  });
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;

  // Phase 1: Z(o, w, j) = sum of T(w, i) M(i, j) over the vertices i of orbital o.  Lanes 0..15 copy
  // M(i, j0 + lane), the next WT lanes T(w0 + lane - 16, i); past the edge the last element, unused.
  const int* pr = perm_r + sd.vtx_off;
  const long mcol = static_cast<long>(sd.ldm) * perm_c[sd.vtx_off + min(j0 + (lane & 15), n - 1)];
  const double2* tsrc = Tr + static_cast<long>(sd.vtx_off) * nw_ext + min(w0 + lane % WT, nw_ext - 1);
  const int jl = lane % 8, wq = lane / 8;  // this lane's sums: columns jl + 8 a, frequencies wq + 4 b
  const bool f32 = sd.m_f32 != 0;
  double2 acc[2][WT / 4];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < WT / 4; ++b)
      acc[a][b] = mk(double(0), double(0));
  tile.orbitals(
      dims.n_orb,
      [&](int v, unsigned char* slot) {
        if (lane < kTileR) {
          const long e = mcol + pr[v];
          if (f32)
            cpAsync<4>(slot + 16 * lane, reinterpret_cast<const float*>(sd.M) + e);
          else
            cpAsync<8>(slot + 16 * lane, sd.M + e);
        }
        else if (lane < kTileR + WT) {
          cpAsync<16>(slot + 16 * lane, tsrc + static_cast<long>(v) * nw_ext);
        }
      },
      [&](const unsigned char* slot) {
        double m[2];
#pragma unroll
        for (int a = 0; a < 2; ++a) {
          const unsigned char* e = slot + 16 * (jl + 8 * a);
          m[a] = f32 ? static_cast<double>(*reinterpret_cast<const float*>(e))
                     : *reinterpret_cast<const double*>(e);
        }
#pragma unroll
        for (int b = 0; b < WT / 4; ++b) {
          const double2 t = *reinterpret_cast<const double2*>(slot + 16 * (kTileR + wq + 4 * b));
#pragma unroll
          for (int a = 0; a < 2; ++a) {
            acc[a][b].x = fma(t.x, m[a], acc[a][b].x);
            acc[a][b].y = fma(t.y, m[a], acc[a][b].y);
          }
        }
      },
      [&](int o) {
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < WT / 4; ++b) {
            tile.Z[o * T::kSums + (wq + 4 * b) * kTileR + jl + 8 * a] = acc[a][b];
            acc[a][b] = mk(double(0), double(0));
          }
      });

  // Phase 2: the cluster transform and the left G0, -1/Nc included.
  const long D = static_cast<long>(R) * nw_ext;
  if constexpr (L > 0) {
    for (int wl = 2 * warp; wl < WT; wl += 2 * T::kWarps) {
      tile.template axisLines<1>(axes, wl);
      const int k = lane % 16;
#pragma unroll 4
      for (int i = 0; i < kTileR; ++i) {  // two elements of the line pair a step: j = j0 + (e % 16)
        const int e = 2 * i + lane / 16, w = w0 + wl + e / kTileR, j = j0 + e % kTileR;
        if (w < nw_ext && j < n)
          Xp[sd.x_off + j * D + static_cast<long>(w) * R + k] = tile.Z[k * T::kSums + wl * kTileR + e];
      }
    }
    return;
  }
  const int k_tasks = (nc + kTaskK<NB> - 1) / kTaskK<NB>;
  for (int task = warp; task < WT * k_tasks; task += T::kWarps) {
    const int wl = task % WT, k0 = task / WT * kTaskK<NB>, w = w0 + wl;
    if (w >= nw_ext)
      continue;
    const double2* g0 = g0s + static_cast<long>(w) * nc * nb * nb;  // (ba, bb, k)
    auto put = [&](int i, int b1, int k, double2 v) {
      const int j = j0 + lane / 8 + 4 * i;
      if (j < n)
        Xp[sd.x_off + j * D + static_cast<long>(w) * R + b1 + nb * k] = v;
    };
    if constexpr (NB == 1) {
      double2 s[4][2];
      tile.template clusterSum<false, 2>(s, dims, 1, 0, wl, k0);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int k = k0 + lane % 8 + 8 * c;
        if (k >= nc)
          continue;
        const double2 g = g0[k];
        const double2 gn = mk(norm * g.x, norm * g.y);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          put(i, 0, k, cmul(gn, s[i][c]));
      }
    }
    else if constexpr (NB > 1) {
      double2 s[NB][4][1];
#pragma unroll
      for (int b = 0; b < NB; ++b)
        tile.template clusterSum<false, 1>(s[b], dims, NB, b, wl, k0);
      const int k = k0 + lane % 8;
      if (k < nc) {
#pragma unroll
        for (int b1 = 0; b1 < NB; ++b1) {
          double2 gn[NB];
#pragma unroll
          for (int b = 0; b < NB; ++b) {
            const double2 g = g0[b1 + NB * (b + NB * k)];
            gn[b] = mk(norm * g.x, norm * g.y);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            double2 v = cmul(gn[0], s[0][i][0]);
#pragma unroll
            for (int b = 1; b < NB; ++b)
              cfma(v, gn[b], s[b][i][0]);
            put(i, b1, k, v);
          }
        }
      }
    }
    else {
      const int k = k0 + lane % 8;
      for (int b1 = 0; b1 < nb; ++b1) {
        double2 v[4] = {};
        for (int b = 0; b < nb; ++b) {
          double2 s[4][1];
          tile.template clusterSum<false, 1>(s, dims, nb, b, wl, k0);
          const double2 g = g0[b1 + nb * (b + nb * min(k, nc - 1))];
          const double2 gn = mk(norm * g.x, norm * g.y);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            cfma(v[i], gn, s[i][0]);
        }
        if (k < nc)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            put(i, b1, k, v[i]);
      }
    }
  }
}

// Column transform + G epilogue.  grid (ceil(rows / 16), ceil(NwExt / WT), n_sectors); the rows of a tile
// are 16 consecutive (w1, r), with half G those from D / 2 on.
template <int WT, int L, int NB>
__global__ void __launch_bounds__(kTileR* WT, WT == 16 ? 2 : 4)
colTransformKernel(const TpDims dims, const SectorDesc* __restrict__ sectors,
                   const int* __restrict__ col_start, const double2* __restrict__ Tc,
                   const double2* __restrict__ Fb,
                   const double2* __restrict__ G0,  // (b1, b2, k, w, s)
                   const __grid_constant__ AxisTransform axes, const double2* __restrict__ Xp, double2* __restrict__ G,
                   long g_sector_stride) {
  using T = Tile<WT, L>;
  const SectorDesc sd = sectors[blockIdx.z];
  const int nw_ext = dims.nw_ext, R = dims.R, nb = NB ? NB : dims.nb, nc = dims.nc;
  const int D = R * nw_ext, row0 = (dims.half_g ? D / 2 : 0) + blockIdx.x * kTileR, w0 = blockIdx.y * WT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const double2* g0s = G0 + static_cast<long>(sd.spin) * nw_ext * nc * nb * nb;
  T tile(smem_raw, dims, Fb, col_start + sd.orb_off, axes,
         [&](int w, int k) { return cmulc(g0s[k + nc * min(w0 + w, nw_ext - 1)], Fb[k * nc + axes.r0]); });
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;

  // Phase 1: Z(o, w2, row) = sum of X'(row, j) conj T(w2, j) over the vertices j of orbital o.
  const double2* xsrc = Xp + sd.x_off + min(row0 + (lane & 15), D - 1);
  const double2* tsrc = Tc + static_cast<long>(sd.vtx_off) * nw_ext + min(w0 + lane % WT, nw_ext - 1);
  const int rl = lane % 8, wq = lane / 8;  // this lane's sums: rows rl + 8 a, frequencies wq + 4 b
  double2 acc[2][WT / 4];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < WT / 4; ++b)
      acc[a][b] = mk(double(0), double(0));
  tile.orbitals(
      dims.n_orb,
      [&](int v, unsigned char* slot) {
        if (lane < kTileR)
          cpAsync<sizeof(double2)>(slot + 16 * lane, xsrc + static_cast<long>(v) * D);
        else if (lane < kTileR + WT)
          cpAsync<16>(slot + 16 * lane, tsrc + static_cast<long>(v) * nw_ext);
      },
      [&](const unsigned char* slot) {
        double2 x[2];
#pragma unroll
        for (int a = 0; a < 2; ++a)
          x[a] = *reinterpret_cast<const double2*>(slot + 16 * (rl + 8 * a));
#pragma unroll
        for (int b = 0; b < WT / 4; ++b) {
          const double2 t = *reinterpret_cast<const double2*>(slot + 16 * (kTileR + wq + 4 * b));
#pragma unroll
          for (int a = 0; a < 2; ++a)
            cfmac(acc[a][b], x[a], t);
        }
      },
      [&](int o) {
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < WT / 4; ++b) {
            tile.Z[o * T::kSums + (wq + 4 * b) * kTileR + rl + 8 * a] = acc[a][b];
            acc[a][b] = mk(double(0), double(0));
          }
      });

  // Phase 2: the cluster transform with conjugate phases, the right G0 and the delta term.
  const double beta = dims.beta;
  double2* out = G + g_sector_stride * (2 * sd.slot + sd.spin);
  if constexpr (L > 0) {
    for (int wl = 2 * warp; wl < WT; wl += 2 * T::kWarps) {
      tile.template axisLines<-1>(axes, wl);
      const int k = lane % 16;
#pragma unroll 4
      for (int i = 0; i < kTileR; ++i) {
        const int e = 2 * i + lane / 16, w2 = w0 + wl + e / kTileR, row = row0 + e % kTileR;
        if (w2 >= nw_ext || row >= D)
          continue;
        const int w1 = row / 16, r = row % 16;
        double2 v = tile.Z[k * T::kSums + wl * kTileR + e];
        if (w1 == w2 && r == k) {
          const double2 dl = g0s[k + nc * w2];
          v.x = fma(beta, dl.x, v.x);
          v.y = fma(beta, dl.y, v.y);
        }
        out[((static_cast<long>(w1) * nw_ext + w2) * 16 + r) * 16 + k] = v;
      }
    }
    return;
  }
  const int k_tasks = (nc + kTaskK<NB> - 1) / kTaskK<NB>;
  for (int task = warp; task < WT * k_tasks; task += T::kWarps) {
    const int wl = task % WT, k0 = task / WT * kTaskK<NB>, w2 = w0 + wl;
    if (w2 >= nw_ext)
      continue;
    const double2* g0 = g0s + static_cast<long>(w2) * nc * nb * nb;  // (ba, bb, k)
    // G(row, w2; b2 k2) += beta G0 on the diagonal, and its store (rows past the edge are dropped).
    auto put = [&](int i, int b2, int k2, double2 v) {
      const int row = row0 + lane / 8 + 4 * i;
      if (row >= D)
        return;
      const int w1 = row / R, r = row - w1 * R, k1 = r / nb;
      if (w1 == w2 && k1 == k2) {
        const double2 dl = g0[(r - nb * k1) + nb * (b2 + nb * k2)];
        v.x = fma(beta, dl.x, v.x);
        v.y = fma(beta, dl.y, v.y);
      }
      out[((static_cast<long>(w1) * nw_ext + w2) * R + r) * R + b2 + nb * k2] = v;
    };
    if constexpr (NB == 1) {
      double2 s[4][2];
      tile.template clusterSum<true, 2>(s, dims, 1, 0, wl, k0);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int k = k0 + lane % 8 + 8 * c;
        if (k >= nc)
          continue;
        const double2 g = g0[k];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          put(i, 0, k, cmul(s[i][c], g));
      }
    }
    else if constexpr (NB > 1) {
      double2 s[NB][4][1];
#pragma unroll
      for (int b = 0; b < NB; ++b)
        tile.template clusterSum<true, 1>(s[b], dims, NB, b, wl, k0);
      const int k = k0 + lane % 8;
      if (k < nc) {
#pragma unroll
        for (int b2 = 0; b2 < NB; ++b2) {
          double2 g[NB];
#pragma unroll
          for (int b = 0; b < NB; ++b)
            g[b] = g0[b + NB * (b2 + NB * k)];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            double2 v = cmul(s[0][i][0], g[0]);
#pragma unroll
            for (int b = 1; b < NB; ++b)
              cfma(v, s[b][i][0], g[b]);
            put(i, b2, k, v);
          }
        }
      }
    }
    else {
      const int k = k0 + lane % 8;
      for (int b2 = 0; b2 < nb; ++b2) {
        double2 v[4] = {};
        for (int b = 0; b < nb; ++b) {
          double2 s[4][1];
          tile.template clusterSum<true, 1>(s, dims, nb, b, wl, k0);
          const double2 g = g0[b + nb * (b2 + nb * min(k, nc - 1))];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            cfma(v[i], s[i][0], g);
        }
        if (k < nc)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            put(i, b2, k, v[i]);
      }
    }
  }
}

}  // namespace

// ------------------------------------------------------------------------------------------------
// Host launchers
// ------------------------------------------------------------------------------------------------
AxisTransform clusterAxes4(int nb, int nc, const double* r_vecs, const double* k_vecs) {
  AxisTransform t{};
  if (nb != 1 || nc != 16)
    return t;
  // The place of each vector on a grid of four values an axis, the sites' with 0 first: map[i + 4 j].
  auto grid = [](const double* v, bool zero_first, double (&axis)[2][4], unsigned char* map) {
    int used = 0, count[2] = {0, 0};
    if (zero_first) {
      axis[0][0] = axis[1][0] = 0;
      count[0] = count[1] = 1;
    }
    for (int i = 0; i < 16; ++i) {
      int at[2];
      for (int c = 0; c < 2; ++c) {
        const double x = v[2 * i + c];
        int j = 0;
        while (j < count[c] && axis[c][j] != x)
          ++j;
        if (j == 4 || x != x)
          return false;
        if (j == count[c])
          axis[c][count[c]++] = x;
        at[c] = j;
      }
      const int g = at[0] + 4 * at[1];
      if (used & (1 << g))
        return false;
      used |= 1 << g;
      map[g] = static_cast<unsigned char>(i);
    }
    return true;  // sixteen different places: all of them
  };
  double r[2][4], k[2][4];
  if (!grid(r_vecs, true, r, t.rmap) || !grid(k_vecs, false, k, t.kmap))
    return t;
  for (int m = 0; m < 4; ++m)
    for (int a = 0; a < 4; ++a) {
      t.x[m][a] = mk(std::cos(k[0][m] * r[0][a]), std::sin(k[0][m] * r[0][a]));
      t.y[m][a] = mk(std::cos(k[1][m] * r[1][a]), std::sin(k[1][m] * r[1][a]));
    }
  t.r0 = t.rmap[0];
  t.on = 1;
  return t;
}

void launchTwiddles(const FrontendArgs& a, cudaStream_t stream) {
  const dim3 grid(a.n_max, a.n_sectors);
  twiddleKernel<<<grid, 128, 0, stream>>>(a.sectors, a.tau, a.perm_r, a.Tr, a.dims.nw_ext, a.dims.beta);
  DCAACC_LAUNCH_CHECK();
  if (a.Tc != a.Tr) {
    twiddleKernel<<<grid, 128, 0, stream>>>(a.sectors, a.tau, a.perm_c, a.Tc, a.dims.nw_ext, a.dims.beta);
    DCAACC_LAUNCH_CHECK();
  }
}

// Which clusters the FP64 and the all-SIMT front-end take, whatever the orders: 4 KB (FP64) an orbital for 32 x 8
// tiles, the phases, and R x R blocks of a few column frequencies within 227 KB.  The kernels' own tiles (Tile,
// Tile32) are smaller, so that what passes fits.
size_t frontendSmemRequirement(const TpDims& d, bool fp64) {
  const size_t real = fp64 ? sizeof(double) : sizeof(float), cplx = 2 * real;
  const size_t R = d.R, orb = d.n_orb, phases = size_t(d.nb) * d.nc * d.nc;
  const size_t row = cplx * (256 * orb + phases + 512) + real * 32 * 65 + sizeof(int) * (orb + 1);
  size_t wc = 16;
  while (wc > 1 && (R * wc > 1024 || cplx * (R * R * wc + R * (R + 1) * wc) > 96 * 1024))
    wc /= 2;
  const size_t col = cplx * (std::max(R * wc * orb, wc * R * (R + 1)) + R * wc * R + phases + 64 * (R + wc)) +
                     sizeof(int) * (orb + 1);
  return std::max(row, col);
}

static bool axes4(const FrontendArgs& a) {
  return a.dims.nb == 1 && a.axes.on;
}

// Frequencies per CTA, 16 or 8, which the tuner chooses between: every element is the same sum in the
// same order either way.  8 alone where 16 does not fit in shared memory.
static int tileWidth(const FrontendArgs& a, const char* family, LaunchTuner::Pick& pk, cudaStream_t stream) {
  const bool wide = (axes4(a) ? Tile<16, 4>::bytes(a.dims) : Tile<16, 0>::bytes(a.dims)) <= 227 * 1024;
  pk = tunePick(a.tuner, tuneKey(family, a.dims.nb, a.dims.nc, a.dims.nw_ext, a.n_max, a.n_sectors, 8),
                wide ? 2 : 1, stream);
  return wide && pk.choice == 0 ? 16 : 8;
}

template <int WT, int L, typename Kernel, typename... Args>
static void launchTile(Kernel k, const TpDims& d, int tiles, int freqs, int sectors, cudaStream_t stream, Args... args) {
  const size_t smem = Tile<WT, L>::bytes(d);
  DCAACC_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  DCAACC_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         int(cudaSharedmemCarveoutMaxShared)));
  k<<<dim3(tiles, ceil_div(freqs, WT), sectors), Tile<WT, L>::kThreads, smem, stream>>>(d, args...);
  DCAACC_LAUNCH_CHECK();
}

template <int WT>
static void launchRowWT(const FrontendArgs& a, double2* Xp, cudaStream_t stream) {
  const int nb = a.dims.nb, tiles = ceil_div(a.n_max, kTileR), freqs = a.dims.nw_ext / (a.dims.half_g ? 2 : 1);
  if (axes4(a)) {
    launchTile<WT, 4>(rowTransformKernel<WT, 4, 1>, a.dims, tiles, freqs, a.n_sectors, stream, a.sectors, a.perm_r, a.perm_c,
                      a.row_start, a.Tr, a.Fb, a.G0, a.axes, Xp);
    return;
  }
  auto k = nb == 1   ? rowTransformKernel<WT, 0, 1>
           : nb == 2 ? rowTransformKernel<WT, 0, 2>
           : nb == 3 ? rowTransformKernel<WT, 0, 3> : rowTransformKernel<WT, 0, 0>;
  launchTile<WT, 0>(k, a.dims, tiles, freqs, a.n_sectors, stream, a.sectors, a.perm_r, a.perm_c, a.row_start, a.Tr, a.Fb, a.G0,
                    a.axes, Xp);
}

void launchRowTransform(const FrontendArgs& a, double2* Xp, cudaStream_t stream) {
  if (a.n_max == 0)
    return;
  LaunchTuner::Pick pk;
  if (tileWidth(a, "row", pk, stream) == 16)
    launchRowWT<16>(a, Xp, stream);
  else
    launchRowWT<8>(a, Xp, stream);
  tuneEnd(a.tuner, pk, stream);
}

template <int WT>
static void launchColWT(const FrontendArgs& a, const double2* Xp, double2* G, long g_sector_stride, cudaStream_t stream) {
  const int nb = a.dims.nb, freqs = a.dims.nw_ext;
  const int tiles = ceil_div(long(a.dims.R) * freqs / (a.dims.half_g ? 2 : 1), kTileR);
  if (axes4(a)) {
    launchTile<WT, 4>(colTransformKernel<WT, 4, 1>, a.dims, tiles, freqs, a.n_sectors, stream, a.sectors, a.col_start, a.Tc, a.Fb,
                      a.G0, a.axes, Xp, G, g_sector_stride);
    return;
  }
  auto k = nb == 1   ? colTransformKernel<WT, 0, 1>
           : nb == 2 ? colTransformKernel<WT, 0, 2>
           : nb == 3 ? colTransformKernel<WT, 0, 3> : colTransformKernel<WT, 0, 0>;
  launchTile<WT, 0>(k, a.dims, tiles, freqs, a.n_sectors, stream, a.sectors, a.col_start, a.Tc, a.Fb, a.G0, a.axes, Xp, G,
                    g_sector_stride);
}

void launchColTransform(const FrontendArgs& a, const double2* Xp, double2* G,
                        long g_sector_stride, cudaStream_t stream) {
  LaunchTuner::Pick pk;
  if (tileWidth(a, "col", pk, stream) == 16)
    launchColWT<16>(a, Xp, G, g_sector_stride, stream);
  else
    launchColWT<8>(a, Xp, G, g_sector_stride, stream);
  tuneEnd(a.tuner, pk, stream);
}

}  // namespace dcaacc
