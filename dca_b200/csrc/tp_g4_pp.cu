// Particle-particle up-down update of a multiband model, mixed path (FP32 G, FP32 batch sums).
//
// Channel PARTICLE_PARTICLE_UP_DOWN (tp_accumulator_cpu.hpp:628-661, updateG4Kernel's PP branch in
// tp_accumulator_kernels.cu):
//   G4(k1, w1, k2, w2, q, wq; b1, b2, b3, b4) += s/2 sum_sigma G_sigma(k1, w1; k2, w2)[b1, b3]
//                                               x G_-sigma(q - k1, m1; q - k2, m2)[b2, b4],
//   m = wq + Nw - 1 - w.
// For fixed (k1, k2, q, w1, w2, wq) the nb^4 entries are a sum of Kronecker products of two nb x nb
// band blocks.  A thread owns one (k1, k2, q, b4) and keeps the nb^3 entries (b1, b2, b3) in
// registers for the whole batch: per measurement and spin it reads nb^2 elements of the A block
// G(w1; w2) and nb of the P block G(m1; m2) and does nb^3 complex FMAs (27 per 12 reads for three
// bands), where the generic staged kernel (tp_g4.cu) reads two elements per entry.  CTA = one
// (w1, w2, wq) tile; per measurement the two spins' A and P blocks (R x R each, R = nb Nc) arrive in
// shared memory by the bulk-copy engine, two measurements a stage, through a three-stage ring.  Items (k1, k2, q, b4) are
// numbered q fastest, then k2, so that the A reads of a warp are broadcasts; items beyond the
// CTA's threads take further passes over the batch.  The batch sum of each entry goes into the
// FP64 running sum with one read-modify-write, as in the staged kernel, spread over the next pass and in
// G4's order: for fixed (k2, q) the entries of a pass's items are one run of G4, so a pass's sums are
// exchanged through shared memory and consecutive lanes take consecutive entries.  The band indices follow its G layout (element (b3, k1; b1, k2) of the A block, (b4, q - k1;
// b2, q - k2) of the P block).
//
// Bound by the FP32 pipe's multiply-adds (45 % of its cycles, 46 % of the issue slots; sixteen warps of 128
// registers hide only part of the shared-memory and G4 latencies).  They are packed pairs, at half the scalar
// ones' issue slots.  8 sites, three bands, Nw = 16, all transfers, four frequency transfers, a batch of 32: 1.23 ms
// with scalar multiply-adds, 1.18 packed, 0.83 with G4 read and written in runs and two measurements a stage.
#include <cuda_runtime.h>

#include <type_traits>

#include "async_copy.cuh"
#include "common.cuh"
#include "packed.cuh"
#include "tp_g4.hpp"
#include "tp_layout.hpp"

namespace dcaacc {

namespace {

constexpr int kPPThreads = 512;
constexpr int kPPStages = 3;  // ring of block sets: copies run two steps ahead
constexpr int kPPMeas = 2;    // measurements per stage
constexpr int kPPPending = 6;  // ints of the pending pass
constexpr int kPPPitch = kPPThreads + 1;  // row of the batch sums in shared memory (distinct banks along the entries)

template <int NB, int NC>
__global__ void __launch_bounds__(kPPThreads, 1)
updateG4PPMultibandKernel(const TpDims dims, const float2* __restrict__ G, long g_sector_stride,
                          const int* __restrict__ signs, int n_slots, const int* __restrict__ k_sub,
                          const int* __restrict__ q_list, const int* __restrict__ wex_list,
                          double2* const* __restrict__ G4, bool atomic, int* __restrict__ err, uint32_t wait_limit) {
  constexpr int NB2 = NB * NB, NB3 = NB2 * NB, NB4 = NB3 * NB;
  constexpr int nc = NC, R = NB * NC;  // compile-time block shape: the band offsets are immediates
  const int nw = dims.nw, nw_ext = dims.nw_ext, nq = dims.nq, ext = dims.ext;
  // wq fastest: the CTAs that read the same A block G(w1; w2) run side by side (one L2 fetch).
  const int iwq = blockIdx.x, w2 = blockIdx.y, w1 = blockIdx.z;
  const int wex = wex_list[iwq];
  constexpr long blk = static_cast<long>(R) * R;
  const int n_items = nc * nc * nq * NB;
  const int n_passes = (n_items + kPPThreads - 1) / kPPThreads;
  const int pass_steps = (n_slots + kPPMeas - 1) / kPPMeas;
  const int n_steps = n_passes * pass_steps;
  const int m1 = wex + nw - 1 - w1 + ext, m2 = wex + nw - 1 - w2 + ext;
  const long offA = (static_cast<long>(w1 + ext) * nw_ext + w2 + ext) * blk;
  const long offP = (static_cast<long>(m1) * nw_ext + m2) * blk;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw);     // [kPPStages] a stage's copies landed
  uint64_t* empty = bar + kPPStages;                         // [kPPStages] every warp is done with it
  float2* stage = reinterpret_cast<float2*>(smem_raw + 64);  // [kPPStages][kPPMeas][spin][A, P][R * R]
  const uint32_t blk_bytes = static_cast<uint32_t>(blk * sizeof(float2));
  auto issue = [&](int step) {
    const int st = step % kPPStages;
    const int m0 = step % pass_steps * kPPMeas, n = min(kPPMeas, n_slots - m0);
    mbarArriveExpectTx(&bar[st], n * 4 * blk_bytes);
    for (int m = 0; m < n; ++m)
      for (int s = 0; s < 2; ++s) {
        float2* dst = stage + ((st * kPPMeas + m) * 4 + 2 * s) * blk;
        const float2* src = G + g_sector_stride * (2 * (m0 + m) + s);
        bulkCopyG2S(dst, src + offA, blk_bytes, &bar[st]);
        bulkCopyG2S(dst + blk, src + offP, blk_bytes, &bar[st]);
      }
  };
  const int t = threadIdx.x;
  const int lane = t % 32;
  if (t == 0) {
    for (int i = 0; i < kPPStages; ++i) {
      mbarInit(&bar[i], 1);
      mbarInit(&empty[i], kPPThreads / 32);
    }
    fenceBarrierInit();
  }
  __syncthreads();
  if (t == 0)
    for (int i = 0; i < kPPStages && i < n_steps; ++i)
      issue(i);

  // G4 strides: entry (b1, b2, b3, b4) + nb^4 (k1 + Nc (w1 + Nw (k2 + Nc (w2 + Nw (q + Nq wq))))).
  const long s_w1 = static_cast<long>(NB4) * nc, s_k2 = s_w1 * nw, s_w2 = s_k2 * nc, s_q = s_w2 * nw,
             s_wq = s_q * nq;
  double2* g4t = G4[0] + w1 * s_w1 + w2 * s_w2 + iwq * s_wq;
  const uint32_t limit = wait_limit ? wait_limit : kWaitLimit;
  // A pass's batch sums wait in shared memory ([entry of an item][item]) and go into the FP64 running sum
  // one entry a thread per measurement of the next pass, so that the read-modify-write latency hides
  // behind that measurement's FMAs (the last pass's sums go at the end).  In G4, the entries of (b4, k1)
  // follow one another for fixed (k2, q): entry j of run r, r = q + Nq k2, j = b + nb^3 (item / (Nq Nc) - bk0).
  float2* fb = stage + kPPStages * kPPMeas * 4 * blk;
  const int n_runs = nq * nc;
  long* run_off = reinterpret_cast<long*>(fb + NB3 * kPPPitch + (NB3 * kPPPitch) % 2);  // [n_runs]
  int* pend_mem = reinterpret_cast<int*>(run_off + n_runs);                // [kPPPending]
  signed char* sgn = reinterpret_cast<signed char*>(pend_mem + kPPPending);  // [n_slots] the measurements' signs
  for (int i = t; i < n_slots; i += kPPThreads)
    sgn[i] = static_cast<signed char>(signs[i]);
  for (int r = t; r < n_runs; r += kPPThreads)
    run_off[r] = r / nq * s_k2 + r % nq * s_q;
  __syncthreads();  // the signs are in place before any warp's first step
  // The pending pass: offset of an item's place from its (b4, k1) and run, number of items, first (b4, k1), run
  // length, and a thread's step from one of its entries to the next one.
  struct Pending {
    int place, count, bk0, run, dr, dj;
  };
  auto pendingOf = [&](int pass) {
    Pending p;
    const int item0 = kPPThreads * pass;
    p.count = min(kPPThreads, n_items - item0);
    p.bk0 = item0 / n_runs;
    p.place = p.bk0 * n_runs - item0;
    p.run = NB3 * ((item0 + p.count - 1) / n_runs - p.bk0 + 1);
    p.dr = kPPThreads / p.run;
    p.dj = kPPThreads - p.dr * p.run;
    return p;
  };
  static_assert(sizeof(Pending) == kPPPending * sizeof(int), "its place in shared memory");
  volatile Pending* pend = reinterpret_cast<volatile Pending*>(pend_mem);  // in shared memory: registers are short
  int fr = n_runs, fj = 0;  // this thread's next entry
  auto flushEntry = [&](double2* dst, float2 v, double2 old) {
    if (atomic) {
      atomicAdd(&dst->x, static_cast<double>(v.x));
      atomicAdd(&dst->y, static_cast<double>(v.y));
    }
    else {
      old.x += static_cast<double>(v.x);
      old.y += static_cast<double>(v.y);
      *dst = old;
    }
  };
  // The next pending entry of this thread: its place in G4 (null: not of this pass) and its sum.
  auto nextEntry = [&](float2& v) -> double2* {
    const int kb = fj / NB3, place = kb * n_runs + fr + pend->place;
    double2* dst = nullptr;
    if (place >= 0 && place < pend->count) {
      v = fb[(fj - NB3 * kb) * kPPPitch + place];
      dst = g4t + run_off[fr] + NB3 * pend->bk0 + fj;
    }
    fr += pend->dr;
    fj += pend->dj;
    if (fj >= pend->run) {
      fj -= pend->run;
      ++fr;
    }
    return dst;
  };
  auto flushRest = [&](auto in_flight) {
    constexpr int kRest = decltype(in_flight)::value;  // entries
    while (fr < n_runs) {
      double2* dst[kRest];
      float2 v[kRest];
      double2 old[kRest];
#pragma unroll
      for (int u = 0; u < kRest; ++u) {
        dst[u] = fr < n_runs ? nextEntry(v[u]) : nullptr;
        if (dst[u] && !atomic)
          old[u] = *dst[u];
      }
#pragma unroll
      for (int u = 0; u < kRest; ++u)
        if (dst[u])
          flushEntry(dst[u], v[u], old[u]);
    }
  };
  int step = 0, st = 0;
  uint32_t phase = 0;
  bool ok = true;
  for (int pass = 0; pass < n_passes; ++pass) {
    const int item = t + kPPThreads * pass;
    const bool live = item < n_items;
    const int it = live ? item : 0;
    const int iq = it % nq, k2 = (it / nq) % nc, b4 = (it / (nq * nc)) % NB, k1 = it / (nq * nc * NB);
    const int q = q_list[iq];
    const int qk1 = k_sub[k1 + nc * q], qk2 = k_sub[k2 + nc * q];
    const int aoff = NB * k1 * R + NB * k2;          // element (b1, b3) at + b3 R + b1
    const int poff = (b4 + NB * qk1) * R + NB * qk2;  // element b2 at + b2
    Pair acc[NB][NB][NB];  // [b1][b2][b3]
#pragma unroll
    for (int b1 = 0; b1 < NB; ++b1)
#pragma unroll
      for (int b2 = 0; b2 < NB; ++b2)
#pragma unroll
        for (int b3 = 0; b3 < NB; ++b3)
          acc[b1][b2][b3] = 0;

    // One measurement; one pending entry of the previous pass is read before it and written after it.
    auto measure = [&](const float2* A0, int sign) {
      double2* fdst = nullptr;
      float2 fv = make_float2(0.f, 0.f);
      double2 fold = make_double2(0., 0.);
      if (fr < n_runs) {
        fdst = nextEntry(fv);
        if (fdst && !atomic)
          fold = *fdst;
      }
      const float2* P0 = A0 + blk;
      const float2* A1 = A0 + 2 * blk;
      const float2* P1 = A0 + 3 * blk;
      if (live) {
        const float hs = 0.5f * static_cast<float>(sign);
        // s/2 P_sigma(b4, q - k1; b2, q - k2), its parts doubled: a p = (ax, ay) px + (-ay, ax) py.
        Pair p0x[NB], p0y[NB], p1x[NB], p1y[NB];
#pragma unroll
        for (int b2 = 0; b2 < NB; ++b2) {
          const float2 x0 = P0[poff + b2], x1 = P1[poff + b2];
          p0x[b2] = pairOf(hs * x0.x, hs * x0.x);
          p0y[b2] = pairOf(hs * x0.y, hs * x0.y);
          p1x[b2] = pairOf(hs * x1.x, hs * x1.x);
          p1y[b2] = pairOf(hs * x1.y, hs * x1.y);
        }
#pragma unroll
        for (int b3 = 0; b3 < NB; ++b3)
#pragma unroll
          for (int b1 = 0; b1 < NB; ++b1) {
            const float2 a0 = A0[aoff + b3 * R + b1], a1 = A1[aoff + b3 * R + b1];
            const Pair a00 = pairOf(a0.x, a0.y), a01 = pairOf(-a0.y, a0.x);
            const Pair a10 = pairOf(a1.x, a1.y), a11 = pairOf(-a1.y, a1.x);
#pragma unroll
            for (int b2 = 0; b2 < NB; ++b2) {
              Pair& c = acc[b1][b2][b3];
              fma2(c, a00, p1x[b2]);
              fma2(c, a01, p1y[b2]);
              fma2(c, a10, p0x[b2]);
              fma2(c, a11, p0y[b2]);
            }
          }
      }
      if (fdst)
        flushEntry(fdst, fv, fold);
    };
    for (int slot = 0; slot < n_slots; slot += kPPMeas, ++step) {
      ok = __all_sync(0xffffffffu, ok && mbarWait(&bar[st], phase, err, limit));
      if (!ok)
        break;
      const float2* S = stage + st * (kPPMeas * 4 * blk);
#pragma unroll 1
      for (int m = 0; m < kPPMeas && slot + m < n_slots; ++m)
        measure(S + m * 4 * blk, sgn[slot + m]);
      __syncwarp();
      if (lane == 0)
        mbarArrive(&empty[st]);  // release: this warp's reads of the stage are done
      if (t == 0 && step + kPPStages < n_steps) {
        // Out of time: the vote above ends this warp's loop, the others time out on the missing copies.
        ok = mbarWait(&empty[st], phase, err, limit);
        if (ok) {
          fenceProxyAsync();
          issue(step + kPPStages);
        }
      }
      if (++st == kPPStages) {
        st = 0;
        phase ^= 1;
      }
    }
    if (__syncthreads_or(!ok))
      return;  // uniform bail-out; the host reports the error word
    flushRest(std::integral_constant<int, 2>{});  // batches shorter than the entries a thread leave some of the previous pass
    __syncthreads();
    if (live) {
#pragma unroll
      for (int b3 = 0; b3 < NB; ++b3)
#pragma unroll
        for (int b2 = 0; b2 < NB; ++b2)
#pragma unroll
          for (int b1 = 0; b1 < NB; ++b1)
            fb[(b1 + NB * b2 + NB2 * b3) * kPPPitch + t] = floatsOf(acc[b1][b2][b3]);
    }
    if (t == 0) {
      const Pending p = pendingOf(pass);
      pend->place = p.place;
      pend->count = p.count;
      pend->bk0 = p.bk0;
      pend->run = p.run;
      pend->dr = p.dr;
      pend->dj = p.dj;
    }
    __syncthreads();
    fr = t / pend->run;
    fj = t - fr * pend->run;
  }
  flushRest(std::integral_constant<int, 9>{});
}

}  // namespace

bool launchUpdateG4PPMultiband(const G4Args& a, const float2* G, long g_sector_stride, cudaStream_t stream) {
  const TpDims& d = a.dims;
  if (d.n_channels != 1 || d.channels[0] != 4 /* PARTICLE_PARTICLE_UP_DOWN */ || d.nb != 3 || d.half_g4 || d.half_g ||
      a.n_slots < 1 || (d.nc != 4 && d.nc != 8))
    return false;
  const size_t smem = 64 + kPPStages * kPPMeas * 4 * size_t(d.R) * d.R * sizeof(float2) +
                      (27 * size_t(kPPPitch) + 1) * sizeof(float2) + sizeof(long) * size_t(d.nq) * d.nc +
                      sizeof(int) * kPPPending + size_t(a.n_slots);
  if (smem > 227 * 1024)
    return false;
  auto k = d.nc == 4 ? updateG4PPMultibandKernel<3, 4> : updateG4PPMultibandKernel<3, 8>;
  DCAACC_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  const dim3 grid(d.nwq, d.nw, d.nw);
  k<<<grid, kPPThreads, smem, stream>>>(d, G, g_sector_stride, a.signs, a.n_slots, a.k_sub, a.q_list, a.wex_list,
                                         a.G4, a.atomic, a.err, a.wait_limit);
  DCAACC_LAUNCH_CHECK();
  return true;
}

}  // namespace dcaacc
