// Direct term of the batched single-band G4 update on the tensor cores for 6 x 6 clusters (all momentum
// transfers, PH-magnetic / PH-charge): tp_g4_mma.cu's products,
//   D_d(k1, l1) = sum_m (-s_m / 2) sum_s G_s(k1 w1; k1 - d w2) G_s(l1 - d w2 + x; l1 w1 + x),
// q = l1 - k1, 36 x 36 for each of the 36 differences d of a frequency tile (w1, w2), K over the batch.
//
// Eight measurements (one K step of the m16n8k16 MMA: eight measurements x two spins) of a tile's whole
// blocks are 332 KB, more than an SM's shared memory.  But the elements with a given d_y = (k1 - k2)_y are, in
// each row k1, one run of six consecutive columns, and every element belongs to one d.  So a CTA takes the
// six d of one d_y and stages 48 bytes of each row, a sixth of the blocks (55 KB per K step, two steps
// deep).  It takes the columns l1 of the first four l1_y or those of the other two (which are the B elements of
// four or two rows lr_y); the twelve CTAs of a tile run next to each other, and two fit on an SM, so that one
// multiplies while the other adds its sums to G4 or waits for its first copies.
//
// Six warps, one per d: rows k1 as three 16-row tiles, columns l1 as three 8-column tiles, or as two (48 x 40
// of 36 x 36 used).  Operands, product order and promotion are those of tp_g4_mma.cu: x = 2^e (hi + lo), lo*hi,
// hi*lo, hi*hi per real product, each step's chain from zero, promoted into FP32 registers with 2^-2e, e from the
// step's largest |G| (gmax).  The sums leave through a table [line][k2][k1_x] (a line is a transfer for each k2), in runs of six consecutive k1 of G4
// (96 bytes) and of the disconnected terms.
//
// Half G: a block of the lower frequency half is read as the conjugate of its mirror with k -> -k (whole
// runs again).  Half G4: only the tiles of tile_order run.
//
// Bound by latencies: the tensor pipe is busy for a quarter of the time, a quarter of it goes to the sums' way
// into G4 (0.42 ms, 0.14 at the memory's rate), the rest to fragment reads and FP16 splits.  Nw = 32, half G and
// half G4, a batch of 128 measurements: 1.59 ms; 1.65 with one CTA of twelve warps on an SM (a batch of 32: 0.71
// and 0.69); 2.13 (0.74) on the FP32 pipe (updateG4SinglebandOuterSplit).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "async_copy.cuh"
#include "common.cuh"
#include "tp_g4.hpp"

namespace dcaacc {
namespace {

constexpr int kL = 6, kNc = kL * kL;
constexpr int kBlk = kNc * kNc;
constexpr int kMeasPerStep = 8;
constexpr uint32_t kRowBytes = kL * sizeof(float2);     // 48: one run of a row
constexpr uint32_t kPartBytes = kNc * kRowBytes;        // 1,728: A or B of one spin
constexpr uint32_t kSlotBytes = 4 * kPartBytes + 32;    // A0 B0 A1 B1 of a measurement + bank skew
constexpr uint32_t kStageBytes = kMeasPerStep * kSlotBytes;
constexpr int kStages = 2;
constexpr int kWarps = kL, kThreads = 32 * kWarps;      // a warp per d
constexpr int kChunks = 4 * kNc * 3;                    // 16-byte copies of a measurement
constexpr int kCopies = (kChunks + kThreads - 1) / kThreads;
constexpr int kSplitY = 4, kSplitCol = kSplitY * kL;    // l1_y, l1 of the CTA with three column tiles
constexpr int kMaxSteps = 32;  // batches of up to 256 measurements
// ... and from 32 on: the split operands' error does not depend on the batch, that of the FP32 chain does.  G4
// against 64 bits, n 100..500: 2.6e-7 at any batch, against 2.4e-7 (12 measurements), 2.7 (24), 2.8 (32) and
// 3.0 (64) in FP32; n < 60: 1.2e-7 against 1.2 (12), 1.6 (24), 1.8 (32) and 2.5.  Over fifteen draws (n 1..1000, Nw
// 4..20, batches of 32 and 64) 0.7e-7 .. 2.1e-7 against 0.9e-7 .. 2.7e-7, larger in one (1.5e-7, 1.1e-7); the median
// relative error of entries below a thousandth of the rms 0.3e-6 .. 0.9e-6 against 0.4e-6 .. 1.9e-6.
constexpr int kMinSlots = 32;
constexpr uint32_t kTableBytes = kSplitCol * kNc * kL * sizeof(float2);
static_assert(kTableBytes <= kStages * kStageBytes, "the flush table reuses the stages");
constexpr uint32_t kOffExp = kStages * kStageBytes;
constexpr uint32_t kOffRun = kOffExp + 4 * kMaxSteps;    // [2][36] source offset of a row's run (A, B)
constexpr uint32_t kOffKsub = kOffRun + 4 * 2 * kNc;     // [a + 36 b] = b - a
constexpr uint32_t kOffKneg = kOffKsub + kBlk;           // k -> -k
constexpr uint32_t kOffQinv = kOffKneg + kNc;            // q -> its position in q_list
constexpr uint32_t kOffSigns = kOffQinv + kNc;           // [m]
constexpr size_t kSmem = kOffSigns + kMaxSteps * kMeasPerStep;
static_assert(kPartBytes == 16 * 3 * kNc, "chunk order");
static_assert(kSmem <= 113 * 1024, "shared memory per CTA");
constexpr int kExpMax = 60;  // |e| <= 60 keeps 2^{+-2e} a normal FP32 number
constexpr int kMaxCh = 2;

__device__ inline uint32_t asU32(__half2 h) {
  return *reinterpret_cast<uint32_t*>(&h);
}
// (x0, x1) = hi + lo, both rounded to nearest, x0 in the low 16 bits.
__device__ inline void splitPair(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x0, x1);
  const float2 hf = __half22float2(h);
  hi = asU32(h);
  lo = asU32(__floats2half2_rn(x0 - hf.x, x1 - hf.y));
}
__device__ inline void mma16816(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ inline int stepExp(float mx) {
  return mx > 0.f ? max(-kExpMax, min(kExpMax, 14 - ilogbf(mx))) : 0;
}
__device__ inline float pow2(int e) {
  return __int_as_float((127 + e) << 23);  // |e| <= 126
}

// One K step of a warp: rows k1 = 16 mt + g + 8 r, columns l1 = 8 (n0 + n) + g; lane (g = lane / 4, t4 = lane % 4)
// holds K pairs (measurement t4 + 4 j; spins 0, 1).  oa / ob: byte offsets of the elements inside a
// measurement slot's A0 / B0 (spin 1 two parts further); rows and columns past 36 count as zero.
template <int NT, bool FULL>
__device__ __forceinline__ void stepMma(const unsigned char* S, const int (&oa)[5], const int (&ob)[NT], bool a4,
                                        bool blast, int t4, int m0, int n_slots, const signed char* sgn, float sc,
                                        float inv, float ca, float cb, float (&re)[3][NT][4], float (&im)[3][NT][4]) {
  float fa[2], fb[2];
  bool valid[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int m = m0 + t4 + 4 * j;
    valid[j] = FULL || m < n_slots;
    fa[j] = valid[j] ? -0.5f * static_cast<float>(sgn[m]) * sc : 0.f;
    fb[j] = valid[j] ? sc : 0.f;
  }
  const float2 z = make_float2(0.f, 0.f);
  auto pair = [&](int j, int off, bool live, float f, float fi, uint32_t& rh, uint32_t& rl, uint32_t& ih, uint32_t& il) {
    const unsigned char* p = S + (t4 + 4 * j) * kSlotBytes + off;
    const bool on = valid[j] && live;
    const float2 x0 = on ? *reinterpret_cast<const float2*>(p) : z;
    const float2 x1 = on ? *reinterpret_cast<const float2*>(p + 2 * kPartBytes) : z;
    splitPair(x0.x * f, x1.x * f, rh, rl);
    splitPair(x0.y * fi, x1.y * fi, ih, il);
  };
  uint32_t brh[NT][2], brl[NT][2], bih[NT][2], bil[NT][2];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int j = 0; j < 2; ++j)
      pair(j, kPartBytes + ob[n], n + 1 < NT || blast, fb[j], fb[j] * cb, brh[n][j], brl[n][j], bih[n][j], bil[n][j]);
#pragma unroll
  for (int mt = 0; mt < 3; ++mt) {
    uint32_t arh[4], arl[4], aih[4], ail[4], naih[4], nail[4];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int k = 2 * j + r;
        if (2 * mt + r < 5) {
          pair(j, oa[2 * mt + r < 5 ? 2 * mt + r : 0], 2 * mt + r < 4 || a4, fa[j], fa[j] * ca, arh[k], arl[k], aih[k],
               ail[k]);
        }
        else {
          arh[k] = arl[k] = aih[k] = ail[k] = 0;  // rows 40 .. 47
        }
        naih[k] = aih[k] ^ 0x80008000u;
        nail[k] = ail[k] ^ 0x80008000u;
      }
    float tr[NT][4], ti[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int k = 0; k < 4; ++k)
        tr[n][k] = ti[n][k] = 0.f;
    // Re = ar br - ai bi, Im = ar bi + ai br; small products first, the chains interleaved.
    auto products = [&](const uint32_t(&ar)[4], const uint32_t(&ai)[4], const uint32_t(&br)[NT][2],
                        const uint32_t(&bi)[NT][2]) {
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        mma16816(tr[n], ar, br[n]);
        mma16816(ti[n], ai, bi[n]);
      }
    };
    products(arh, arh, brl, bil);
    products(arl, arl, brh, bih);
    products(naih, aih, bil, brl);
    products(nail, ail, bih, brh);
    products(arh, arh, brh, bih);
    products(naih, aih, bih, brh);
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        re[mt][n][k] = fmaf(tr[n][k], inv, re[mt][n][k]);
        im[mt][n][k] = fmaf(ti[n][k], inv, im[mt][n][k]);
      }
  }
}

struct Tables {
  const int* step_exp;
  const unsigned char *ksub, *kneg;
  const signed char* sgn;
};

// The table's line of entry (k1, l1): the l1 that belongs to the first k1 of its run and the same q = l1 - k1.
__device__ inline int lineOf(const Tables& tb, int k1, int l1) {
  return tb.ksub[tb.kneg[k1 / kL * kL] + kNc * tb.ksub[k1 + kNc * l1]];
}

// The batch loop of a warp: columns l1 from 8 N0 on, NT tiles of 8, and its part of the flush table.
template <int NT, int N0, typename Advance>
__device__ __forceinline__ void batchProduct(unsigned char* smem, const Tables& tb, int d, bool mir_a, bool mir_b,
                                             int n_slots, Advance advance) {
  constexpr int n0 = N0;
  const int lane = threadIdx.x % 32, g = lane >> 2, t4 = lane & 3;
  // Element (k1, k2 = k1 - d) of A: staged row k1, column k2_x of the run (mirrored: (-k2)_x); element
  // (lr = l1 - d, l1) of B: staged row lr, column l1_x (mirrored: (-l1)_x).
  int oa[5], ob[NT];
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const int k1 = min(8 * i + g, kNc - 1), k2 = tb.ksub[d + kNc * k1];
    oa[i] = k1 * kRowBytes + ((mir_a ? tb.kneg[k2] : k2) % kL) * sizeof(float2);
  }
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    const int l1 = min(8 * (n0 + n) + g, kNc - 1), lr = tb.ksub[d + kNc * l1];
    ob[n] = lr * kRowBytes + ((mir_b ? tb.kneg[l1] : l1) % kL) * sizeof(float2);
  }
  const bool a4 = 32 + g < kNc, blast = 8 * (n0 + NT - 1) + g < kNc;
  const float ca = mir_a ? -1.f : 1.f, cb = mir_b ? -1.f : 1.f;
  float re[3][NT][4], im[3][NT][4];
#pragma unroll
  for (int mt = 0; mt < 3; ++mt)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int k = 0; k < 4; ++k)
        re[mt][n][k] = im[mt][n][k] = 0.f;
  const int n_steps = (n_slots + kMeasPerStep - 1) / kMeasPerStep;
  for (int step = 0; step < n_steps; ++step) {
    advance(step);  // this step has landed for the whole CTA; the copies of a later one start
    const unsigned char* S = smem + step % kStages * kStageBytes;
    const int e = tb.step_exp[step], m0 = step * kMeasPerStep;
    if (m0 + kMeasPerStep <= n_slots)
      stepMma<NT, true>(S, oa, ob, a4, blast, t4, m0, n_slots, tb.sgn, pow2(e), pow2(-2 * e), ca, cb, re, im);
    else
      stepMma<NT, false>(S, oa, ob, a4, blast, t4, m0, n_slots, tb.sgn, pow2(e), pow2(-2 * e), ca, cb, re, im);
  }
  __syncthreads();  // every warp is done with the stages
  float2* table = reinterpret_cast<float2*>(smem);
#pragma unroll
  for (int mt = 0; mt < 3; ++mt)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int k1 = 16 * mt + g + 8 * (k >> 1), l1 = 8 * (n0 + n) + 2 * t4 + (k & 1);
        if (k1 < kNc && l1 < kNc)
          table[((lineOf(tb, k1, l1) - 8 * N0) * kNc + tb.ksub[d + kNc * k1]) * kL + k1 % kL] =
              make_float2(re[mt][n][k], im[mt][n][k]);
      }
  __syncthreads();
}

__global__ void __launch_bounds__(kThreads, 2)
updateG4DirectMma36(const TpDims dims, const float2* __restrict__ G, long g_sector_stride,
                    const int* __restrict__ signs, int n_slots, const int* __restrict__ k_sub,
                    const int* __restrict__ q_list, const int* __restrict__ wex_list, const int* __restrict__ gmax,
                    const unsigned* __restrict__ tile_order, const float2* __restrict__ disc,
                    double2* const* __restrict__ G4, bool atomic) {
  extern __shared__ __align__(16) unsigned char smem[];
  int* step_exp = reinterpret_cast<int*>(smem + kOffExp);
  int* run = reinterpret_cast<int*>(smem + kOffRun);
  unsigned char* ksub = smem + kOffKsub;
  unsigned char* kneg = smem + kOffKneg;
  unsigned char* qinv = smem + kOffQinv;
  signed char* sgn = reinterpret_cast<signed char*>(smem + kOffSigns);
  const int t = threadIdx.x, warp = t / 32, lane = t % 32;
  const int nw = dims.nw, nw_ext = dims.nw_ext, nq = dims.nq, n_ch = dims.n_channels;
  const int part = blockIdx.x % (2 * kL), tile = blockIdx.x / (2 * kL);  // the twelve CTAs of a tile run next to each other
  const int dy = part >> 1;
  const bool wide = (part & 1) == 0;  // columns l1 < 24, or the others
  const int per_wq = tile_order ? nw * nw / 2 : nw * nw;
  int w1, w2;
  if (tile_order) {
    const unsigned v = tile_order[tile % per_wq];
    w1 = static_cast<int>(v & 0xffffu);
    w2 = static_cast<int>(v >> 16);
  }
  else {
    w1 = tile % per_wq % nw;
    w2 = tile % per_wq / nw;
  }
  const int iwq = tile / per_wq, wex = wex_list[iwq];
  const int w1e = w1 + dims.ext, w2e = w2 + dims.ext, w1x = w1e + wex, w2x = w2e + wex;
  const bool mir_a = dims.half_g && 2 * w1e < nw_ext, mir_b = dims.half_g && 2 * w2x < nw_ext;
  auto block = [&](int wr, int wc, bool mir) {
    return (mir ? static_cast<long>(nw_ext - 1 - wr) * nw_ext + nw_ext - 1 - wc
                : static_cast<long>(wr) * nw_ext + wc) * kBlk;
  };
  const long b_A = block(w1e, w2e, mir_a), b_B = block(w2x, w1x, mir_b);
  const int n_steps = (n_slots + kMeasPerStep - 1) / kMeasPerStep;

  for (int e = t; e < kBlk; e += kThreads)
    ksub[e] = static_cast<unsigned char>(k_sub[e]);
  const int z0 = k_sub[0];  // k_0 - k_0: the zero momentum
  for (int e = t; e < kNc; e += kThreads) {
    qinv[q_list[e]] = static_cast<unsigned char>(e);
    kneg[e] = static_cast<unsigned char>(k_sub[e + kNc * z0]);
  }
  for (int m = t; m < n_slots; m += kThreads)
    sgn[m] = static_cast<signed char>(signs[m]);
  for (int step = warp; step < n_steps; step += kWarps) {
    const int m0 = step * kMeasPerStep;
    float mx = lane < 2 * min(kMeasPerStep, n_slots - m0) ? __int_as_float(gmax[2 * m0 + lane]) : 0.f;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    if (lane == 0)
      step_exp[step] = stepExp(mx);
  }
  __syncthreads();
  // Source offset of each staged row's run.  A, row k1: columns k1 - d, d_y = dy; B, row lr: columns lr + d.
  for (int e = t; e < 2 * kNc; e += kThreads) {
    const int r = e % kNc, d = kL * dy;
    if (e < kNc) {
      const int c = ksub[d + kNc * r];
      run[e] = mir_a ? kneg[r] * kNc + kneg[c] / kL * kL : r * kNc + c / kL * kL;
    }
    else {
      const int c = ksub[kneg[d] + kNc * r];
      run[e] = mir_b ? kneg[r] * kNc + kneg[c] / kL * kL : r * kNc + c / kL * kL;
    }
  }
  __syncthreads();

  // This thread's copies of a measurement, 16-byte chunk t + kThreads i: part A0 B0 A1 B1, row, third; without
  // the B rows lr = l1 - d of the other columns l1.
  int src[kCopies];  // element of its block, or -1
#pragma unroll
  for (int i = 0; i < kCopies; ++i) {
    const int c = t + kThreads * i, p = c / (3 * kNc) % 4, row = c % (3 * kNc) / 3, third = c % 3;
    const int l1 = ksub[kneg[kL * dy] + kNc * row];  // row + d: y of the columns that read this row of B
    const bool need = c < kChunks && (!(p & 1) || (l1 < kSplitCol) == wide);
    src[i] = !need ? -1 : (p & 1) ? run[kNc + row] + 2 * third : run[row] + 2 * third;
  }
  auto copyStep = [&](int step) {
    if (step < n_steps) {
      const uint32_t to = smemAddr(smem) + step % kStages * kStageBytes + 16 * t;  // chunks lie in order
      const int n = min(kMeasPerStep, n_slots - step * kMeasPerStep);
      const float2* base = G + g_sector_stride * (2 * kMeasPerStep * static_cast<long>(step));
#pragma unroll
      for (int i = 0; i < kCopies; ++i) {
        if (src[i] < 0)
          continue;
        const int p = (t + kThreads * i) / (3 * kNc);
        const float2* from = base + (p >> 1) * g_sector_stride + ((p & 1) ? b_B : b_A) + src[i];
        for (int m = 0; m < n; ++m)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 16 * kThreads * i + m * kSlotBytes),
                       "l"(from + 2 * m * g_sector_stride)
                       : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int s = 0; s < kStages - 1; ++s)
    copyStep(s);
  auto advance = [&](int step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();
    copyStep(step + kStages - 1);
  };
  const Tables tb{step_exp, ksub, kneg, sgn};
  const int d = kL * dy + warp;
  if (wide)
    batchProduct<3, 0>(smem, tb, d, mir_a, mir_b, n_slots, advance);
  else
    batchProduct<2, 3>(smem, tb, d, mir_a, mir_b, n_slots, advance);

  // Flush: k1_x fastest, then k2, then the line; U entries' loads in flight.
  const float2* table = reinterpret_cast<const float2*>(smem);
  const int line0 = wide ? 0 : kSplitCol, entries = (wide ? kSplitCol : kNc - kSplitCol) * kNc * kL;
  const long M = static_cast<long>(kNc) * nw;
  const long s_w1 = kNc, s_k2 = s_w1 * nw, s_w2 = s_k2 * kNc, s_q = s_w2 * nw, s_wq = s_q * nq;
  constexpr int U = 9;
  for (int c = 0; c < n_ch; ++c)
    for (int base = t; base < entries; base += U * kThreads) {
      double2 o[U];
      float2 v[U];
      long at[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int idx = min(base + u * kThreads, entries - 1);
        const int kx = idx % kL, k2 = idx / kL % kNc, l1 = line0 + idx / (kL * kNc);
        // k1 = k2 + d has y = (k2 + d)_y; the run's x are those of the table.
        const int k1 = ksub[kneg[kL * dy] + kNc * k2] / kL * kL, qi = qinv[ksub[k1 + kNc * l1]];
        at[u] = k1 + kx + w1 * s_w1 + k2 * s_k2 + w2 * s_w2 + qi * s_q + iwq * s_wq;
        const float2 dv = __ldg(disc + ((static_cast<long>(iwq * nq + qi) * n_ch + c) * M + k2 +
                                        static_cast<long>(kNc) * w2) * M + k1 + kx + static_cast<long>(kNc) * w1);
        const float2 x = table[idx];
        v[u] = make_float2(x.x + dv.x, x.y + dv.y);
        o[u] = atomic ? make_double2(0., 0.) : G4[c][at[u]];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (base + u * kThreads >= entries)
          continue;
        double2* p = G4[c] + at[u];
        if (atomic) {
          atomicAdd(&p->x, static_cast<double>(v[u].x));
          atomicAdd(&p->y, static_cast<double>(v[u].y));
        }
        else {
          *p = make_double2(o[u].x + static_cast<double>(v[u].x), o[u].y + static_cast<double>(v[u].y));
        }
      }
    }
}

}  // namespace

bool directTc36Applies(const G4Args& a) {
  return a.dims.nb == 1 && a.dims.nc == kNc && a.grid6 && a.q_all && a.gmax != nullptr && a.dims.n_channels <= kMaxCh &&
         a.n_slots >= kMinSlots && a.n_slots <= kMaxSteps * kMeasPerStep;
}

void launchDirectTc36(const G4Args& a, const float2* G, long g_sector_stride, const float2* disc, cudaStream_t stream) {
  const TpDims& d = a.dims;
  DCAACC_CUDA_CHECK(cudaFuncSetAttribute(updateG4DirectMma36, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmem)));
  const long tiles = long(d.nw) * d.nw * d.nwq / (a.tile_order ? 2 : 1);  // half G4: w1 >= Nw / 2 only
  updateG4DirectMma36<<<static_cast<unsigned>(tiles * 2 * kL), kThreads, kSmem, stream>>>(
      d, G, g_sector_stride, a.signs, a.n_slots, a.k_sub, a.q_list, a.wex_list, a.gmax, a.tile_order, disc, a.G4, a.atomic);
  DCAACC_LAUNCH_CHECK();
}

}  // namespace dcaacc
