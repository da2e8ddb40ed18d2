// Front-end of the mixed path factored by orbital in FP32: M(tau, tau') -> G(k1, w1; k2, w2) for every
// sector of a batch.
//
// The same two steps as the FP64 front-end (tp_frontend.cu; the reference's CachedNdft<GPU>::execute,
// cached_ndft_gpu.hpp:131-252, SpaceTransform2DGpu::execute, space_transform_2D_gpu.hpp:116-171, and
// computeG, tp_accumulator_kernels.cu:73-217),
//   row     X'(b1 k1 w1, j) = -1/Nc sum_b G0(b1, b; k1, w1) sum_r e^{i k1 (r + a_b)}
//                             sum_{i in orbital (b, r)} T(w1, i) M(i, j)
//   column  G(b1 k1 w1; b2 k2 w2) = sum_b [sum_r e^{-i k2 (r + a_b)} sum_{j in (b, r)} X'(.., j) conj T(w2, j)]
//                             G0(b, b2; k2, w2) + beta G0 delta,
// with FP32 operands, products and sums rounded to nearest; twiddles, phases and G0 factors are
// computed in FP64 and rounded once.  With the mirror symmetry (half_g) only the rows w1 >= NwExt / 2
// are computed.
//
// Why not the tensor cores: as dense products (P M and X' Q^H, tp_frontend_tc.cu) the two steps take
// 4 D n^2 and 8 D^2 n flops three times over (split FP16) and three operand builders; grouped by
// orbital they take 4 NwExt n^2 and 8 D NwExt n, nb Nc times fewer, which the FP32 pipe does in less
// time.  Half G, per batch, operand builders included: 4x4, Nw = 64, n 50..400, 64 measurements 0.66 -> 0.48 ms
// (column step 0.35, row step 0.086, sort of M 0.032); 6x6, Nw = 32, n 300..1000, 128 measurements 8.4 (whole
// G) -> 2.3 ms (1.19, 0.64, 0.43).  The G4 of a 4x4 batch is off by 2.8e-7 of the 64-bit sums instead of 5.9e-7.
//
// CTA = 32 rows of G (row step: 32 columns of M) x WT frequencies, eight or sixteen warps.
// Phase 1: the warps take the orbitals from a counter.  A warp holds the whole 32 x WT tile, 4 x WT/4
// sums a lane, and streams its orbital's vertices, two (row step: four) at a time, through its own
// ring of asynchronous 16-byte copies.
// The multiply-adds are packed pairs (fma.f32x2): the same peak as scalar ones at half the issue
// slots, which leaves room for the shared-memory reads.  Column step: X' (x, y) times (c, c) and (s, s)
// in two sums, combined into X' conj T at the end; the twiddles are stored doubled so that one 16-byte
// read gives both factors.  Row step: T (c, s) times (M, M).
// Phase 2: the cluster transform of the sums in shared memory.  On an L x L cluster (L = 4, 6) an
// FFT, one (row, frequency) pair a thread, in place; the result leaves row by row (the sums of an
// orbital are padded by one, so that lanes along k and lanes along rows both read distinct banks).
// Otherwise the matrix of phases, 4 x 2 sums a lane.  The 4x4 column step keeps the
// FP32 pipe busy for a third of its time and shared memory for 60 %; two CTAs per SM (128 registers a
// thread) leave four warps per scheduler to hide both.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "async_copy.cuh"
#include "common.cuh"
#include "packed.cuh"
#include "tp_frontend.hpp"

namespace dcaacc {

namespace {

constexpr int kLong = 32;  // rows of G or columns of M per tile
constexpr int kRing = 4;   // ring slots per warp
constexpr int kColV = 2;   // vertices per ring slot, column step
constexpr int kRowV = 4;   // ... row step (M is read four sorted rows at a time)

// Shared memory by 32-bit address: an immediate offset per access and no generic addressing.
template <int OFF = 0>
__device__ inline Pair lds64(uint32_t a) {
  Pair v;
  asm volatile("ld.shared.b64 %0, [%1+%2];" : "=l"(v) : "r"(a), "n"(OFF));
  return v;
}
template <int OFF = 0>
__device__ inline ulonglong2 lds128(uint32_t a) {
  ulonglong2 v;
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2+%3];" : "=l"(v.x), "=l"(v.y) : "r"(a), "n"(OFF));
  return v;
}
template <int OFF = 0>
__device__ inline void sts64(uint32_t a, Pair v) {
  asm volatile("st.shared.b64 [%0+%1], %2;" ::"r"(a), "n"(OFF), "l"(v) : "memory");
}
__device__ inline void cpAsync16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ inline void cpAsyncCommit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ inline void cpAsyncWait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Matsubara frequency of extended index w (vertex_frequency_domain.hpp, EXTENDED).
__device__ inline double extFreq(int w, int nw_ext, double beta) {
  const int half = nw_ext / 2;
  if (w >= half)
    return M_PI / beta * (1 + 2 * (w - half));
  return -M_PI / beta * (1 + 2 * (half - 1 - w));
}

// Twiddles of the row-sorted vertices, T2 (c, s), and of the column-sorted ones, T4 (c, c, s, s):
// [vertex][w], e^{i w tau} in FP64 (x = tau w as in CachedNdft<CPU>::computeT, cached_ndft_cpu.hpp:151-156)
// rounded to FP32.  Only w >= NwExt / 2 is evaluated; the other half is its conjugate.
__global__ void twiddle32Kernel(const SectorDesc* __restrict__ sectors, const double* __restrict__ tau,
                                const int* __restrict__ perm_r, const int* __restrict__ perm_c,
                                float2* __restrict__ T2, float4* __restrict__ T4, int nw_ext, double beta) {
  const SectorDesc sd = sectors[blockIdx.y];
  const int half = nw_ext / 2;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < sd.n * half; idx += gridDim.x * blockDim.x) {
    const int v = idx / half, w = half + idx % half;
    const double om = extFreq(w, nw_ext, beta);
    const long at = static_cast<long>(sd.vtx_off + v) * nw_ext;
    double s, c;
    const int vr = perm_r[sd.vtx_off + v], vc = perm_c[sd.vtx_off + v];
    sincos(tau[sd.vtx_off + vr] * om, &s, &c);
    T2[at + w] = make_float2(static_cast<float>(c), static_cast<float>(s));
    T2[at + nw_ext - 1 - w] = make_float2(static_cast<float>(c), static_cast<float>(-s));
    if (vc != vr)
      sincos(tau[sd.vtx_off + vc] * om, &s, &c);
    const float cf = static_cast<float>(c), sf = static_cast<float>(s);
    T4[at + w] = make_float4(cf, cf, sf, sf);
    T4[at + nw_ext - 1 - w] = make_float4(cf, cf, -sf, -sf);
  }
}

// M in sorted order, FP32: Ms[sector][j][i] = M(perm_r[i], perm_c[j]), rows of Kr floats.  One warp per
// column j: it is read contiguously into the warp's shared-memory row, the permuted entries come from
// there.  Bound by the read of M.
constexpr int kSortWarps = 8;
__global__ void __launch_bounds__(32 * kSortWarps)
sortM32Kernel(const SectorDesc* __restrict__ sectors, const int* __restrict__ perm_r, const int* __restrict__ perm_c,
              int Kr, int row_floats, float* __restrict__ Ms) {
  extern __shared__ float mrows[];  // [warps][row_floats]
  const SectorDesc sd = sectors[blockIdx.y];
  const int n = sd.n, warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int j = blockIdx.x * (blockDim.x / 32) + warp;
  if (j >= n)
    return;
  float* row = mrows + warp * row_floats;
  const int* pr = perm_r + sd.vtx_off;
  const long col = static_cast<long>(sd.ldm) * perm_c[sd.vtx_off + j];
  constexpr int U = 8;  // loads in flight per lane
  for (int i0 = lane; i0 < n; i0 += 32 * U) {
    double m[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      m[u] = i0 + 32 * u < n ? loadM(sd, col + i0 + 32 * u) : 0.;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + 32 * u < n)
        row[i0 + 32 * u] = static_cast<float>(m[u]);
  }
  __syncwarp();
  float* out = Ms + (static_cast<long>(blockIdx.y) * Kr + j) * Kr;
#pragma unroll 4
  for (int i = lane; i < n; i += 32)
    out[i] = row[pr[i]];
}

// The tile of one CTA in shared memory: the warps' rings, the orbitals' sums Z[slot][w][l] (l = 0..31
// along the tile's long side, stored at l ^ 8 (w & 1): the two frequencies that a half-warp stores
// at once fall in distinct banks), the factors (FFT: C[w][slot]; matrix: phases F[b][r][k], k padded with
// zeros), the orbital starts, the FFT's slot of each orbital and the counter.
template <int WT, int L>
struct Tile32 {
  static constexpr int kWarps = L == 6 && WT == 16 ? 16 : 8;  // 36 orbitals' sums leave room for one CTA per SM
  static constexpr int kThreads = 32 * kWarps;
  // CTAs an SM: the matrix forms' steps are chains of short loops.  2x2, Nw = 24, a batch of 64, n 20..60, 100..200 and
  // 200..450: row step 17, 47 and 129 us with two, 13, 36 and 98 with four; column step 29, 43 and 65 with two, 23, 35 and
  // 53 with three (60 with four: spills).
  static constexpr int kRowResident = L == 6 && WT == 16 ? 1 : L == 0 && WT == 8 ? 4 : 2;
  static constexpr int kColResident = L == 6 && WT == 16 ? 1 : L == 0 && WT == 8 ? 3 : 2;
  static constexpr int kSub = WT / 4;           // frequencies of a lane
  static constexpr int kSums = kLong * WT + 1;  // stride of an orbital's sums
  static constexpr int kSlotBytes = 512 + 32 * WT;
  uint32_t ring, z_addr, f_addr;  // shared addresses of the rings, the sums and the factors
  float2 *Z, *F;
  int *start, *slot_of, *next, *slot_k;

  __host__ __device__ static int kPad(const TpDims& d) {
    return d.nb == 1 ? (d.nc + 15) / 16 * 16 : (d.nc + 7) / 8 * 8;
  }
  __host__ __device__ static int factors(const TpDims& d) {
    return L ? WT * L * L : d.nb * d.nc * kPad(d);
  }
  __host__ __device__ static size_t bytes(const TpDims& d) {
    return size_t(kWarps) * kRing * kSlotBytes + sizeof(float2) * ((size_t(d.n_orb) * kSums + 1) / 2 * 2 + factors(d)) +
           sizeof(int) * (2 * d.n_orb + 2 + L * L);
  }
  __device__ Tile32(unsigned char* raw, const TpDims& d) {
    Z = reinterpret_cast<float2*>(raw + kWarps * kRing * kSlotBytes);
    F = Z + (d.n_orb * kSums + 1) / 2 * 2;  // 16-byte aligned
    ring = smemAddr(raw);
    z_addr = smemAddr(Z);
    f_addr = smemAddr(F);
    start = reinterpret_cast<int*>(F + factors(d));
    slot_of = start + d.n_orb + 1;
    next = slot_of + d.n_orb;
    slot_k = next + 1;
  }
  // Element l of line w in slot 0; slot s is s kSums further.
  __device__ uint32_t lineAddr(int w, int l) const {
    return z_addr + 8 * (w * kLong + (l ^ ((w & 1) << 3)));
  }

  // Starts, counter, and the factors of phase 2: factor(w, k) in FFT form.
  template <typename Factor>
  __device__ void fill(const TpDims& d, const double2* __restrict__ Fb, const int* __restrict__ orb_start,
                       const ColFft& fft, Factor factor) {
    if constexpr (L > 0) {
      for (int i = threadIdx.x; i < WT * L * L; i += kThreads)
        F[i] = factor(i / (L * L), static_cast<int>(fft.kmap[i % (L * L)]));
    }
    else {
      const int kp = kPad(d);
      for (int i = threadIdx.x; i < d.nb * d.nc * kp; i += kThreads) {
        const int k = i % kp, r = (i / kp) % d.nc, b = i / (kp * d.nc);
        F[i] = k < d.nc ? to_f2(Fb[(b * d.nc + k) * d.nc + r]) : make_float2(0.f, 0.f);
      }
    }
    for (int i = threadIdx.x; i <= d.n_orb; i += kThreads)
      start[i] = orb_start[i];
    for (int i = threadIdx.x; i < d.n_orb; i += kThreads) {
      if constexpr (L > 0) {
        slot_of[fft.rmap[i]] = i;
        slot_k[fft.kmap[i]] = i;
      }
      else {
        slot_of[i] = i;
      }
    }
    if (threadIdx.x == 0)
      *next = 0;
    __syncthreads();
  }

  // Phase 1: hands the orbitals to the warps.  begin(g) points this lane's copies at vertex g; issue(slot) starts those
  // of the next V vertices into a ring slot; use(slot, lo, hi, first) adds vertices lo .. hi - 1 of a landed slot
  // (first: they start the sums); done(s) stores the sums of the orbital in slot s.  ALIGNED: slots start at
  // multiples of V.  The copies may run past an orbital's last vertex, by less than V vertices.
  template <int V, bool ALIGNED, typename Begin, typename Issue, typename Use, typename Done>
  __device__ void orbitals(int n_orb, Begin begin, Issue issue, Use use, Done done) {
    const int lane = threadIdx.x % 32;
    const uint32_t mine = ring + (threadIdx.x / 32) * kRing * kSlotBytes;
    for (;;) {
      int o = 0;
      if (lane == 0)
        o = atomicAdd(next, 1);
      o = __shfl_sync(0xffffffffu, o, 0);
      if (o >= n_orb)
        break;
      const int v0 = start[o], v1 = start[o + 1];
      const uint32_t z = z_addr + 8 * kSums * slot_of[o];
      if (v0 == v1) {  // no vertices: its sums are zero
        for (int i = lane; i < kSums; i += 32)
          sts64(z + 8 * i, 0);
        continue;
      }
      const int g0 = ALIGNED ? v0 / V * V : v0;
      __syncwarp();  // every lane is done with the previous orbital's slots
      begin(g0);
#pragma unroll
      for (int p = 0; p < kRing - 1; ++p) {
        if (g0 + p * V < v1)
          issue(mine + p * kSlotBytes);
        cpAsyncCommit();
      }
      cpAsyncWait<kRing - 2>();
      __syncwarp();
      if (g0 + (kRing - 1) * V < v1)
        issue(mine + (kRing - 1) * kSlotBytes);
      cpAsyncCommit();
      use(mine, v0 - g0, v1 - g0, std::true_type{});
      uint32_t fill_slot = mine, cur = mine + kSlotBytes;
      for (int left = v1 - g0 - V; left > 0; left -= V) {
        cpAsyncWait<kRing - 2>();
        __syncwarp();  // this slot has landed for every lane, and every lane is done with the one before
        if (left > (kRing - 1) * V)
          issue(fill_slot);
        cpAsyncCommit();
        use(cur, 0, left, std::false_type{});
        fill_slot = cur;
        cur = cur == mine + (kRing - 1) * kSlotBytes ? mine : cur + kSlotBytes;
      }
      done(z);
    }
    cpAsyncWait<0>();
    __syncthreads();
  }

  // Matrix phase 2: acc[i][c] = sum_r Z(b, r; w, l0 + 4 i) F(b, k0 + lane % 8 + 8 c; r), F conjugated when CONJ.
  template <bool CONJ, int KC>
  __device__ void clusterSum(float2 (&acc)[4][KC], const TpDims& d, int nb, int b, int w, int l0, int k0) const {
    const int kp = kPad(d);
    const float2* f = F + b * d.nc * kp + k0 + threadIdx.x % 8;
    const float2* z = Z + b * kSums + w * kLong;
    int off[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      off[i] = (l0 + 4 * i) ^ ((w & 1) << 3);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < KC; ++c)
        acc[i][c] = make_float2(0.f, 0.f);
#pragma unroll 2
    for (int r = 0; r < d.nc; ++r, z += nb * kSums, f += kp) {
      float2 zv[4], fv[KC];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        zv[i] = z[off[i]];
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
};

// x times -i (SIGN < 0) or i.
template <int SIGN>
__device__ inline Pair rot(Pair x) {
  const float2 v = floatsOf(x);
  return SIGN < 0 ? pairOf(v.y, -v.x) : pairOf(-v.y, v.x);
}
// In-place DFT of L points at stride S, X[m] = sum_x e^{SIGN 2 pi i m x / L} z[x] (L = 4, or 6 as two
// 3-point DFTs and twiddles).
template <int SIGN, int L, int S>
__device__ inline void dftL(Pair* z) {
  if constexpr (L == 4) {
    const Pair t0 = add2(z[0], z[2 * S]), t1 = sub2(z[0], z[2 * S]), t2 = add2(z[S], z[3 * S]);
    const Pair t3 = rot<SIGN>(sub2(z[S], z[3 * S]));
    z[0] = add2(t0, t2);
    z[2 * S] = sub2(t0, t2);
    z[S] = add2(t1, t3);
    z[3 * S] = sub2(t1, t3);
  }
  else {
    static_assert(L == 6, "4 or 6 points");
    constexpr float h = 0.86602540378443864676f;  // sin(pi / 3)
    // y1 = a - (b + c) / 2 + SIGN i h (b - c), y2 its counterpart with -SIGN.
    auto dft3 = [&](Pair a, Pair b, Pair c, Pair& y0, Pair& y1, Pair& y2) {
      const Pair s = add2(b, c), d = rot<SIGN>(sub2(b, c));
      y0 = add2(a, s);
      Pair m = a;
      fma2(m, s, pairOf(-0.5f, -0.5f));
      y1 = y2 = m;
      fma2(y1, d, pairOf(h, h));
      fma2(y2, d, pairOf(-h, -h));
    };
    Pair e0, e1, e2, o0, o1, o2;
    dft3(z[0], z[2 * S], z[4 * S], e0, e1, e2);
    dft3(z[S], z[3 * S], z[5 * S], o0, o1, o2);
    // o_m e^{SIGN 2 pi i m / 6} = +-o_m / 2 + h SIGN i o_m, added to and taken from e_m.
    auto twiddle = [&](Pair o, float re) {
      Pair t = rot<SIGN>(o), x = 0;
      fma2(x, o, pairOf(re, re));
      fma2(x, t, pairOf(h, h));
      return x;
    };
    o1 = twiddle(o1, 0.5f);
    o2 = twiddle(o2, -0.5f);
    z[0] = add2(e0, o0);
    z[S] = add2(e1, o1);
    z[2 * S] = add2(e2, o2);
    z[3 * S] = sub2(e0, o0);
    z[4 * S] = sub2(e1, o1);
    z[5 * S] = sub2(e2, o2);
  }
}

// Phase 2 in FFT form for line w: thread = l; the sums of sites (a, b) in slots a + L b become factor times
// the transform at momenta (m, n), in slots m + L n.
template <int SIGN, int WT, int L, int G>
__device__ inline void loadLine(uint32_t line, Pair (&z)[L * L]) {
  if constexpr (G < L * L) {
    z[G] = lds64<8 * Tile32<WT, L>::kSums * G>(line);
    loadLine<SIGN, WT, L, G + 1>(line, z);
  }
}
template <int WT, int L, int G>
__device__ inline void storeLine(uint32_t line, uint32_t factors, const Pair (&z)[L * L]) {
  if constexpr (G < L * L) {
    const ulonglong2 f = lds128<8 * G>(factors);
    const float2 a = cmul(floatsOf(f.x), floatsOf(z[G])), b = cmul(floatsOf(f.y), floatsOf(z[G + 1]));
    sts64<8 * Tile32<WT, L>::kSums * G>(line, pairOf(a.x, a.y));
    sts64<8 * Tile32<WT, L>::kSums * (G + 1)>(line, pairOf(b.x, b.y));
    storeLine<WT, L, G + 2>(line, factors, z);
  }
}
template <int SIGN, int WT, int L>
__device__ inline void fftLine(const Tile32<WT, L>& t, int w) {
  const uint32_t line = t.lineAddr(w, threadIdx.x % 32);
  Pair z[L * L];
  loadLine<SIGN, WT, L, 0>(line, z);
#pragma unroll
  for (int b = 0; b < L; ++b)
    dftL<SIGN, L, 1>(z + L * b);
#pragma unroll
  for (int m = 0; m < L; ++m)
    dftL<SIGN, L, L>(z + m);
  storeLine<WT, L, 0>(line, t.f_addr + 8 * L * L * w, z);
  __syncwarp();
}

// The finished lines, row by row: per step 32 consecutive elements (l, k), k fastest, of the line's 32 rows
// l.  The steps' pattern of (l, k) repeats every kPeriod rows (two rows, or eight in nine steps), so a lane
// keeps its offsets of one period.
template <int WT, int L>
struct Drain {
  static constexpr int kRows = L == 4 ? 2 : 8, kSteps = kRows * L * L / 32;
  uint32_t off[kSteps];  // bytes from the line's start
  int l0[kSteps], k0[kSteps];
  __device__ explicit Drain(const Tile32<WT, L>& t) {
#pragma unroll
    for (int i = 0; i < kSteps; ++i) {
      const int e = threadIdx.x % 32 + 32 * i;
      l0[i] = e / (L * L);
      k0[i] = e % (L * L);
      off[i] = 8 * (t.slot_k[k0[i]] * Tile32<WT, L>::kSums + l0[i]);
    }
  }
  // put(l, k, e, v) for the elements with l < rows; e = k + L L l.
  template <typename Put>
  __device__ void line(const Tile32<WT, L>& t, int w, int rows, Put put) const {
    const uint32_t z = t.z_addr + 8 * kLong * w, sw = (w & 1) << 6;
#pragma unroll
    for (int p = 0; p < kLong / kRows; ++p) {
      // Rows l0 + kRows p stored at l ^ 8 (w & 1): l0 < 8 stays in place.
      const uint32_t zp = z + ((8 * kRows * p & ~63u) ^ sw) + (8 * kRows * p & 63u);
#pragma unroll
      for (int i = 0; i < kSteps; ++i) {
        const int l = l0[i] + kRows * p;
        if (l < rows)
          put(l, k0[i], static_cast<int>(threadIdx.x % 32) + 32 * i + kRows * L * L * p, floatsOf(lds64(zp + off[i])));
      }
    }
  }
};

// Momenta of one matrix phase 2 task: 16 of one band, or 8 with all the bands.
template <int NB>
constexpr int kTaskK = NB == 1 ? 16 : 8;

// G0 factor of (k, w) and the band phase at the origin site, for the FFT forms.
__device__ inline double2 originPhase(const double2* __restrict__ Fb, int k, int nc, int r0) {
  return Fb[k * nc + r0];
}

// Row step.  grid (ceil(n_max / 32), ceil(frequencies / WT), n_sectors); X'(row - row0, j) at
// x_off + j rows + row - row0.  L: cluster FFT (4, 6) or 0; NB: bands (1, 2, 3), 0 for any number.
template <int WT, int L, int NB>
__global__ void __launch_bounds__(Tile32<WT, L>::kThreads, Tile32<WT, L>::kRowResident)
rowTransform32Kernel(const TpDims dims, const SectorDesc* __restrict__ sectors, const int* __restrict__ row_start,
                     const float2* __restrict__ T2, const float* __restrict__ Ms, int Kr,
                     const double2* __restrict__ Fb, const double2* __restrict__ G0,
                     const __grid_constant__ ColFft fft, int w_lo,
                     float2* __restrict__ Xp) {
  using T = Tile32<WT, L>;
  const SectorDesc sd = sectors[blockIdx.z];
  const int n = sd.n, j0 = blockIdx.x * kLong, nw_ext = dims.nw_ext, w0 = w_lo + blockIdx.y * WT;
  if (j0 >= n)
    return;
  const int R = dims.R, nb = NB ? NB : dims.nb, nc = dims.nc;
  const long rows = static_cast<long>(R) * (nw_ext - w_lo);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T tile(smem_raw, dims);
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const double2* g0s = G0 + static_cast<long>(sd.spin) * nw_ext * nc * nb * nb;
  const double norm = -1.0 / nc;
  tile.fill(dims, Fb, row_start + sd.orb_off, fft, [&](int w, int k) {
    const double2 g = g0s[k + nc * min(w0 + w, nw_ext - 1)], f = originPhase(Fb, k, nc, fft.r0);
    return make_float2(static_cast<float>(norm * (g.x * f.x - g.y * f.y)),
                       static_cast<float>(norm * (g.x * f.y + g.y * f.x)));
  });

  // Phase 1: lane l copies M(i .. i + 3, j0 + l), then two frequencies of one of the four vertices' twiddles (past
  // the edge the last ones, unused).
  constexpr int kHalfW = WT / 2;
  const float* msrc = Ms + (static_cast<long>(blockIdx.z) * Kr + j0 + lane) * Kr;
  const float2* tsrc = T2 + static_cast<long>(sd.vtx_off) * nw_ext + min(w0 + 2 * (lane % kHalfW), nw_ext - 2);
  const int l8 = lane % 8, wq = lane / 8;  // this lane's sums: columns l8 + 8 a, frequencies wq + 4 b
  Pair acc[4][T::kSub];
  const float* mp = nullptr;
  const float2* tp = nullptr;
  tile.template orbitals<kRowV, true>(
      dims.n_orb,
      [&](int g) {
        mp = msrc + g;
        tp = tsrc + static_cast<long>(g + lane / kHalfW) * nw_ext;
      },
      [&](uint32_t slot) {
        cpAsync16(slot + 16 * lane, mp);
        if (lane < kRowV * kHalfW)
          cpAsync16(slot + 512 + 16 * lane, tp);
        mp += kRowV;
        tp += kRowV * nw_ext;
      },
      [&](uint32_t slot, int lo, int hi, auto first) {
        const uint32_t ma = slot + 16 * l8, ta = slot + 512 + 8 * wq;
        ulonglong2 m4[4];
        m4[0] = lds128<0>(ma);
        m4[1] = lds128<128>(ma);
        m4[2] = lds128<256>(ma);
        m4[3] = lds128<384>(ma);
        bool fresh = decltype(first)::value;
#pragma unroll
        for (int u = 0; u < kRowV; ++u) {
          if (u < lo || u >= hi)
            continue;
          Pair t[T::kSub];
#pragma unroll
          for (int b = 0; b < T::kSub; ++b)
            t[b] = lds64(ta + 8 * (WT * u + 4 * b));
#pragma unroll
          for (int a = 0; a < 4; ++a) {
            const float2 m2 = floatsOf(u < 2 ? m4[a].x : m4[a].y);
            const float x = (u & 1) ? m2.y : m2.x;
            const Pair m = pairOf(x, x);
#pragma unroll
            for (int b = 0; b < T::kSub; ++b) {
              if (fresh)
                acc[a][b] = mul2(t[b], m);
              else
                fma2(acc[a][b], t[b], m);
            }
          }
          fresh = false;
        }
      },
      [&](uint32_t z) {
        const uint32_t za = z + 8 * (wq * kLong + l8);
        const uint32_t sw = (wq & 1) << 6;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const uint32_t zi = za + ((64u * a) ^ sw);
#pragma unroll
          for (int b = 0; b < T::kSub; ++b)
            sts64(zi + 32 * kLong * b, acc[a][b]);
        }
      });

  // Phase 2: cluster transform, left G0 and -1/Nc.
  float2* out = Xp + sd.x_off;
  if constexpr (L > 0) {
    const Drain<WT, L> drain(tile);
    for (int wl = warp; wl < WT && w0 + wl < nw_ext; wl += T::kWarps) {
      fftLine<1>(tile, wl);
      float2* o = out + j0 * rows + static_cast<long>(w0 + wl - w_lo) * R;
      drain.line(tile, wl, n - j0, [&](int l, int k, int, float2 v) { o[l * rows + k] = v; });
    }
  }
  else {
    const int k_tasks = (nc + kTaskK<NB> - 1) / kTaskK<NB>;
    for (int task = warp; task < 2 * WT * k_tasks; task += T::kWarps) {
      const int wl = (task / 2) % WT, l0 = (task & 1) * 16 + lane / 8, k0 = task / (2 * WT) * kTaskK<NB>, w = w0 + wl;
      if (w >= nw_ext)
        continue;
      const double2* g0 = g0s + static_cast<long>(w) * nc * nb * nb;  // (ba, bb, k)
      auto g0n = [&](int i) { return make_float2(static_cast<float>(norm * g0[i].x), static_cast<float>(norm * g0[i].y)); };
      auto put = [&](int i, int b1, int k, float2 v) {
        const int j = j0 + l0 + 4 * i;
        if (j < n)
          out[j * rows + static_cast<long>(w - w_lo) * R + b1 + nb * k] = v;
      };
      if constexpr (NB == 1) {
        auto momenta = [&](auto kc) {
          constexpr int KC = decltype(kc)::value;
          float2 s[4][KC];
          tile.template clusterSum<false, KC>(s, dims, 1, 0, wl, l0, k0);
#pragma unroll
          for (int c = 0; c < KC; ++c) {
            const int k = k0 + lane % 8 + 8 * c;
            if (k >= nc)
              continue;
            const float2 g = g0n(k);
#pragma unroll
            for (int i = 0; i < 4; ++i)
              put(i, 0, k, cmul(g, s[i][c]));
          }
        };
        if (nc <= 8)  // half of sixteen momenta would be padding
          momenta(std::integral_constant<int, 1>{});
        else
          momenta(std::integral_constant<int, 2>{});
      }
      else if constexpr (NB > 1) {
        float2 s[NB][4][1];
#pragma unroll
        for (int b = 0; b < NB; ++b)
          tile.template clusterSum<false, 1>(s[b], dims, NB, b, wl, l0, k0);
        const int k = k0 + lane % 8;
        if (k < nc) {
#pragma unroll
          for (int b1 = 0; b1 < NB; ++b1) {
            float2 g[NB];
#pragma unroll
            for (int b = 0; b < NB; ++b)
              g[b] = g0n(b1 + NB * (b + NB * k));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float2 v = cmul(g[0], s[0][i][0]);
#pragma unroll
              for (int b = 1; b < NB; ++b)
                cfma(v, g[b], s[b][i][0]);
              put(i, b1, k, v);
            }
          }
        }
      }
      else {
        const int k = k0 + lane % 8;
        for (int b1 = 0; b1 < nb; ++b1) {
          float2 v[4] = {};
          for (int b = 0; b < nb; ++b) {
            float2 s[4][1];
            tile.template clusterSum<false, 1>(s, dims, nb, b, wl, l0, k0);
            const float2 g = g0n(b1 + nb * (b + nb * min(k, nc - 1)));
#pragma unroll
            for (int i = 0; i < 4; ++i)
              cfma(v[i], g, s[i][0]);
          }
          if (k < nc)
#pragma unroll
            for (int i = 0; i < 4; ++i)
              put(i, b1, k, v[i]);
        }
      }
    }
  }
}

// v + beta g, rounded once: beta and g are no FP32 numbers, and beta's rounding would be in every delta term alike.
__device__ inline float2 addDelta(float2 v, double beta, double2 g) {
  return make_float2(static_cast<float>(fma(beta, g.x, static_cast<double>(v.x))),
                     static_cast<float>(fma(beta, g.y, static_cast<double>(v.y))));
}

// Column step.  grid (ceil(rows / 32), ceil(NwExt / WT), n_sectors), rows = D - row0.  gmax (or null):
// [2 slot + spin] raised to the sector's largest |Re|, |Im| of G (float bits).
template <int WT, int L, int NB>
__global__ void __launch_bounds__(Tile32<WT, L>::kThreads, Tile32<WT, L>::kColResident)
colTransform32Kernel(const TpDims dims, const SectorDesc* __restrict__ sectors, const int* __restrict__ col_start,
                     const float4* __restrict__ T4, const double2* __restrict__ Fb, const double2* __restrict__ G0,
                     const __grid_constant__ ColFft fft, int row0, const float2* __restrict__ Xp, float2* __restrict__ G,
                     long g_sector_stride, int* __restrict__ gmax) {
  using T = Tile32<WT, L>;
  const SectorDesc sd = sectors[blockIdx.z];
  const int nw_ext = dims.nw_ext, R = L ? L * L : dims.R, nb = NB ? NB : dims.nb, nc = L ? L * L : dims.nc;
  const int rows = R * nw_ext - row0, t0 = blockIdx.x * kLong, w0 = blockIdx.y * WT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T tile(smem_raw, dims);
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const double2* g0s = G0 + static_cast<long>(sd.spin) * nw_ext * nc * nb * nb;
  tile.fill(dims, Fb, col_start + sd.orb_off, fft, [&](int w, int k) {
    const double2 g = g0s[k + nc * min(w0 + w, nw_ext - 1)], f = originPhase(Fb, k, nc, fft.r0);
    return make_float2(static_cast<float>(g.x * f.x + g.y * f.y), static_cast<float>(g.y * f.x - g.x * f.y));
  });

  // Phase 1: of the two vertices of a slot, half a warp copies X' (two rows a lane) and WT lanes the doubled
  // twiddles.
  const float2* xsrc = Xp + sd.x_off + min(t0 + 2 * (lane % 16), rows - 2);
  const float4* tsrc = T4 + static_cast<long>(sd.vtx_off) * nw_ext + min(w0 + lane % WT, nw_ext - 1);
  const int l8 = lane % 8, wq = lane / 8;  // this lane's sums: rows l8 + 8 a, frequencies wq + 4 b
  Pair ac[4][T::kSub], as[4][T::kSub];     // X' c and X' s
  const float2* xp = nullptr;
  const float4* tp = nullptr;
  tile.template orbitals<kColV, false>(
      dims.n_orb,
      [&](int g) {
        xp = xsrc + static_cast<long>(g + lane / 16) * rows;
        tp = tsrc + static_cast<long>(g + lane / WT) * nw_ext;
      },
      [&](uint32_t slot) {
        cpAsync16(slot + 16 * lane, xp);
        if (lane < kColV * WT)
          cpAsync16(slot + 512 + 16 * lane, tp);
        xp += kColV * rows;
        tp += kColV * nw_ext;
      },
      [&](uint32_t slot, int, int hi, auto first) {
        const uint32_t xa = slot + 8 * l8, ta = slot + 512 + 16 * wq;
#pragma unroll
        for (int u = 0; u < kColV; ++u) {
          if (u >= hi)
            continue;
          constexpr bool kFirst = decltype(first)::value;
          Pair x[4];
#pragma unroll
          for (int a = 0; a < 4; ++a)
            x[a] = lds64(xa + 256 * u + 64 * a);
#pragma unroll
          for (int b = 0; b < T::kSub; ++b) {
            const ulonglong2 t = lds128(ta + 16 * (WT * u + 4 * b));
#pragma unroll
            for (int a = 0; a < 4; ++a) {
              if (kFirst && u == 0) {
                ac[a][b] = mul2(x[a], t.x);
                as[a][b] = mul2(x[a], t.y);
              }
              else {
                fma2(ac[a][b], x[a], t.x);
                fma2(as[a][b], x[a], t.y);
              }
            }
          }
        }
      },
      [&](uint32_t z) {
        const uint32_t za = z + 8 * (wq * kLong + l8);
        const uint32_t sw = (wq & 1) << 6;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const uint32_t zi = za + ((64u * a) ^ sw);
#pragma unroll
          for (int b = 0; b < T::kSub; ++b) {
            const float2 c = floatsOf(ac[a][b]), sn = floatsOf(as[a][b]);
            sts64(zi + 32 * kLong * b, pairOf(c.x + sn.y, c.y - sn.x));  // X' conj T
          }
        }
      });

  // Phase 2: cluster transform with conjugate phases, right G0, delta term.
  float2* out = G + g_sector_stride * (2 * sd.slot + sd.spin);
  float gabs = 0.f;
  auto note = [&](float2 v) { gabs = fmaxf(gabs, fmaxf(fabsf(v.x), fabsf(v.y))); };
  if constexpr (L > 0) {
    // The tile's rows lie in one run of G per w1: element e of a line is at first + e, after the first split
    // elements jump further, and so on every R rows.
    const int row_a = row0 + t0, w1_a = row_a / R;
    const long jump = static_cast<long>(nw_ext - 1) * R * R;
    const int split = (R - (row_a - w1_a * R)) * R;
    const Drain<WT, L> drain(tile);
    for (int wl = warp; wl < WT && w0 + wl < nw_ext; wl += T::kWarps) {
      const int w2 = w0 + wl;
      fftLine<-1>(tile, wl);
      {
        const int row = row_a + lane, w1 = row / R, k1 = row - w1 * R;
        if (w1 == w2) {
          const double2 g = g0s[k1 + nc * w2];
          const uint32_t at = tile.lineAddr(wl, lane) + 8 * T::kSums * tile.slot_k[k1];
          const float2 z = floatsOf(lds64(at));
          const float2 v = addDelta(z, dims.beta, g);
          sts64(at, pairOf(v.x, v.y));
        }
      }
      __syncwarp();
      float2* o = out + ((static_cast<long>(w1_a) * nw_ext + w2) * R + row_a - w1_a * R) * R;
      drain.line(tile, wl, rows - t0, [&](int, int, int e, float2 v) {
        note(v);
        // At most three runs of 16 rows, two of 36, meet a tile of 32.
        float2* run = e >= split ? o + jump : o;
        if (L == 4 && e >= split + R * R)
          run += jump;
        run[e] = v;
      });
    }
  }
  else {
    const int k_tasks = (nc + kTaskK<NB> - 1) / kTaskK<NB>;
    for (int task = warp; task < 2 * WT * k_tasks; task += T::kWarps) {
      const int wl = (task / 2) % WT, l0 = (task & 1) * 16 + lane / 8, k0 = task / (2 * WT) * kTaskK<NB>, w2 = w0 + wl;
      if (w2 >= nw_ext)
        continue;
      const double2* g0 = g0s + static_cast<long>(w2) * nc * nb * nb;  // (ba, bb, k)
      auto put = [&](int i, int b2, int k2, float2 v) {
        if (t0 + l0 + 4 * i >= rows)
          return;
        const int row = row0 + t0 + l0 + 4 * i;
        const int w1 = row / R, r = row - w1 * R, k1 = r / nb;
        if (w1 == w2 && k1 == k2)
          v = addDelta(v, dims.beta, g0[(r - nb * k1) + nb * (b2 + nb * k2)]);
        note(v);
        out[((static_cast<long>(w1) * nw_ext + w2) * R + r) * R + b2 + nb * k2] = v;
      };
      if constexpr (NB == 1) {
        auto momenta = [&](auto kc) {
          constexpr int KC = decltype(kc)::value;
          float2 s[4][KC];
          tile.template clusterSum<true, KC>(s, dims, 1, 0, wl, l0, k0);
#pragma unroll
          for (int c = 0; c < KC; ++c) {
            const int k = k0 + lane % 8 + 8 * c;
            if (k >= nc)
              continue;
            const float2 g = to_f2(g0[k]);
#pragma unroll
            for (int i = 0; i < 4; ++i)
              put(i, 0, k, cmul(s[i][c], g));
          }
        };
        if (nc <= 8)  // half of sixteen momenta would be padding
          momenta(std::integral_constant<int, 1>{});
        else
          momenta(std::integral_constant<int, 2>{});
      }
      else if constexpr (NB > 1) {
        float2 s[NB][4][1];
#pragma unroll
        for (int b = 0; b < NB; ++b)
          tile.template clusterSum<true, 1>(s[b], dims, NB, b, wl, l0, k0);
        const int k = k0 + lane % 8;
        if (k < nc) {
#pragma unroll
          for (int b2 = 0; b2 < NB; ++b2) {
            float2 g[NB];
#pragma unroll
            for (int b = 0; b < NB; ++b)
              g[b] = to_f2(g0[b + NB * (b2 + NB * k)]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float2 v = cmul(s[0][i][0], g[0]);
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
          float2 v[4] = {};
          for (int b = 0; b < nb; ++b) {
            float2 s[4][1];
            tile.template clusterSum<true, 1>(s, dims, nb, b, wl, l0, k0);
            const float2 g = to_f2(g0[b + nb * (b2 + nb * min(k, nc - 1))]);
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
  if (gmax) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
      gabs = fmaxf(gabs, __shfl_xor_sync(0xffffffffu, gabs, off));
    if (lane == 0 && gabs > 0.f)
      atomicMax(gmax + 2 * sd.slot + sd.spin, __float_as_int(gabs));
  }
}

constexpr size_t kMaxSmem = 227 * 1024;

// The cluster FFT that applies: 4, 6, or 0 (matrix).
int fftLength(const TpDims& d, const ColFft& fft) {
  return d.nb == 1 && fft.on && (fft.L == 4 || fft.L == 6) ? fft.L : 0;
}

template <int WT>
size_t tileBytes(const TpDims& d, int L) {
  return L == 4 ? Tile32<WT, 4>::bytes(d) : L == 6 ? Tile32<WT, 6>::bytes(d) : Tile32<WT, 0>::bytes(d);
}

// Frequencies per CTA: 16 or 8, which the tuner chooses between (every element is the same sum in the same
// order); 8 or 4 alone where the wider tile does not fit in shared memory.
int tileWidth(const FrontendArgs& a, int L, const char* family, LaunchTuner::Pick& pk, cudaStream_t stream) {
  const bool fit16 = tileBytes<16>(a.dims, L) <= kMaxSmem, fit8 = tileBytes<8>(a.dims, L) <= kMaxSmem;
  pk = tunePick(a.tuner, tuneKey(family, a.dims.nb, a.dims.nc, a.dims.nw_ext, a.n_max, a.n_sectors, 4),
                fit16 ? 2 : 1, stream);
  return fit16 && pk.choice == 0 ? 16 : fit8 ? 8 : 4;
}

template <int WT, int L, int NB>
void launchRow(const FrontendArgs& a, const Front32Workspace& w, int w_lo, cudaStream_t stream) {
  const TpDims& d = a.dims;
  auto k = rowTransform32Kernel<WT, L, NB>;
  constexpr int threads = Tile32<WT, L>::kThreads;
  const size_t smem = Tile32<WT, L>::bytes(d);
  DCAACC_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  DCAACC_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         int(cudaSharedmemCarveoutMaxShared)));
  k<<<dim3(ceil_div(a.n_max, kLong), ceil_div(d.nw_ext - w_lo, WT), a.n_sectors), threads, smem, stream>>>(
      d, a.sectors, a.row_start, w.T2, w.Ms, w.Kr, a.Fb, a.G0, w.fft, w_lo, w.X);
  DCAACC_LAUNCH_CHECK();
}

template <int WT, int L, int NB>
void launchCol(const FrontendArgs& a, const Front32Workspace& w, int row0, float2* G, long g_sector_stride, int* gmax,
               cudaStream_t stream) {
  const TpDims& d = a.dims;
  auto k = colTransform32Kernel<WT, L, NB>;
  constexpr int threads = Tile32<WT, L>::kThreads;
  const size_t smem = Tile32<WT, L>::bytes(d);
  DCAACC_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  DCAACC_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         int(cudaSharedmemCarveoutMaxShared)));
  k<<<dim3(ceil_div(long(d.R) * d.nw_ext - row0, kLong), ceil_div(d.nw_ext, WT), a.n_sectors), threads, smem, stream>>>(
      d, a.sectors, a.col_start, w.T4, a.Fb, a.G0, w.fft, row0, w.X, G, g_sector_stride, gmax);
  DCAACC_LAUNCH_CHECK();
}

// Calls f.template operator()<WT, L, NB>() for the runtime values.
template <int WT, typename F>
void dispatchLNb(int L, int nb, F f) {
  if (L == 4)
    f.template operator()<WT, 4, 1>();
  else if (L == 6)
    f.template operator()<WT, 6, 1>();
  else if (nb == 1)
    f.template operator()<WT, 0, 1>();
  else if (nb == 2)
    f.template operator()<WT, 0, 2>();
  else if (nb == 3)
    f.template operator()<WT, 0, 3>();
  else
    f.template operator()<WT, 0, 0>();
}
template <typename F>
void dispatch(int wt, int L, int nb, F f) {
  if (wt == 16)
    dispatchLNb<16>(L, nb, f);
  else if (wt == 8)
    dispatchLNb<8>(L, nb, f);
  else
    dispatchLNb<4>(L, nb, f);
}

struct RowLauncher {
  const FrontendArgs& a;
  const Front32Workspace& w;
  int w_lo;
  cudaStream_t stream;
  template <int WT, int L, int NB>
  void operator()() const {
    launchRow<WT, L, NB>(a, w, w_lo, stream);
  }
};
struct ColLauncher {
  const FrontendArgs& a;
  const Front32Workspace& w;
  int row0;
  float2* G;
  long g_sector_stride;
  int* gmax;
  cudaStream_t stream;
  template <int WT, int L, int NB>
  void operator()() const {
    launchCol<WT, L, NB>(a, w, row0, G, g_sector_stride, gmax, stream);
  }
};

}  // namespace

bool front32Applies(const TpDims& d, int max_order) {
  return tileBytes<4>(d, 0) <= kMaxSmem && size_t(max_order) * sizeof(float) <= 200 * 1024;
}

int launchFront32Prep(const FrontendArgs& a, const Front32Workspace& w, cudaStream_t stream) {
  const TpDims& d = a.dims;
  if (a.n_max == 0)
    return 0;
  const unsigned gx = static_cast<unsigned>(ceil_div(long(a.n_max) * (d.nw_ext / 2), 256));
  twiddle32Kernel<<<dim3(gx, a.n_sectors), 256, 0, stream>>>(a.sectors, a.tau, a.perm_r, a.perm_c, w.T2, w.T4, d.nw_ext,
                                                             d.beta);
  DCAACC_LAUNCH_CHECK();
  // Eight warps a block, fewer where their rows do not fit in shared memory.
  const int floats = std::min(a.n_max, w.Kr);
  int warps = kSortWarps;
  while (warps > 1 && size_t(warps) * floats * sizeof(float) > 100 * 1024)
    warps /= 2;
  const size_t smem = size_t(warps) * floats * sizeof(float);
  DCAACC_CUDA_CHECK(cudaFuncSetAttribute(sortM32Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  sortM32Kernel<<<dim3(ceil_div(a.n_max, warps), a.n_sectors), 32 * warps, smem, stream>>>(a.sectors, a.perm_r, a.perm_c,
                                                                                         w.Kr, floats, w.Ms);
  DCAACC_LAUNCH_CHECK();
  return 2;
}

void launchFront32Row(const FrontendArgs& a, const Front32Workspace& w, cudaStream_t stream) {
  if (a.n_max == 0)
    return;
  const int L = fftLength(a.dims, w.fft);
  LaunchTuner::Pick pk;
  const int wt = tileWidth(a, L, "row32", pk, stream);
  dispatch(wt, L, a.dims.nb, RowLauncher{a, w, a.dims.half_g ? a.dims.nw_ext / 2 : 0, stream});
  tuneEnd(a.tuner, pk, stream);
}

void launchFront32Col(const FrontendArgs& a, const Front32Workspace& w, float2* G, long g_sector_stride, int* gmax,
                      cudaStream_t stream) {
  if (gmax)
    DCAACC_CUDA_CHECK(cudaMemsetAsync(gmax, 0, sizeof(int) * size_t(a.n_sectors), stream));
  const int L = fftLength(a.dims, w.fft);
  const int row0 = a.dims.half_g ? a.dims.R * a.dims.nw_ext / 2 : 0;
  LaunchTuner::Pick pk;
  const int wt = tileWidth(a, L, "col32", pk, stream);
  dispatch(wt, L, a.dims.nb, ColLauncher{a, w, row0, G, g_sector_stride, gmax, stream});
  tuneEnd(a.tuner, pk, stream);
}

}  // namespace dcaacc
