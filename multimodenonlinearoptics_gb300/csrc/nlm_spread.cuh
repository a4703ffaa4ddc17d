// nlm_spread.cuh -- one propagation on a cluster of four, eight or sixteen CTAs with ONE point per thread.
//
// Every CTA holds M = N/C points, one per thread: N = 512 on C = 4 CTAs gives four warps on each of four SMs.
// C = 8 doubles the SMs of a 2048- or 4096-point propagation, and C = 16 (a non-portable cluster size) doubles
// them again for the longest marches of a ragged batch and for full grids.  The transforms:
//   time domain:       CTA c, thread j  <->  point n = c + C t(j),  t(j) = g + G l
//   frequency domain:  CTA c, thread j  <->  bin   k = j + M c
// with l = j mod 32 (lane), g = j / 32 (warp) and G = M / 32 warps: the time ownership strides the
// CTA's points over the lanes so that each warp's 32 points are one decimated sub-sequence.
// forward:  the M-point DFT over the CTA's strided points as 32 x G: a 32-point DFT inside each warp
//           (lanes exchange through shuffles: no shared memory, no barrier), the twiddle W_M^(g l),
//           then a G-point DFT across the warps through shared memory (one barrier: each thread reads its
//           lane's G values and forms its own output); then the twiddle exp(-2 pi i c j / N) and the C-point
//           DFT over the CTAs: every thread pushes its value to all C CTAs through distributed shared
//           memory, and each thread combines the C values of its own column for its CTA's output row;
// inverse:  the C-point inverse DFT over the CTAs first, the conjugate twiddle, then the local inverse
//           (the G-point DFT across warps, the conjugate W_M^(g l), the 32-point DFT in the warps;
//           unscaled, 1/N is in the tables).  It runs the forward transform's parts on values with real and
//           imaginary part swapped.
//
// The values are FP64 on both sides and 64-bit integers inside (nlm_fx.cuh says why and how).  A warp issues one
// FP64 instruction in 64 cycles on its scheduler, so the ~30 of a transform in FP64 took about 1 us however
// few points there were; an IMAD.WIDE or a 64-bit addition takes two cycles.  Every warp scales its 32 points
// by its own exponent (a bound on its 2-norm in half bits, from two warp reductions and no barrier).  These codes
// cross the cluster, in a forward transform while the warps' DFTs run, and each warp then shifts its values to the
// total's exponent.  Starting below 2^59, the norm grows by sqrt(32) in the warps, sqrt(G) across them and sqrt(C)
// across the CTAs, and is shifted back where it would pass 2^61.5 (spread_shift).
// Exchanges over the cluster: each value travels by st.async, which counts its bytes on the receiving warp's
// mbarrier, and a warp waits for the C x 32 values of its own columns.  No barrier of the cluster and no fence
// of earlier global stores: with cluster barriers those were a third of a step.  Two mbarriers per warp and two
// halves of the receive buffer serve the exchanges in turn: a thread writes half n again only after it has
// received exchange n + 1 from the thread that reads that column, which pushed it after reading half n.
// Waits give up after wait.polls polls (kExchangePolls unless the caller limits them) and raise *wait.err.  The thread
// then neither waits nor sends any more (an mbarrier whose phase is open takes no further arrival), so its peers give
// up too, and every CTA runs to the closing cluster barrier.  After it spread_drain waits, again with a limit, for what
// is still on its way into this CTA's memory.
// Shared memory: M twiddles, two M-point exchange buffers (alternating: a thread writes a buffer only after
// the barrier that every reader of that buffer's previous contents has passed), the two halves of C x M values.
// M is a power of two of at least 32, N = C M at most 4096.
#pragma once
#include <climits>

#include <cooperative_groups.h>

#include "nlm_fx.cuh"
#include "nlm_propagate.cuh"

namespace cg = cooperative_groups;

namespace nlm {

constexpr int kSpreadC = 4;
static_assert(kSpreadSmemPerPoint == spread_smem_per_point(kSpreadC), "twiddles, exchange buffers, receive halves");
constexpr int kSpreadA0 = 59;      // log2 bound of a warp's 2-norm on entry
constexpr int kSpreadPeak = 5;     // half bits the norm may stand above it
constexpr int kSpreadZero = -(1 << 20), kSpreadBad = 1 << 20;   // codes of a zero warp, of one with Inf or NaN
constexpr int kSpreadMaxCodes = 4096 / 32 * 4;                  // warps of a cluster times fields

struct SpreadFFT {
  const int4* twM;      // [M] exp(-2 pi i m / M) in Q62, shared memory
  int4 twC;             // exp(-2 pi i c j / N) of this thread (rank c, thread j)
  int4 wgl;             // W_M^(g l)
  int4 w16, w8, w4;     // the lane's factors of the warp stages of 16, 8 and 4
  int4* buf;            // [2][K][M] exchange buffers of the local transform
  int4* recv;           // [2][C][K][M] cluster receive buffers
  int* ecode;           // [2][K][C][G] exponent codes of the cluster's warps
  unsigned ebar;        // shared address of the CTA's two mbarriers for them
  int ephase;           // the next of the two
  unsigned bar;         // shared address of this warp's two mbarriers
  unsigned parity;      // bits 0, 1: the phases that the warp's mbarriers complete next; 2, 3: the codes'
  ExchangeWait wait;
  int dead;             // not 0: the exchange of bit dead - 1 of parity has timed out; no more waiting, no more sending
  int M, rank, j;
  int l, g, t;          // lane, warp and local time index g + (M / 32) l of this thread
  int sel, phase;       // next exchange buffer / receive half
  int base;             // cluster rank of the group's first CTA (clusters holding two groups of four)
};

__device__ __forceinline__ unsigned spread_saddr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// Sets up the spread transform of this CTA: the M-point twiddles (every C-th entry of the N-point Q62
// table `tw`), this thread's factors and the warps' mbarriers.  The cluster must pass a barrier (cl.sync) after
// it and before the first exchange, and one after the last.  K: fields transformed
// together (the _k forms), which sizes the exchange and receive buffers.
template <int C = kSpreadC, int K = 1>
__device__ __forceinline__ void spread_init(SpreadFFT& f, double2* smem, const int4* __restrict__ tw, int M, int rank,
                                            ExchangeWait wait) {
  __shared__ int s_ecode[2 * kSpreadMaxCodes];
  __shared__ unsigned long long s_bar[2 * 16 + 2];
  f.M = M;
  f.rank = rank;
  f.j = threadIdx.x;
  f.l = f.j & 31;
  f.g = f.j >> 5;
  f.t = f.g + (M >> 5) * f.l;
  f.sel = 0;
  f.phase = 0;
  f.base = 0;
  f.ecode = s_ecode;
  f.ephase = 0;
  f.bar = spread_saddr(s_bar + 2 * f.g);
  f.ebar = spread_saddr(s_bar + 2 * 16);
  f.parity = 0;
  f.wait = wait;
  f.dead = 0;
  int4* twM = reinterpret_cast<int4*>(smem);
  f.buf = twM + M;
  f.recv = twM + (1 + 2 * K) * M;
  for (int k = threadIdx.x; k < M; k += blockDim.x) twM[k] = tw[(long long)k * C];
  f.twM = twM;
  f.twC = tw[(long long)rank * f.j];
  if (f.l < 2) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(f.bar + 8 * f.l) : "memory");
    if (f.g == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(f.ebar + 8 * f.l) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  // decimation in frequency: the upper lane of a pair takes W_2s^(l mod s), the lower one 1
  auto lane = [&](int s) { return twM[(f.l & s) ? (f.l & (s - 1)) * (M / (2 * s)) : 0]; };
  f.w16 = lane(16);
  f.w8 = lane(8);
  f.w4 = lane(4);
  f.wgl = twM[f.g * f.l];
}

// Whether the mbarrier's phase `par` completes within `polls` polls.
__device__ __forceinline__ bool spread_poll(unsigned bar, unsigned par, int polls) {
  for (int n = 0; n < polls; n++) {
    unsigned ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(par)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// Waits for the phase of an mbarrier that bit `bit` of f.parity names, and moves on to the next one.
__device__ __forceinline__ void spread_wait(SpreadFFT& f, unsigned bar, int bit) {
  if (f.dead) return;
  if (spread_poll(bar, (f.parity >> bit) & 1, f.wait.polls)) {
    f.parity ^= 1u << bit;
    return;
  }
  f.dead = 1 + bit;
  if (f.wait.err) *(volatile int*)f.wait.err = 1;
}

// After the closing cluster barrier: all that the cluster sends has been sent.  A thread that has waited for every
// exchange has received all of it; one that gave up waits for that exchange, and 64 us for any that a peer sent after
// it, before its CTA's memory is given up.
__device__ __forceinline__ void spread_drain(const SpreadFFT& f) {
  if (!f.dead) return;
  const int bit = f.dead - 1;
  spread_poll(bit < 2 ? f.bar + 8 * bit : f.ebar + 8 * (bit - 2), (f.parity >> bit) & 1, kExchangePolls);
  for (int n = 0; n < 64; n++) __nanosleep(1000);
}

// Local time index of thread j of a CTA of M threads (the time ownership above).
__device__ __forceinline__ int spread_time_index(int j, int M) { return (j >> 5) + (M >> 5) * (j & 31); }

__device__ __forceinline__ fxc spread_shfl(fxc v, int src) {
  return fxc{__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src)};
}
__device__ __forceinline__ fxc spread_swap(fxc v) { return fxc{v.y, v.x}; }

// Places to shift before a stage that adds `grow` half bits to a norm standing `level` half bits above 2^A0.
__device__ __forceinline__ int spread_shift(int level, int grow) { return max(0, (level + grow - kSpreadPeak + 1) >> 1); }

struct SpreadPoint {
  fxc y;
  int h;
};

// The point as integers below the warp's exponent, and the warp's code h (norm^2 < 2^h).
__device__ __forceinline__ SpreadPoint spread_enter(double2 x) {
  auto top = [](double2 v) {
    return __reduce_max_sync(0xffffffffu, max((unsigned)__double2hiint(v.x) & 0x7fffffffu, (unsigned)__double2hiint(v.y) & 0x7fffffffu));
  };
  int e = (int)(top(x) >> 20), lift = 0;
  if (e < 256) {   // tiny or zero: lifted, so that exponents and conversions stay in range
    x = cscale(x, kFxLift);
    e = (int)(top(x) >> 20);
    lift = 900;
  }
  const int off = (127 << 20) - (e << 20);
  const float p = __int_as_float(max((__double2hiint(x.x) & 0x7fffffff) + off, 0) << 3);
  const float q = __int_as_float(max((__double2hiint(x.y) & 0x7fffffff) + off, 0) << 3);
  const unsigned S = __reduce_add_sync(0xffffffffu, (unsigned)(fmaf(p, p, q * q) * 65536.f) + 2u);
  const int h = 2 * (e - 1023) + 16 - __clz((int)S);   // S < 2^(32 - clz), in units of 2^-16
  const int rel = 62 - kSpreadA0 + 1023 + ((h + 1) >> 1);
  const fxc y = e == 0 ? fxc{0, 0} : fxc{fx_from(x.x, rel), fx_from(x.y, rel)};
  return SpreadPoint{y, e == 0 ? kSpreadZero : e == 0x7ff ? kSpreadBad : h - 2 * lift};
}

// y 2^(ceil(h / 2) - A0 + places) as FP64
__device__ __forceinline__ double2 spread_leave(fxc y, int h, int places) {
  const int k = ((h + 1) >> 1) - kSpreadA0 + places;
  const bool fast = k > -1000 && k < 900;
  double2 x = make_double2(fx_to(y.x, fast ? k : 0), fx_to(y.y, fast ? k : 0));
  if (!fast) {
    if (h > kSpreadBad / 2) x.x = x.y = __longlong_as_double(0x7ff8000000000000LL);
    else if (h < kSpreadZero / 2) x = czero();
    else x = make_double2(scalbn(x.x, k), scalbn(x.y, k));
  }
  return x;
}

__device__ __forceinline__ fxc spread_align(fxc v, int r) { return fxc{fx_align(v.x, r), fx_align(v.y, r)}; }

// Output r of the P-point DFT of v: sum_c W_P^(r c) v_c.  r is the same for the whole warp.
template <int P>
__device__ __forceinline__ fxc spread_combine(const fxc (&v)[P], int r, const int4* __restrict__ twM, int M) {
  const bool odd = (r & 1) != 0;
  auto pm = [odd](fxc a, fxc b) { return odd ? fxsub(a, b) : fxadd(a, b); };   // a + (-1)^r b
  auto quarter = [r](fxc a, fxc b) {                                         // a + (-i)^r b
    switch (r & 3) {
      case 0: return fxadd(a, b);
      case 1: return fxc{a.x + b.y, a.y - b.x};
      case 2: return fxsub(a, b);
      default: return fxc{a.x - b.y, a.y + b.x};
    }
  };
  if constexpr (P == 2) {
    return pm(v[0], v[1]);
  } else if constexpr (P == 4) {
    return quarter(pm(v[0], v[2]), pm(v[1], v[3]));
  } else if constexpr (P == 8) {
    // u_c = v_c + (-1)^r v_(c+4); w_c = u_c + W_4^r u_(c+2); out = w_0 + W_8^r w_1
    fxc u[4];
#pragma unroll
    for (int c = 0; c < 4; c++) u[c] = pm(v[c], v[c + 4]);
    return fxadd(quarter(u[0], u[2]), fx_cmul(quarter(u[1], u[3]), twM[(r & 7) * (M / 8)], 2));
  } else {
    static_assert(P == 16, "2, 4, 8 or 16 points");
    fxc u[8], w[4];
#pragma unroll
    for (int c = 0; c < 8; c++) u[c] = pm(v[c], v[c + 8]);
#pragma unroll
    for (int c = 0; c < 4; c++) w[c] = quarter(u[c], u[c + 4]);
    const int4 w8 = twM[(r & 7) * (M / 8)];
    const fxc y0 = fxadd(w[0], fx_cmul(w[2], w8, 2)), y1 = fxadd(w[1], fx_cmul(w[3], w8, 2));
    return fxadd(y0, fx_cmul(y1, twM[r * (M / 16)], 2));
  }
}

// Output r of the P-point DFT of the P values at p, p + stride, ... in shared memory.
template <int P>
__device__ __forceinline__ fxc spread_gather(const int4* p, int stride, int r, const int4* twM, int M) {
  fxc v[P];
#pragma unroll
  for (int c = 0; c < P; c++) v[c] = fx_unpack(p[c * stride]);
  return spread_combine<P>(v, r, twM, M);
}
// sixteen warps: a call, since its code in every transform of every kernel would be most of the library
static __device__ __noinline__ fxc spread_gather16(const int4* p, int r, const int4* twM, int M) {
  return spread_gather<16>(p, 32, r, twM, M);
}
__device__ __forceinline__ fxc spread_gather_warps(const int4* p, int r, const int4* twM, int M) {
  switch (M >> 5) {
    case 2: return spread_gather<2>(p, 32, r, twM, M);
    case 4: return spread_gather<4>(p, 32, r, twM, M);
    case 8: return spread_gather<8>(p, 32, r, twM, M);
    default: return spread_gather16(p, r, twM, M);
  }
}

// 32-point DFT over the lanes: lane l holds element l on entry and bin l on return.  Decimation in
// frequency: stage s pairs lane l with l ^ s, the lower lane takes a + b, the upper (a - b) W_2s^(l mod s);
// then every lane takes its bit-reversed lane's value.  The norm grows by sqrt(32).
__device__ __forceinline__ fxc spread_warp_dft(fxc x, int4 w16, int4 w8, int4 w4, int l) {
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) {
    const long long neg = (l & s) ? -1 : 0;
    const fxc p = fxc{__shfl_xor_sync(0xffffffffu, x.x, s), __shfl_xor_sync(0xffffffffu, x.y, s)};
    fxc t = fxc{p.x + ((x.x ^ neg) - neg), p.y + ((x.y ^ neg) - neg)};
    if (s >= 4) t = fx_cmul(t, s == 16 ? w16 : s == 8 ? w8 : w4, 2);
    if (s == 2 && (l & 3) == 3) t = fxc{t.y, -t.x};   // W_4 = -i
    x = t;
  }
  return spread_shfl(x, (int)(__brev((unsigned)l) >> 27));
}

// y[m] = f(m, y[m]) for K fields.  Up to three in one stretch of code; four two at a time, since a step of four in one
// stretch (about 100 KB of instructions) does not stay in the instruction cache and each warp fetches it again: Chi2SHGOPA,
// 1024 points on eight CTAs, 31.2 us a step in one stretch, 24.2 by one mode at a time (K = 1), 22.8 so; 512 points 23.8,
// 20.9 and 19.7; only at 128 points, one warp per CTA, is one stretch the faster (16.0 against 16.5).
template <int K, class F>
__device__ __forceinline__ void spread_each(fxc (&y)[K], F f) {
  if constexpr (K < 4) {
#pragma unroll
    for (int m = 0; m < K; m++) y[m] = f(m, y[m]);
  } else {
    static_assert(K % 2 == 0, "two fields at a time");
#pragma unroll 1
    for (int m = 0; m < K; m += 2) {
      const fxc a = f(m, y[0]), b = f(m + 1, y[1]);
#pragma unroll
      for (int q = 0; q < K - 2; q++) y[q] = y[q + 2];
      y[K - 2] = a;
      y[K - 1] = b;
    }
  }
}

// G-point DFT across the warps of a CTA for every lane.
template <int K>
__device__ __forceinline__ void spread_cross(SpreadFFT& f, fxc (&x)[K]) {
  if (f.M == 32) return;   // one warp
  int4* b = f.buf + f.sel * K * f.M;
#pragma unroll
  for (int m = 0; m < K; m++) b[m * f.M + f.j] = fx_pack(x[m]);
  __syncthreads();
  spread_each(x, [&](int m, fxc) { return spread_gather_warps(b + m * f.M + f.l, f.g, f.twM, f.M); });
  f.sel ^= 1;
}

// C-point DFT over the cluster's CTAs, in two halves.  Push: thread j of every CTA sends its value to column j of
// row `rank` in all C CTAs.
template <int C, int K>
__device__ __forceinline__ void spread_push(SpreadFFT& f, const fxc (&y)[K]) {
  static_assert(C == 4 || C == 8 || C == 16, "four, eight or sixteen CTAs");
  if (f.dead) return;
  const int M = f.M;
  const unsigned bar = f.bar + 8 * f.phase;
  const unsigned dst = spread_saddr(f.recv + ((long long)f.phase * C + f.rank) * K * M + f.j);
  if (f.l == 0)
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(C * K * 32 * 16) : "memory");
#pragma unroll
  for (int m = 0; m < K; m++) {
    const int4 out = fx_pack(y[m]);
#pragma unroll
    for (int v = 0; v < C; v++) {
      unsigned rd, rb;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rd) : "r"(dst + 16 * m * M), "r"(f.base + v));
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rb) : "r"(bar), "r"(f.base + v));
      asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(rd),
                   "r"(out.x), "r"(out.y), "r"(out.z), "r"(out.w), "r"(rb)
                   : "memory");
    }
  }
}

// Pull: the C values of this thread's column, combined into output `rank` of their C-point DFT.
template <int C, int K>
__device__ __forceinline__ void spread_pull(SpreadFFT& f, fxc (&y)[K]) {
  const int4* half = f.recv + (long long)f.phase * C * K * f.M;
  spread_wait(f, f.bar + 8 * f.phase, f.phase);
  spread_each(y, [&](int m, fxc) { return spread_gather<C>(half + m * f.M + f.j, K * f.M, f.rank, f.twM, f.M); });
  f.phase ^= 1;
}

// a w / 2^s
__device__ __forceinline__ fxc spread_mul(fxc a, int4 w, int s) { return fx_cmul(a, w, 2 - s); }

// The warps' codes over the cluster: lane v sends the warp's to CTA v, and every warp then knows all C G of them and
// shifts its values to the exponent of the total once.  A forward transform sends them before its warp DFTs and
// needs them after.  The halves of ecode alternate; a warp writes half n again after code exchange n + 1, for which
// every warp of the cluster has read half n.
template <int C, int K>
__device__ __forceinline__ void spread_push_codes(SpreadFFT& f, const int (&h)[K]) {
  if (f.dead) return;
  const int G = f.M >> 5;
  const unsigned bar = f.ebar + 8 * f.ephase;
  if (f.j == 0)
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(C * K * G * 4) : "memory");
  if (f.l < C) {
    const unsigned cd = spread_saddr(f.ecode + ((f.ephase * K) * C + f.rank) * G + f.g);
    unsigned rd, rb;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rd) : "r"(cd), "r"(f.base + f.l));
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rb) : "r"(bar), "r"(f.base + f.l));
#pragma unroll
    for (int m = 0; m < K; m++)
      asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(rd + 4 * m * C * G),
                   "r"(h[m]), "r"(rb)
                   : "memory");
  }
}

// The code of the total of n <= 32 Q warps' codes (lane l takes l, l + 32, ...).
template <int Q>
__device__ __forceinline__ int spread_total(const int* cd, int n, int l) {
  int v[Q], top = kSpreadZero;
#pragma unroll
  for (int q = 0; q < Q; q++) {
    v[q] = l + 32 * q < n ? cd[l + 32 * q] : kSpreadZero;
    top = max(top, v[q]);
  }
  top = __reduce_max_sync(0xffffffffu, top);
  unsigned s = 0;
#pragma unroll
  for (int q = 0; q < Q; q++)
    if (l + 32 * q < n) s += 65536u >> min(top - v[q], 31);
  s = __reduce_add_sync(0xffffffffu, s);
  return top + 16 - __clz((int)(s - 1));   // top + ceil(log2(s / 65536))
}

template <int C, int K>
__device__ __forceinline__ void spread_pull_codes(SpreadFFT& f, fxc (&y)[K], int (&h)[K]) {
  const int n = C * (f.M >> 5);
  const int* cd = f.ecode + f.ephase * K * n;
  spread_wait(f, f.ebar + 8 * f.ephase, 2 + f.ephase);
  f.ephase ^= 1;
#pragma unroll
  for (int m = 0; m < K; m++) {
    const int tot = spread_total<C == 4 ? 2 : 4>(cd + m * n, n, f.l);   // at most 16 warps per CTA, 128 per cluster
    y[m] = spread_align(y[m], min(((tot + 1) >> 1) - ((h[m] + 1) >> 1), 62));
    h[m] = tot;
  }
}

// time-domain ownership -> frequency-domain ownership, K fields together.  Returns in `places` the shifts so far:
// y = X 2^(A0 - ceil(h / 2) - places), h the cluster's code, the norm at most `level` half bits above 2^A0.
template <int C, int K>
__device__ __forceinline__ void spread_forward(SpreadFFT& f, const double2 (&x)[K], fxc (&y)[K], int (&h)[K], int& places,
                                               int& level) {
  const int g = 26 - __clz(f.M), lc = fx_log2(C);   // log2 G: the half bits a G-point DFT adds (M = 32 G)
  const int s1 = spread_shift(5, g), s2 = spread_shift(5 + g - 2 * s1, lc);
#pragma unroll
  for (int m = 0; m < K; m++) {
    const SpreadPoint p = spread_enter(x[m]);
    y[m] = p.y;
    h[m] = p.h;
  }
  spread_push_codes<C, K>(f, h);
  spread_each(y, [&](int, fxc v) { return spread_warp_dft(v, f.w16, f.w8, f.w4, f.l); });
  spread_pull_codes<C, K>(f, y, h);
  spread_each(y, [&](int, fxc v) { return f.g > 0 ? spread_mul(v, f.wgl, s1) : fx_shift(v, s1); });
  spread_cross<K>(f, y);
  spread_each(y, [&](int, fxc v) { return spread_mul(v, f.twC, s2); });
  spread_push<C, K>(f, y);
  spread_pull<C, K>(f, y);
  places = s1 + s2;
  level = 5 + g - 2 * s1 + lc - 2 * s2;
}

// The inverse transform's part after its push (of swapped values): pull, DFT across the warps, in the warps.
// level: of the pushed values.
template <int C, int K>
__device__ __forceinline__ void spread_backward(SpreadFFT& f, fxc (&y)[K], int& places, int level) {
  const int g = 26 - __clz(f.M), lc = fx_log2(C);
  // the last product shifts two places at most: the one before it takes what that leaves
  const int s1 = max(0, (level + lc + g - 3) >> 1), s2 = spread_shift(level + lc + g - 2 * s1, 5);
  spread_pull<C, K>(f, y);
  spread_each(y, [&](int, fxc v) { return spread_mul(v, f.twC, s1); });
  spread_cross<K>(f, y);
  spread_each(y, [&](int, fxc v) {
    return spread_warp_dft(f.g > 0 ? spread_mul(v, f.wgl, s2) : fx_shift(v, s2), f.w16, f.w8, f.w4, f.l);
  });
  places += s1 + s2;
}

template <int C, int K>
__device__ __forceinline__ void spread_fwd_k(SpreadFFT& f, double2 (&x)[K]) {
  fxc y[K];
  int h[K], places, level;
  spread_forward<C, K>(f, x, y, h, places, level);
#pragma unroll
  for (int m = 0; m < K; m++) x[m] = spread_leave(y[m], h[m], places);
}

// frequency-domain ownership -> time-domain ownership (unscaled), K fields.  store(m, v) receives each field's
// frequency-domain value while the exchange is in flight.
template <int C, int K, class Store>
__device__ __forceinline__ void spread_inv_store_k(SpreadFFT& f, double2 (&x)[K], Store store) {
  fxc y[K];
  int h[K], places = 0;
#pragma unroll
  for (int m = 0; m < K; m++) {
    const SpreadPoint p = spread_enter(x[m]);
    y[m] = spread_swap(p.y);
    h[m] = p.h;
  }
  spread_push_codes<C, K>(f, h);
  spread_pull_codes<C, K>(f, y, h);
  spread_push<C, K>(f, y);
#pragma unroll
  for (int m = 0; m < K; m++) store(m, x[m]);
  spread_backward<C, K>(f, y, places, 0);
#pragma unroll
  for (int m = 0; m < K; m++) x[m] = spread_leave(spread_swap(y[m]), h[m], places);
}

// Forward transform, factors, inverse transform, with the values in integers throughout: one exponent decision
// and one conversion each way for both transforms.  fac: this thread's Q62 factors per field (relative to 2^et).
// want: spec(m, v) receives the spectrum times its factor, while the inverse's exchange is in flight.
template <int C, int K, class Spec>
__device__ __forceinline__ void spread_pair_k(SpreadFFT& f, double2 (&x)[K], const int4 (&fac)[K], int et, bool want,
                                              Spec spec) {
  fxc y[K];
  int h[K], places, level;
  spread_forward<C, K>(f, x, y, h, places, level);
  const int g = 26 - __clz(f.M), lc = fx_log2(C);
  // leave the inverse's two products no more than they can shift
  const int s = max(spread_shift(level, lc), (level + lc + g - 7) >> 1);
#pragma unroll
  for (int m = 0; m < K; m++) y[m] = spread_swap(spread_mul(y[m], fac[m], s));
  places += s;
  spread_push<C, K>(f, y);
  if (want) {
#pragma unroll
    for (int m = 0; m < K; m++) spec(m, spread_leave(spread_swap(y[m]), h[m], places + et));
  }
  spread_backward<C, K>(f, y, places, level - 2 * s);
#pragma unroll
  for (int m = 0; m < K; m++) x[m] = spread_leave(spread_swap(y[m]), h[m], places + et);
}

// One field.
template <int C = kSpreadC>
__device__ __forceinline__ double2 spread_fwd(SpreadFFT& f, double2 x) {
  double2 v[1] = {x};
  spread_fwd_k<C, 1>(f, v);
  return v[0];
}

template <int C = kSpreadC, class Store>
__device__ __forceinline__ double2 spread_inv_store(SpreadFFT& f, double2 x, Store store) {
  double2 v[1] = {x};
  spread_inv_store_k<C, 1>(f, v, [&](int, double2 s) { store(s); });
  return v[0];
}

template <int C = kSpreadC>
__device__ __forceinline__ double2 spread_inv(SpreadFFT& f, double2 x) {
  return spread_inv_store<C>(f, x, [](double2) {});
}

template <int C = kSpreadC>
__device__ __forceinline__ double2 spread_pair(SpreadFFT& f, double2 x, int4 fac, int et) {
  double2 v[1] = {x};
  const int4 q[1] = {fac};
  spread_pair_k<C, 1>(f, v, q, et, false, [](int, double2) {});
  return v[0];
}

template <int C = kSpreadC, class Spec>
__device__ __forceinline__ double2 spread_pair_spec(SpreadFFT& f, double2 x, int4 fac, int et, bool want, Spec spec) {
  double2 v[1] = {x};
  const int4 q[1] = {fac};
  spread_pair_k<C, 1>(f, v, q, et, want, [&](int, double2 s) { spec(s); });
  return v[0];
}

// A factor of modulus at most 1 as Q62 halves (exact: 53 bits).
__device__ __forceinline__ int4 fx_factor(double2 v) {
  const long long x = __double2ll_rn(v.x * 0x1p62), y = __double2ll_rn(v.y * 0x1p62);
  int4 r;
  fx_split(x, r.x, r.y);
  fx_split(y, r.z, r.w);
  return r;
}
// The same out of line, for the ends of a march: the state travels by value, so that the march's copy stays in
// registers.
struct SpreadCall {
  SpreadFFT f;
  double2 x;
};
template <int C>
__device__ __noinline__ SpreadCall spread_fwd_call(SpreadFFT f, double2 x) {
  x = spread_fwd<C>(f, x);
  return SpreadCall{f, x};
}
template <int C>
__device__ __noinline__ SpreadCall spread_inv_call(SpreadFFT f, double2 x) {
  x = spread_inv<C>(f, x);
  return SpreadCall{f, x};
}
template <int C = kSpreadC>
__device__ __forceinline__ double2 spread_fwd_end(SpreadFFT& f, double2 x) {
  const SpreadCall r = spread_fwd_call<C>(f, x);
  f.sel = r.f.sel, f.phase = r.f.phase, f.ephase = r.f.ephase, f.parity = r.f.parity, f.dead = r.f.dead;
  return r.x;
}
template <int C = kSpreadC>
__device__ __forceinline__ double2 spread_inv_end(SpreadFFT& f, double2 x) {
  const SpreadCall r = spread_inv_call<C>(f, x);
  f.sel = r.f.sel, f.phase = r.f.phase, f.ephase = r.f.ephase, f.parity = r.f.parity, f.dead = r.f.dead;
  return r.x;
}

__device__ __forceinline__ int4 fx_conj(int4 w) { return make_int4(w.x, w.y, -w.z, -w.w); }

}  // namespace nlm
