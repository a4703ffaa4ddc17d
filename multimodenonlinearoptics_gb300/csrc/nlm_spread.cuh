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
//           memory, one cluster barrier, and each thread combines the C values of its own column for
//           its CTA's output row;
// inverse:  the C-point inverse DFT over the CTAs first, the conjugate twiddle, then the local inverse
//           (the G-point DFT across warps, the conjugate W_M^(g l), the 32-point DFT in the warps;
//           unscaled, 1/N is in the tables).  It runs the forward transform's parts on values with real and
//           imaginary part swapped.
//
// The values are FP64 on both sides and 64-bit integers inside (nlm_fx.cuh says why and how).  A warp issues one
// FP64 instruction in 64 cycles on its scheduler, so the ~30 of a transform in FP64 took about 1 us however
// few points there were; an IMAD.WIDE or a 64-bit addition takes two cycles.  Every warp scales its 32 points
// by its own exponent (a bound on its 2-norm in half bits, from two warp reductions and no barrier) and sends
// that code along with its values through each exchange; the receivers shift the values to the exponent of
// the total.  Starting below 2^59, the norm grows by sqrt(32) in the warps, sqrt(G) across them and sqrt(C)
// across the CTAs, and is shifted back where it would pass 2^61.5 (spread_shift).
// Shared memory: M twiddles, two M-point exchange buffers (alternating: a thread writes a buffer only after
// the barrier that every reader of that buffer's previous contents has passed), and two halves of C x M
// cluster receive buffers (alternating per transform: a CTA writes a half only after the cluster barrier that
// its readers passed after their last read of it); the exponent codes lie beside each.
// M is a power of two of at least 32, N = C M at most 4096.
#pragma once
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
  int* code;            // [2][K][G] exponent codes of the exchange buffers
  int* rcode;           // [2][C][K][G] and of the receive buffers
  int M, rank, j;
  int l, g, t;          // lane, warp and local time index g + (M / 32) l of this thread
  int sel, phase;       // next exchange buffer / receive half
  int base;             // cluster rank of the group's first CTA (clusters holding two groups of four)
};

// Sets up the spread transform of this CTA: the M-point twiddles (every C-th entry of the N-point Q62
// table `tw`) and this thread's factors.  Ends with a CTA barrier.  K: fields transformed
// together (spread_fwd_k, spread_inv_store_k), which sizes the exchange and receive buffers.
template <int C = kSpreadC, int K = 1>
__device__ __forceinline__ void spread_init(SpreadFFT& f, double2* smem, const int4* __restrict__ tw, int M, int rank) {
  __shared__ int s_code[2 * 4 * 16], s_rcode[2 * kSpreadMaxCodes];
  f.M = M;
  f.rank = rank;
  f.j = threadIdx.x;
  f.l = f.j & 31;
  f.g = f.j >> 5;
  f.t = f.g + (M >> 5) * f.l;
  f.sel = 0;
  f.phase = 0;
  f.base = 0;
  f.code = s_code;
  f.rcode = s_rcode;
  int4* twM = reinterpret_cast<int4*>(smem);
  f.buf = twM + M;
  f.recv = twM + (1 + 2 * K) * M;
  for (int k = threadIdx.x; k < M; k += blockDim.x) twM[k] = tw[(long long)k * C];
  f.twM = twM;
  f.twC = tw[(long long)rank * f.j];
  __syncthreads();
  // decimation in frequency: the upper lane of a pair takes W_2s^(l mod s), the lower one 1
  auto lane = [&](int s) { return twM[(f.l & s) ? (f.l & (s - 1)) * (M / (2 * s)) : 0]; };
  f.w16 = lane(16);
  f.w8 = lane(8);
  f.w4 = lane(4);
  f.wgl = twM[f.g * f.l];
}

// Local time index of thread j of a CTA of M threads (the time ownership above).
__device__ __forceinline__ int spread_time_index(int j, int M) { return (j >> 5) + (M >> 5) * (j & 31); }

__device__ __forceinline__ fxc spread_shfl(fxc v, int src) {
  return fxc{__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src)};
}
__device__ __forceinline__ fxc spread_swap(fxc v) { return fxc{v.y, v.x}; }

// Places to shift before a stage that adds `grow` half bits to a norm standing `level` half bits above 2^A0.
__device__ __forceinline__ int spread_shift(int level, int grow) { return max(0, (level + grow - kSpreadPeak + 1) >> 1); }

// The point as integers below the warp's exponent; returns the warp's code h (norm^2 < 2^h).
__device__ __forceinline__ int spread_enter(double2 x, fxc& y) {
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
  y = e == 0 ? fxc{0, 0} : fxc{fx_from(x.x, rel), fx_from(x.y, rel)};
  return e == 0 ? kSpreadZero : e == 0x7ff ? kSpreadBad : h - 2 * lift;
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

// The code of the total of P fields' codes, and each one's shift to it.
template <int P>
__device__ __forceinline__ int spread_total(const int (&h)[P], int (&r)[P]) {
  int top = h[0];
#pragma unroll
  for (int c = 1; c < P; c++) top = max(top, h[c]);
  float s = 0.f;
#pragma unroll
  for (int c = 0; c < P; c++) s += __int_as_float(max(127 + h[c] - top, 0) << 23);
  const int tot = top + ((__float_as_int(s) + 0x7fffff) >> 23) - 127;
  const int a = (tot + 1) >> 1;
#pragma unroll
  for (int c = 0; c < P; c++) r[c] = min(a - ((h[c] + 1) >> 1), 62);
  return tot;
}

// v >> r, rounded
__device__ __forceinline__ fxc spread_align(fxc v, int r) {
  const long long half = (1LL << r) >> 1;
  return fxc{(v.x + half) >> r, (v.y + half) >> r};
}

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

// 32-point DFT over the lanes: lane l holds element l on entry and bin l on return.  Decimation in
// frequency: stage s pairs lane l with l ^ s, the lower lane takes a + b, the upper (a - b) W_2s^(l mod s);
// then every lane takes its bit-reversed lane's value.  The norm grows by sqrt(32).
template <int K>
__device__ __forceinline__ void spread_warp_dft(const SpreadFFT& f, fxc (&x)[K]) {
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) {
    const long long neg = (f.l & s) ? -1 : 0;
#pragma unroll
    for (int m = 0; m < K; m++) {
      const fxc p = fxc{__shfl_xor_sync(0xffffffffu, x[m].x, s), __shfl_xor_sync(0xffffffffu, x[m].y, s)};
      fxc t = fxc{p.x + ((x[m].x ^ neg) - neg), p.y + ((x[m].y ^ neg) - neg)};
      if (s >= 4) t = fx_cmul(t, s == 16 ? f.w16 : s == 8 ? f.w8 : f.w4, 2);
      if (s == 2 && (f.l & 3) == 3) t = fxc{t.y, -t.x};   // W_4 = -i
      x[m] = t;
    }
  }
  const int src = (int)(__brev((unsigned)f.l) >> 27);
#pragma unroll
  for (int m = 0; m < K; m++) x[m] = spread_shfl(x[m], src);
}

// G-point DFT across the warps of a CTA for every lane; h: the warp's codes in, the CTA's out.
template <int G, int K>
__device__ __forceinline__ void spread_cross_g(SpreadFFT& f, fxc (&x)[K], int (&h)[K]) {
  int4* b = f.buf + f.sel * K * f.M;
  int* cd = f.code + f.sel * K * G;
#pragma unroll
  for (int m = 0; m < K; m++) {
    b[m * f.M + f.j] = fx_pack(x[m]);
    if (f.l == 0) cd[m * G + f.g] = h[m];
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < K; m++) {
    int hs[G], r[G];
    fxc v[G];
#pragma unroll
    for (int c = 0; c < G; c++) hs[c] = cd[m * G + c];
    h[m] = spread_total<G>(hs, r);
#pragma unroll
    for (int c = 0; c < G; c++) v[c] = spread_align(fx_unpack(b[m * f.M + c * 32 + f.l]), r[c]);
    x[m] = spread_combine<G>(v, f.g, f.twM, f.M);
  }
  f.sel ^= 1;
}

template <int K>
__device__ __forceinline__ void spread_cross(SpreadFFT& f, fxc (&x)[K], int (&h)[K]) {
  switch (f.M >> 5) {
    case 2: spread_cross_g<2>(f, x, h); break;
    case 4: spread_cross_g<4>(f, x, h); break;
    case 8: spread_cross_g<8>(f, x, h); break;
    case 16: spread_cross_g<16>(f, x, h); break;
    default: break;   // one warp
  }
}

// C-point DFT over the cluster's CTAs: thread j of every CTA pushes its value to column j of row `rank` in all
// C CTAs (and lane v of each warp its code to CTA v); after the barrier thread j of CTA r forms output r.
template <int C, int K>
__device__ __forceinline__ void spread_exchange(SpreadFFT& f, fxc (&y)[K], int (&h)[K], cg::cluster_group& cl) {
  static_assert(C == 4 || C == 8 || C == 16, "four, eight or sixteen CTAs");
  const int M = f.M, G = M >> 5;
  int4* half = f.recv + (long long)f.phase * C * K * M;
  int* cd = f.rcode + f.phase * C * K * G;
  int4 out[K];
#pragma unroll
  for (int m = 0; m < K; m++) out[m] = fx_pack(y[m]);
#pragma unroll
  for (int v = 0; v < C; v++) {
    int4* dst = cl.map_shared_rank(half + (long long)f.rank * K * M + f.j, f.base + v);
#pragma unroll
    for (int m = 0; m < K; m++) dst[m * M] = out[m];
  }
  if (f.l < C) {
    int* dst = cl.map_shared_rank(cd + f.rank * K * G + f.g, f.base + f.l);
#pragma unroll
    for (int m = 0; m < K; m++) dst[m * G] = h[m];
  }
  cl.sync();
#pragma unroll
  for (int m = 0; m < K; m++) {
    int hs[C], r[C];
    fxc v[C];
#pragma unroll
    for (int c = 0; c < C; c++) hs[c] = cd[(c * K + m) * G + f.g];
    h[m] = spread_total<C>(hs, r);
#pragma unroll
    for (int c = 0; c < C; c++) v[c] = spread_align(fx_unpack(half[((long long)c * K + m) * M + f.j]), r[c]);
    y[m] = spread_combine<C>(v, f.rank, f.twM, M);
  }
  f.phase ^= 1;
}

// a w / 2^s
__device__ __forceinline__ fxc spread_mul(fxc a, int4 w, int s) { return fx_cmul(a, w, 2 - s); }

// time-domain ownership -> frequency-domain ownership, K fields together: one barrier and one cluster barrier for
// all of them
template <int C, int K>
__device__ __forceinline__ void spread_fwd_k(SpreadFFT& f, double2 (&x)[K], cg::cluster_group& cl) {
  const int g = 26 - __clz(f.M);   // log2 G, the half bits a G-point DFT adds (M = 32 G)
  const int s1 = spread_shift(5, g), s2 = spread_shift(5 + g - 2 * s1, fx_log2(C));
  fxc y[K];
  int h[K];
#pragma unroll
  for (int m = 0; m < K; m++) h[m] = spread_enter(x[m], y[m]);
  spread_warp_dft<K>(f, y);
#pragma unroll
  for (int m = 0; m < K; m++) y[m] = f.g > 0 ? spread_mul(y[m], f.wgl, s1) : fx_shift(y[m], s1);
  spread_cross<K>(f, y, h);
#pragma unroll
  for (int m = 0; m < K; m++) y[m] = spread_mul(y[m], f.twC, s2);
  spread_exchange<C, K>(f, y, h, cl);
#pragma unroll
  for (int m = 0; m < K; m++) x[m] = spread_leave(y[m], h[m], s1 + s2);
}

// frequency-domain ownership -> time-domain ownership (unscaled), K fields.  store(m, v) receives each field's
// frequency-domain value right after the exchange's cluster barrier (the barrier's release fence then does not
// wait for the store, which drains during the local transform).
template <int C, int K, class Store>
__device__ __forceinline__ void spread_inv_store_k(SpreadFFT& f, double2 (&x)[K], cg::cluster_group& cl, Store store) {
  const int g = 26 - __clz(f.M), lc = fx_log2(C);
  // the second product shifts two places at most: the first takes what that leaves
  const int s1 = max(0, (lc + g - 3) >> 1), s2 = spread_shift(lc + g - 2 * s1, 5);
  fxc y[K];
  int h[K];
#pragma unroll
  for (int m = 0; m < K; m++) {
    h[m] = spread_enter(x[m], y[m]);
    y[m] = spread_swap(y[m]);
  }
  spread_exchange<C, K>(f, y, h, cl);
#pragma unroll
  for (int m = 0; m < K; m++) {
    store(m, x[m]);
    y[m] = spread_mul(y[m], f.twC, s1);
  }
  spread_cross<K>(f, y, h);
#pragma unroll
  for (int m = 0; m < K; m++) y[m] = f.g > 0 ? spread_mul(y[m], f.wgl, s2) : fx_shift(y[m], s2);
  spread_warp_dft<K>(f, y);
#pragma unroll
  for (int m = 0; m < K; m++) x[m] = spread_leave(spread_swap(y[m]), h[m], s1 + s2);
}

// n bare cluster barriers: the transform slots of a group that has no transform to do while the other
// group of the same cluster does (every exchange ends with a barrier of the whole cluster)
__device__ __forceinline__ void spread_idle(cg::cluster_group& cl, int n) {
  for (int q = 0; q < n; q++) cl.sync();
}

// One field.
template <int C = kSpreadC>
__device__ __forceinline__ double2 spread_fwd(SpreadFFT& f, double2 x, cg::cluster_group& cl) {
  double2 v[1] = {x};
  spread_fwd_k<C, 1>(f, v, cl);
  return v[0];
}

template <int C = kSpreadC, class Store>
__device__ __forceinline__ double2 spread_inv_store(SpreadFFT& f, double2 x, cg::cluster_group& cl, Store store) {
  double2 v[1] = {x};
  spread_inv_store_k<C, 1>(f, v, cl, [&](int, double2 s) { store(s); });
  return v[0];
}

template <int C = kSpreadC>
__device__ __forceinline__ double2 spread_inv(SpreadFFT& f, double2 x, cg::cluster_group& cl) {
  return spread_inv_store<C>(f, x, cl, [](double2) {});
}

}  // namespace nlm
