// nlm_fx.cuh -- block fixed-point transforms: the FFT pairs of the split-step march on the integer pipes.
//
// GB300 issues 2 FP64 lanes per clock and SM (measured 2.06), but 64 lanes of IMAD.WIDE or 64-bit adds
// (measured 65.3 and 65.8).  A transform needs no floating point: its values all lie below the field's
// 2-norm, and its rounding error is only ever small relative to that norm.  So the field enters a
// transform pair as 64-bit integers with one exponent for the whole field, chosen from its 2-norm such
// that no intermediate sum can overflow, runs forward transform, table product and inverse transform in
// integers, and leaves as FP64.  Everything point-wise stays FP64.
//
// Precision.  One unit in the last place is 2^-54 or less of the field's rms value on grids of up to 4096 points,
// against 2^-53 of each value for FP64; additions are exact, only products round (to nearest, without a mean error).
// Chi2PDC Green's function, 1024 points x 1000 steps, against an 80-bit evaluation of the same steps (two pumps):
// C 4.3e-14 (FP64 passes 1.1e-13), S 1.4e-13 to 1.8e-13 (1.9e-13 to 2.3e-13); 128 points x 200 steps: C 5.7e-15
// (1.9e-14), S 3.9e-14 to 1.0e-13 (1.1e-13 to 2.3e-13).
//
// Measured (same workload, 2048 propagations): 281 -> 48 ms; 460 instructions per point and step, at 2.2 of the 4
// an SM issues per clock, the IMAD pipe 61 % and the ALU 52 % busy, FP64 (the RK4 matrices) 31 %.
//
// Scaling.  Twiddles and tables are Q62 (w = W / 2^62, |w| <= 1).  A product keeps the bits from 2^64 up, a quarter
// of x w, shifted back up by 2 - S places in a pass that shifts by S; its untwiddled legs are shifted by S.  The S
// are static (fx_pass_shift): the norm of a field that enters below 2^60 peaks below 2^62 through the
// passes.
#pragma once
#include <type_traits>

#include "nlm_device.cuh"

namespace nlm {

struct fxc {
  long long x, y;
};

__device__ __forceinline__ fxc fxadd(fxc a, fxc b) { return fxc{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ fxc fxsub(fxc a, fxc b) { return fxc{a.x - b.x, a.y - b.y}; }

// x = h 2^32 + l with a signed l
__device__ __forceinline__ void fx_split(long long x, int& h, int& l) {
  l = (int)x;
  h = (int)(x >> 32) + (int)((unsigned)l >> 31);
}
__device__ __forceinline__ long long fx_mad(int a, int b, long long c) { return c + (long long)a * b; }

// a w 2^(ls-64) rounded, w balanced halves {re h, re l, im h, im l}.  With |a| < 2^62 (modulus) and |w| <= 2^62
// every 64-bit sum below stays under 2^62.6; the dropped low x low products have mean zero.
__device__ __forceinline__ fxc fx_cmul(fxc a, int4 w, int ls) {
  int xh, xl, yh, yl;
  fx_split(a.x, xh, xl);
  fx_split(a.y, yh, yl);
  const long long rnd = 1LL << (31 - ls);
  const long long m = fx_mad(yl, -w.z, fx_mad(yh, -w.w, fx_mad(xl, w.x, fx_mad(xh, w.y, rnd))));
  const long long n = fx_mad(yl, w.x, fx_mad(yh, w.y, fx_mad(xl, w.z, fx_mad(xh, w.w, rnd))));
  long long re = fx_mad(yh, -w.z, fx_mad(xh, w.x, m >> 32));
  long long im = fx_mad(yh, w.x, fx_mad(xh, w.z, n >> 32));
  if (ls) {
    re = (long long)((unsigned long long)re << ls) | ((unsigned)m >> (32 - ls));
    im = (long long)((unsigned long long)im << ls) | ((unsigned)n >> (32 - ls));
  }
  return fxc{re, im};
}

// a / 2^s rounded to nearest, ties to even: the twiddle-free legs of a pass.  A rounding with a mean error would
// add the same field every step, and grow with the step count instead of its square root.
__device__ __forceinline__ long long fx_shift1(long long x, int s) {
  return (x + ((1 << (s - 1)) - 1) + (((unsigned)x >> s) & 1u)) >> s;
}
__device__ __forceinline__ fxc fx_shift(fxc a, int s) {
  return s ? fxc{fx_shift1(a.x, s), fx_shift1(a.y, s)} : a;
}

// u / sqrt(2) = u + u (1/sqrt(2) - 1), the constant in Q64 as balanced halves
__device__ __forceinline__ long long fx_rsqrt2(long long u) {
  constexpr int ch = -1257966796, cl = -102865788;
  int h, l;
  fx_split(u, h, l);
  const long long m = fx_mad(l, ch, fx_mad(h, cl, 1LL << 31));
  return fx_mad(h, ch, u + (m >> 32));
}

// Small DFTs, kernel e^{-2 pi i qs/r}.  The inverse transform is the forward one on values whose real and imaginary
// parts are swapped, before and after: one copy of the passes serves both directions.
__device__ __forceinline__ void fxdft4(fxc& a0, fxc& a1, fxc& a2, fxc& a3) {
  const fxc t0 = fxadd(a0, a2), t1 = fxsub(a0, a2), t2 = fxadd(a1, a3), t3 = fxsub(a1, a3);
  a0 = fxadd(t0, t2);
  a2 = fxsub(t0, t2);
  a1 = fxc{t1.x + t3.y, t1.y - t3.x};   // t1 - i t3
  a3 = fxc{t1.x - t3.y, t1.y + t3.x};   // t1 + i t3
}

__device__ __forceinline__ void fxdft8(fxc& x0, fxc& x1, fxc& x2, fxc& x3, fxc& x4, fxc& x5, fxc& x6, fxc& x7) {
  fxc e0 = x0, e1 = x2, e2 = x4, e3 = x6, o0 = x1, o1 = x3, o2 = x5, o3 = x7;
  fxdft4(e0, e1, e2, e3);
  fxdft4(o0, o1, o2, o3);
  x0 = fxadd(e0, o0);
  x4 = fxsub(e0, o0);
  x2 = fxc{e2.x + o2.y, e2.y - o2.x};
  x6 = fxc{e2.x - o2.y, e2.y + o2.x};
  // w o1 = (p1, m1) with w = (1 - i)/sqrt2, w^3 o3 = (m3, -p3) with w^3 = (-1 - i)/sqrt2
  const long long p1 = fx_rsqrt2(o1.x + o1.y), m1 = fx_rsqrt2(o1.y - o1.x);
  const long long p3 = fx_rsqrt2(o3.x + o3.y), m3 = fx_rsqrt2(o3.y - o3.x);
  x1 = fxc{e1.x + p1, e1.y + m1};
  x5 = fxc{e1.x - p1, e1.y - m1};
  x3 = fxc{e3.x + m3, e3.y - p3};
  x7 = fxc{e3.x - m3, e3.y + p3};
}

template <int r, int R>
__device__ __forceinline__ void fxdft_r(fxc (&x)[R], int u, int B) {
  if constexpr (r == 2) {
    const fxc t = x[u];
    x[u] = fxadd(t, x[u + B]);
    x[u + B] = fxsub(t, x[u + B]);
  } else if constexpr (r == 4) {
    fxdft4(x[u], x[u + B], x[u + 2 * B], x[u + 3 * B]);
  } else {
    fxdft8(x[u], x[u + B], x[u + 2 * B], x[u + 3 * B], x[u + 4 * B], x[u + 5 * B], x[u + 6 * B], x[u + 7 * B]);
  }
}

// Exchange buffers: two of fx_buffer(N) 16-byte values, used in turn (one barrier per exchange: a thread
// writes a buffer only after the barrier that the other buffer's readers follow).  Entry a sits at
// a + a / 8, so that the stride-8 writes of the first pass fall on different banks.
__device__ __forceinline__ int fx_at(int a) { return a + (a >> 3); }

// where exp(-2 pi i q / r), q < r, starts in the table of roots of the odd radices 3, 5 and 7
__host__ __device__ constexpr int fx_root_at(int r) { return r == 3 ? 0 : r == 5 ? 3 : 8; }

// NT: the grid's size where the kernel is instantiated for it (every offset is then a constant), 0 where it
// comes with the launch.
template <int NT>
struct FxField {   // NT = kFxGen: a grid that is not a power of two
  int4* buf;         // two exchange buffers
  const int4* tw;    // the passes' twiddles, Q62
  uint2* red;        // one (exponent, sum) pair per warp of the group
  int n, t, j, sel, mid;
  int grid;               // the grid's points (n where the transform has as many)
  const int4* chirp;      // convolution form: FxArgs::chirp, conv
  const int4* conv;
  const FFTPlanH* plan;   // the general plan's radices, and its roots of unity (fx_root_at)
  const int4* root;
  __device__ __forceinline__ int N() const { return NT > 0 ? NT : n; }
  template <int R>
  __device__ __forceinline__ int T() const {
    return NT > 0 ? NT / R : t;
  }
  // thread j's points that the grid has
  __device__ __forceinline__ bool has(int at) const { return NT > 0 || at < grid; }
  // radix of the second pass where it is not the plan's main one, else 1
  template <int r>
  __device__ __forceinline__ int small() const {
    if (NT <= 0) return mid;
    int n2 = NT;
    while (n2 >= r && n2 % r == 0) n2 /= r;
    return n2;
  }
};

__device__ __forceinline__ int4 fx_pack(fxc a) {
  return make_int4((int)a.x, (int)(a.x >> 32), (int)a.y, (int)(a.y >> 32));
}
__device__ __forceinline__ fxc fx_unpack(int4 v) {
  return fxc{(long long)(((unsigned long long)(unsigned)v.y << 32) | (unsigned)v.x),
             (long long)(((unsigned long long)(unsigned)v.w << 32) | (unsigned)v.z)};
}

// One pass.  tw: this pass's twiddles, w_(L r)^(q k) at (q - 1) L + k, so that consecutive threads read
// consecutive entries.  T and L are multiples of 8 or L < 8 divides the 8-blocks of fx_at evenly, so every
// access is one base plus an offset common to all threads.
template <int R, int r, int NT>
__device__ __forceinline__ void fx_pass(FxField<NT>& f, fxc (&x)[R], const int4* __restrict__ tw, int L, int S, bool last) {
  constexpr int B = R / r;
  const int T = f.template T<R>(), j = f.j;
  if (L > 1) {
    const int4* b = f.buf + f.sel * fx_buffer(f.N()) + fx_at(j);
    f.sel ^= 1;
#pragma unroll
    for (int v = 0; v < R; v++) x[v] = fx_unpack(b[fx_at(v * T)]);
#pragma unroll
    for (int u = 0; u < B; u++) {
      const int4* w = tw + ((j + u * T) & (L - 1));
      x[u] = fx_shift(x[u], S);
#pragma unroll
      for (int q = 1; q < r; q++) x[u + q * B] = fx_cmul(x[u + q * B], w[(q - 1) * L], 2 - S);
    }
  }
#pragma unroll
  for (int u = 0; u < B; u++) fxdft_r<r>(x, u, B);
  if (!last) {
#pragma unroll
    for (int u = 0; u < B; u++) {
      const int jp = j + u * T;
      const int k = jp & (L - 1);
      int4* b = f.buf + f.sel * fx_buffer(f.N()) + fx_at((jp - k) * r + k);
#pragma unroll
      for (int s = 0; s < r; s++) b[fx_at(s * L)] = fx_pack(x[u + s * B]);
    }
    __syncthreads();
  }
}

template <int V>
struct FxInt {
  static constexpr int value = V;
};

// The forward transform of the plan of make_plan(N, R): passes of radix R (8, 4 or 2) with one of another radix (1:
// none) in second place; ownership j + v T in and out.  f.tw holds the passes' twiddles one after another.
template <int R, int NT>
__device__ __forceinline__ void fx_fft_pow2(FxField<NT>& f, fxc (&x)[R]) {
  constexpr int r = R >= 8 ? 8 : R >= 4 ? 4 : 2;
  const int N = f.N(), mid = f.template small<r>();
  int L = 1, level = 0;
  const int4* tw = f.tw;
  auto pass = [&](auto radix) {
    constexpr int q = decltype(radix)::value;
    const int S = L > 1 ? fx_pass_shift(level, q) : 0;
    fx_pass<R, q>(f, x, tw, L, S, L * q == N);
    if (L > 1) tw += (q - 1) * L;
    level += fx_log2(q) - 2 * S;
    L *= q;
  };
  pass(FxInt<r>{});
  if (r == 8 && mid == 4) pass(FxInt<4>{});
  else if (r > 2 && mid == 2) pass(FxInt<2>{});
  if constexpr (NT > 0) {
#pragma unroll
    for (int p = 0; p < 12; p++)
      if (L < N) pass(FxInt<r>{});
  } else {
#pragma unroll 1
    while (L < N) pass(FxInt<r>{});
  }
}

// Shifts the group's field (2-norm below 2^62) to a norm just below 2^kFxA0 and returns the places: left, or right where
// negative.  The norm from the high words, each one unit up, in FP32.
template <int R, int NT>
__device__ __forceinline__ int fx_raise(FxField<NT>& f, fxc (&x)[R]) {
  float s = 0.f;
#pragma unroll
  for (int v = 0; v < R; v++) {
    const float p = fabsf((float)(int)(x[v].x >> 32)) + 1.f, q = fabsf((float)(int)(x[v].y >> 32)) + 1.f;
    s = fmaf(p, p, s);
    s = fmaf(q, q, s);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((f.j & 31) == 0) f.red[f.j >> 5] = make_uint2((unsigned)__float_as_int(s), 0u);
  __syncthreads();
  const int W = f.template T<R>() >> 5;
  s = 0.f;
  for (int q = 0; q < W; q++) s += __int_as_float((int)f.red[q].x);
  // norm^2 < 2^64 s < 2^(64 + e + 1); 1.0001: the roundings of 16 x 32 x 8 sums
  const int e = (__float_as_int(s * 1.0001f) >> 23) - 127;
  const int up = kFxA0 - 32 - ((e + 2) >> 1);
#pragma unroll
  for (int v = 0; v < R; v++) {
    x[v] = up >= 0 ? fxc{(long long)((unsigned long long)x[v].x << up), (long long)((unsigned long long)x[v].y << up)}
                   : fx_shift(x[v], -up);
  }
  return up;
}

// Grids of N points with a prime factor that has no pass (NT = 0, f.chirp set): with 2 t k = t^2 + k^2 - (k - t)^2 the
// transform is a convolution with the conjugate chirp, run cyclically on L >= 2 N - 1 points, L a power of two
// (Bluestein 1970): x c, forward transform over L, x conv, inverse transform, x c.  Points past the grid are zero.
// The chirp's transform is a comb and the points past the grid are dropped, so the norm falls by as much as 2^6 on the
// way, by how much depends on the field: it is raised before each transform over L, and the products are not shifted
// (1022 points, error of a transform of noise: 2.5e-16 without, 8.0e-17 with).  fresh: the field stands just below 2^A0
// already.  Returns the places that the result stands above the static scale (FxArgs::sh); its norm is below 2^62.
template <int R, int NT>
__device__ __forceinline__ int fx_fft(FxField<NT>& f, fxc (&x)[R], bool fresh) {
  if constexpr (NT > 0) {
    fx_fft_pow2(f, x);
    return 0;
  } else {
    int up = 0;
    const bool conv = f.chirp != nullptr;
    auto chirp = [&]() {
#pragma unroll
      for (int v = 0; v < R; v++) {
        const int t = f.j + v * f.t;
        x[v] = t < f.grid ? fx_cmul(x[v], __ldg(f.chirp + t), 2) : fxc{0, 0};
      }
    };
    if (conv) {
      if (!fresh) up = fx_raise(f, x);
      chirp();
    }
#pragma unroll 1
    for (int d = 0; d < (conv ? 2 : 1); d++) {
      fx_fft_pow2(f, x);
      if (conv) {
        if (d == 0) {
#pragma unroll
          for (int v = 0; v < R; v++) x[v] = fx_cmul(x[v], __ldg(f.conv + f.j + v * f.t), 2);
          up += fx_raise(f, x);
        }
#pragma unroll
        for (int v = 0; v < R; v++) x[v] = fxc{x[v].y, x[v].x};
      }
    }
    if (conv) chirp();
    return up;
  }
}

// Smallest a with ||x||_2 < 2^a over the group's points (T a multiple of 32), from the high words: the warp's largest
// exponent, then the squares relative to it in FP32 (the 20-bit significands truncated, the sums rounded up).
// Returns a + 1023; 0 when every value is zero or subnormal; more than 2046 + 1 when one is infinite or NaN.
template <int R, int NT>
__device__ __forceinline__ int fx_norm(FxField<NT>& f, const double2 (&x)[R]) {
  unsigned m = 0;
#pragma unroll
  for (int v = 0; v < R; v++) {
    m = max(m, (unsigned)__double2hiint(x[v].x) & 0x7fffffffu);
    m = max(m, (unsigned)__double2hiint(x[v].y) & 0x7fffffffu);
  }
  m = __reduce_max_sync(0xffffffffu, m);
  const int e = (int)(m >> 20);
  const int off = (127 << 20) - (e << 20);
  float s = 0.f;
#pragma unroll
  for (int v = 0; v < R; v++) {
    const float p = __int_as_float(max((__double2hiint(x[v].x) & 0x7fffffff) + off, 0) << 3);
    const float q = __int_as_float(max((__double2hiint(x[v].y) & 0x7fffffff) + off, 0) << 3);
    s = fmaf(p, p, s);
    s = fmaf(q, q, s);
  }
  // s < 8 R; in units of 2^-16
  const unsigned w = __reduce_add_sync(0xffffffffu, (unsigned)(s * 65536.f) + 2u);
  if ((f.j & 31) == 0) f.red[f.j >> 5] = make_uint2((unsigned)e, w);
  __syncthreads();
  const int W = f.template T<R>() >> 5;
  int E = 0;
  unsigned S = 0;
  if constexpr (NT > 0) {
    uint2 p[NT > 0 ? NT / R / 32 : 1];
#pragma unroll
    for (int q = 0; q < NT / R / 32; q++) {
      p[q] = f.red[q];
      E = max(E, (int)p[q].x);
    }
#pragma unroll
    for (int q = 0; q < NT / R / 32; q++) S += (p[q].y >> min(31, 2 * (E - (int)p[q].x))) + 1u;
  } else {
    for (int q = 0; q < W; q++) E = max(E, (int)f.red[q].x);
    for (int q = 0; q < W; q++) {
      const uint2 p = f.red[q];
      S += (p.y >> min(31, 2 * (E - (int)p.x))) + 1u;
    }
  }
  if (E == 0) return 0;
  if (E == 0x7ff) return 4095;
  const int nb = 32 - __clz((int)S);          // S < 2^nb, norm^2 < 2^(nb - 16) 4^(E - 1023)
  return E + ((nb - 15) >> 1);                 // ceil((nb - 16) / 2), nb >= 16
}

// d 2^(A0 - a) rounded to an integer, rel = 62 - A0 + (a + 1023) with |d| < 2^a
__device__ __forceinline__ long long fx_from(double d, int rel) {
  const int hi = __double2hiint(d);
  const unsigned lo = (unsigned)__double2loint(d);
  const unsigned mh = (__funnelshift_l(lo, (unsigned)hi, 10) & 0x3fffffffu) | 0x40000000u;
  const unsigned long long m = ((unsigned long long)mh << 32) | (lo << 10);
  const int sh = min(rel - 1 - ((hi >> 20) & 0x7ff), 63);   // one bit more than the result has, for the rounding
  const long long v = (long long)(((m >> sh) + 1) >> 1), s = (long long)(hi >> 31);
  return (v ^ s) - s;
}

// v 2^k as a double, rounded to nearest, by integer operations (a conversion or two FP64 additions would take the
// FP64 pipe that the point-wise step needs); the result must be zero or a normal number.
__device__ __forceinline__ double fx_to(long long v, int k) {
  const int sgn = (int)(v >> 32) >> 31;
  const long long s = sgn;
  const unsigned long long m = (unsigned long long)((v ^ s) - s);
  const unsigned hi = (unsigned)(m >> 32), lo = (unsigned)m;
  const unsigned w = hi ? hi : lo;
  // p: position of the top bit (the conversion truncates, so its exponent is exact)
  const int p = (__float_as_int(__uint2float_rz(w)) >> 23) - 127 + (hi ? 32 : 0);
  const unsigned long long n = ((m << (62 - p)) + 0x200u) >> 10;   // 53 bits, bit 52 set
  const int h = (int)(n >> 32) + ((1022 + p + k) << 20);
  return w ? __hiloint2double(h | (sgn & (int)0x80000000), (int)(unsigned)n) : 0.0;
}

// ---- grids that are not powers of two (NT = kFxGen) ---------------------------------------------
// T threads (whole warps) of R points, j + v T for those below N.  The points go to an exchange buffer, every pass
// reads one buffer and writes the other (butterfly b < N / r: inputs b + q N / r, k = b mod L, twiddle q k, outputs
// (b - k) r + k + s L), and the result comes back to the owners.  A thread takes the butterflies b = j + u T.
constexpr int kFxGen = -1;

// sum of c[q] a[q] (Q62 constants, q < n), rounded; the cross products are folded in pairs, whose sums stay below 2^63
template <int n>
__device__ __forceinline__ long long fx_dot(const int (&ah)[n], const int (&al)[n], const int2 (&c)[n]) {
  long long acc = 0;
  std::conditional_t<(n > 2), unsigned long long, unsigned> low = 0;   // carries only from the second pair on
#pragma unroll
  for (int q = 0; q < n; q += 2) {
    long long m = fx_mad(al[q], c[q].x, fx_mad(ah[q], c[q].y, q == 0 ? 1LL << 29 : 0));
    if (q + 1 < n) m = fx_mad(al[q + 1], c[q + 1].x, fx_mad(ah[q + 1], c[q + 1].y, m));
    acc += m >> 32;
    low += (unsigned)m;
    acc = fx_mad(ah[q], c[q].x, acc);
    if (q + 1 < n) acc = fx_mad(ah[q + 1], c[q + 1].x, acc);
  }
  if constexpr (n > 2) acc += (long long)(low >> 32);
  return (long long)((unsigned long long)acc << 2) | ((unsigned)low >> 30);
}

// r-point DFT, r an odd prime, of values whose norm is at most 2^62 / sqrt(r).  With a_q = x_q + x_(r-q),
// b_q = x_q - x_(r-q), y_s and y_(r-s) are x_0 + sum cos(2 pi q s / r) a_q -+ i sum sin(2 pi q s / r) b_q.  root: cos
// and -sin of 2 pi q / r in Q62 halves.
template <int r>
__device__ __forceinline__ void fx_odd_dft(fxc (&x)[r], const int4* root) {
  constexpr int h = (r - 1) / 2;
  int axh[h], axl[h], ayh[h], ayl[h], bxh[h], bxl[h], byh[h], byl[h];
  const fxc x0 = x[0];
#pragma unroll
  for (int q = 1; q <= h; q++) {
    const fxc a = fxadd(x[q], x[r - q]), b = fxsub(x[q], x[r - q]);
    x[0] = fxadd(x[0], a);
    fx_split(a.x, axh[q - 1], axl[q - 1]);
    fx_split(a.y, ayh[q - 1], ayl[q - 1]);
    fx_split(b.x, bxh[q - 1], bxl[q - 1]);
    fx_split(b.y, byh[q - 1], byl[q - 1]);
  }
#pragma unroll
  for (int s = 1; s <= h; s++) {
    int2 cs[h], sn[h];
#pragma unroll
    for (int q = 1; q <= h; q++) {
      const int4 w = root[(q * s) % r];
      cs[q - 1] = make_int2(w.x, w.y);
      sn[q - 1] = make_int2(w.z, w.w);   // -sin
    }
    const long long cx = x0.x + fx_dot<h>(axh, axl, cs), cy = x0.y + fx_dot<h>(ayh, ayl, cs);
    const long long dx = fx_dot<h>(bxh, bxl, sn), dy = fx_dot<h>(byh, byl, sn);   // -sum sin b
    x[s] = fxc{cx - dy, cy + dx};        // C + i D, D = -sum sin b
    x[r - s] = fxc{cx + dy, cy - dx};
  }
}

template <int R, int r>
__device__ __forceinline__ void fx_gen_pass(const FxField<kFxGen>& f, const int4* __restrict__ src, int4* __restrict__ dst,
                                            const int4* __restrict__ tw, int L, int S) {
  constexpr int U = (R + r - 1) / r;
  const int nb = f.n / r;
#pragma unroll 1
  for (int u = 0; u < U; u++) {
    const int b = f.j + u * f.t;
    if (b < nb) {
      const int k = b % L;
      fxc x[r];
#pragma unroll
      for (int q = 0; q < r; q++) {
        x[q] = fx_unpack(src[fx_at(b + q * nb)]);
        if (q > 0 && L > 1) x[q] = fx_cmul(x[q], tw[(q - 1) * L + k], 2 - S);
      }
      if (L > 1) x[0] = fx_shift(x[0], S);
      if constexpr (r == 2 || r == 4 || r == 8) {
        fxdft_r<r>(x, 0, 1);
      } else {
        fx_odd_dft<r>(x, f.root + fx_root_at(r));
      }
      const int base = (b - k) * r + k;
#pragma unroll
      for (int s = 0; s < r; s++) dst[fx_at(base + s * L)] = fx_pack(x[s]);
    }
  }
}

template <int R>
__device__ __forceinline__ int fx_fft(FxField<kFxGen>& f, fxc (&x)[R], bool) {
  f.sel ^= 1;
  int4* b = f.buf + f.sel * fx_buffer(f.n);
#pragma unroll
  for (int v = 0; v < R; v++)
    if (f.j + v * f.t < f.n) b[fx_at(f.j + v * f.t)] = fx_pack(x[v]);
  int L = 1, level = 0;
  const int4* tw = f.tw;
#pragma unroll 1
  for (int p = 0; p < f.plan->nPass; p++) {
    const int r = f.plan->radix[p];
    const int S = fx_gen_shift(level, r);
    __syncthreads();
    int4* d = f.buf + (f.sel ^ 1) * fx_buffer(f.n);
    switch (r) {
      case 2: fx_gen_pass<R, 2>(f, b, d, tw, L, S); break;
      case 3: fx_gen_pass<R, 3>(f, b, d, tw, L, S); break;
      case 4: fx_gen_pass<R, 4>(f, b, d, tw, L, S); break;
      case 5: fx_gen_pass<R, 5>(f, b, d, tw, L, S); break;
      case 7: fx_gen_pass<R, 7>(f, b, d, tw, L, S); break;
      default: fx_gen_pass<R, 8>(f, b, d, tw, L, S); break;
    }
    level += fx_gen_growth(r) - 16 * S;
    if (L > 1) tw += (r - 1) * L;
    L *= r;
    f.sel ^= 1;
    b = d;
  }
  __syncthreads();
#pragma unroll
  for (int v = 0; v < R; v++) x[v] = f.j + v * f.t < f.n ? fx_unpack(b[fx_at(f.j + v * f.t)]) : fxc{0, 0};
  return 0;
}

constexpr double kFxLift = 0x1p900;   // applied to fields of tiny or zero norm

// The field as integers of 2-norm below 2^A0; returns a + 1023 (norm < 2^a), 0 for a zero field, 4095 for one with
// infinite or NaN values.  *lift: the power of two applied first.
template <int R, int NT>
__device__ __forceinline__ int fx_enter(FxField<NT>& f, double2 (&x)[R], fxc (&y)[R], int A0, int* lift) {
  int a = fx_norm(f, x);
  *lift = 0;
  if (a < 256) {
#pragma unroll
    for (int v = 0; v < R; v++) x[v] = cscale(x[v], kFxLift);
    __syncthreads();
    a = fx_norm(f, x);
    *lift = 900;
  }
  const int rel = 62 - A0 + a;
#pragma unroll
  for (int v = 0; v < R; v++) y[v] = a == 0 ? fxc{0, 0} : fxc{fx_from(x[v].x, rel), fx_from(x[v].y, rel)};
  return a;
}

template <int R>
__device__ __forceinline__ void fx_leave(const fxc (&y)[R], double2 (&x)[R], int k, bool bad) {
  const bool fast = k > -1000 && k < 900;
  const int k0 = fast ? k : 0;
#pragma unroll
  for (int v = 0; v < R; v++) x[v] = make_double2(fx_to(y[v].x, k0), fx_to(y[v].y, k0));
  if (!fast) {
#pragma unroll
    for (int v = 0; v < R; v++) x[v] = make_double2(scalbn(x[v].x, k), scalbn(x[v].y, k));
  }
  if (bad) {
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
#pragma unroll
    for (int v = 0; v < R; v++) x[v] = make_double2(nan, nan);
  }
}

}  // namespace nlm
