// prop_fx.cuh -- one-CTA split-step kernels with block fixed-point transforms (nlm_fx.cuh).
//
// One CTA of T = N / R threads runs one propagation at a time, groups claimed like in nlm_propagate.cuh.  The march
// is a loop over stages so that the kernel holds one forward and one inverse transform:
//   stage 0:        [forward if the input is in the time domain]  x exp(+i dz/2 D) (of a spectrum: in FP64)
//   stage i:        RK4 step i point-wise in FP64, forward, x dispStep (the last stage's with exp(-i dz/2 D))
// (nZ > 1), each followed by the inverse transform unless it is the last and only the spectrum is wanted.
#pragma once
#include "nlm_fx.cuh"
#include "nlm_propagate.cuh"

namespace nlm {

// Launch bounds: the grid's threads (at least 128, at most 512 resident per SM: 128 registers each).
__host__ __device__ constexpr int fx_threads(int NT, int R) { return NT <= 0 ? 512 : NT / R < 128 ? 128 : NT / R; }

template <int NT>
__device__ __forceinline__ void fx_begin(FxField<NT>& f, const FxArgs& fx, const FFTPlanH& plan, int4* smem) {
  f.n = fx.L ? fx.L : plan.N;
  f.grid = plan.N;
  f.chirp = fx.chirp;
  f.conv = fx.conv;
  f.t = plan.T;
  f.j = threadIdx.x;
  f.sel = 0;
  f.mid = plan.nPass > 1 && plan.radix[1] != plan.radix[0] ? plan.radix[1] : 1;
  for (int k = threadIdx.x; k < f.n; k += blockDim.x) smem[k] = fx.tw[k];
  f.tw = smem;
  f.plan = &plan;
  f.root = fx.root;
  f.buf = smem + f.N();
  f.red = reinterpret_cast<uint2*>(smem + f.N() + 2 * fx_buffer(f.N()));
  __syncthreads();
}

template <int NT>
__device__ __forceinline__ int4 fx_load(const FxField<NT>& f, const int4* __restrict__ table, int t) {
  return __ldg(table + (NT <= 0 ? min(t, f.grid - 1) : t));
}

// One mode through [forward x table] [inverse].  spec(v, value) receives the spectrum (1/N folded in, as the tables
// have it) when wantF; x is the field after the inverse, or the spectrum without it.  Without the forward transform x
// is a spectrum times its factors: their product is FP64's, since a spectrum that no transform has rounded relative to
// its norm would lose bits of its small values here.
template <int R, int NT, class Spec>
__device__ __forceinline__ void fx_pair(FxField<NT>& f, const FxArgs& fx, double2 (&x)[R], const int4* __restrict__ table,
                                        int et, bool fwd, bool inv, bool wantF, Spec spec) {
  if (!fwd && !inv) return;
  fxc y[R];
  int lift;
  const int a = fx_enter(f, x, y, fx.A0, &lift);
  const bool bad = a > 2200;
  int k = a - 1023 - fx.A0 - lift;
#pragma unroll 1
  for (int dir = 0; dir < 2; dir++) {
    if (dir == 0 ? fwd : inv) {
      k += fx.sh - fx_fft(f, y, dir == 0 || !fwd);
    }
    if (dir == 0 && fwd) {
      k += et + 2 - fx.ls;
#pragma unroll
      for (int v = 0; v < R; v++) y[v] = fx_cmul(y[v], fx_load(f, table, f.j + v * f.template T<R>()), fx.ls);
      if (wantF) {
        fx_leave<R>(y, x, k, bad);
#pragma unroll
        for (int v = 0; v < R; v++) spec(v, x[v]);
      }
    }
#pragma unroll
    for (int v = 0; v < R; v++) y[v] = fxc{y[v].y, y[v].x};
  }
  if (inv) fx_leave<R>(y, x, k, bad);
}

// One propagation.
template <int M, int R, int NT, class Point>
__device__ __forceinline__ void fx_propagate(const PropArgs& a, FxField<NT>& f, long long inst, Point point) {
  const FxArgs& fx = a.fx;
  const int N = NT > 0 ? NT : f.grid, T = f.template T<R>(), j = f.j;
  const long long ms = (long long)a.nZ * N;
  const int last = a.nZ - 1;
  double2 x[M][R];
  if (a.inKind == 0) {
    const long long pair = inst >> 1;
    const int bin = (int)(pair % N), im = (int)(pair / N);
    const int mode = a.impModes[im < kMaxModes ? im : 0];
    const double2 val = (inst & 1) ? make_double2(0.0, 1.0) : make_double2(1.0, 0.0);
#pragma unroll
    for (int m = 0; m < M; m++)
#pragma unroll
      for (int v = 0; v < R; v++) x[m][v] = (m == mode && j + v * T == bin) ? val : czero();
  } else {
    const double2* row = a.in + inst * a.inStride;
#pragma unroll
    for (int m = 0; m < M; m++) {
      int seg = -1;
      if (m == a.inputMode) seg = 0;
      else if (a.inputMode < 1 && m < a.inChannels) seg = m;
#pragma unroll
      for (int v = 0; v < R; v++) x[m][v] = seg >= 0 && f.has(j + v * T) ? row[(long long)seg * N + j + v * T] : czero();
    }
  }
  if (!a.inTime) {
#pragma unroll
    for (int m = 0; m < M; m++)
#pragma unroll
      for (int v = 0; v < R; v++) {
        const int t = j + v * T;
        if (!f.has(t)) continue;
        x[m][v] = cmul(x[m][v], __ldg(a.half + (long long)m * N + t));
        if (a.gridF) a.gridF[m * ms + t] = cscale(x[m][v], (double)N);
      }
  }
  for (int i = 0; i <= last; i++) {
    if (i > 0) point(i, x);
    const bool end = i == last;
    const bool fwd = i > 0 || a.inTime, inv = !end || a.inTime || a.gridT != nullptr;
    const int which = i == 0 ? 2 : !end ? 0 : 1;
    // the modes in turn through one copy of the pair: mode m sits in x[0] during its turn
#pragma unroll 1
    for (int m = 0; m < M; m++) {
      const int4* table = fx.tab + ((long long)which * M + m) * N;
      fx_pair(f, fx, x[0], table, fx.et, fwd, inv, a.gridF != nullptr || !inv, [&](int v, double2 s) {
        if (a.gridF && f.has(j + v * T)) a.gridF[m * ms + (long long)i * N + j + v * T] = cscale(s, (double)N);
      });
      if (a.gridT) {
#pragma unroll
        for (int v = 0; v < R; v++)
          if (f.has(j + v * T)) a.gridT[m * ms + (long long)i * N + j + v * T] = x[0][v];
      }
      if (a.ckpt && !end && i % a.ckK == 0) {
#pragma unroll
        for (int v = 0; v < R; v++)
          if (f.has(j + v * T)) a.ckpt[((inst * a.ckN + i / a.ckK) * M + m) * (long long)N + j + v * T] = x[0][v];
      }
      if constexpr (M > 1) {
#pragma unroll
        for (int v = 0; v < R; v++) {
          const double2 t = x[0][v];
#pragma unroll
          for (int q = 0; q < M - 1; q++) x[q][v] = x[q + 1][v];
          x[M - 1][v] = t;
        }
      }
    }
  }
  store_output<M, R, NT <= 0>(a, inst, true, j, x, a.inTime ? 1.0 : (double)N);
  __syncthreads();
}

template <int M, int R, int NT, class Point>
__device__ __forceinline__ void fx_march(const PropArgs& a, Point point) {
  extern __shared__ int4 fxsm[];
  __shared__ long long s_group;
  FxField<NT> f;
  fx_begin(f, a.fx, a.plan, fxsm);
  for (long long local = blockIdx.x; local < a.nInst; local = next_group(a, local, &s_group))
    fx_propagate<M, R, NT>(a, f, a.instBase + local, point);
}

// Step i of a pump-driven solver as its per-point real (2M) x (2M) matrix (layout as k_propagate_linear).
template <int M, int R, int NT>
__device__ __forceinline__ void fx_matrix_step(const PropArgs& a, int i, int N, int T, int j, double2 (&x)[M][R]) {
  constexpr int D = 2 * M;
  const double2* mat = reinterpret_cast<const double2*>(a.prop) + (long long)(i - 1) * (D * M) * N;
#pragma unroll
  for (int v = 0; v < R; v++) {
    const int t = j + v * T;
    if (NT <= 0 && t >= N) continue;   // past the grid: zeros stay zero
    double in[D], out[D];
#pragma unroll
    for (int m = 0; m < M; m++) {
      in[2 * m] = x[m][v].x;
      in[2 * m + 1] = x[m][v].y;
    }
#pragma unroll
    for (int r = 0; r < D; r++) {
      const double2 e0 = __ldg(mat + (long long)(r * M) * N + t);
      double s = fma(e0.y, in[1], e0.x * in[0]);
#pragma unroll
      for (int c = 1; c < M; c++) {
        const double2 e = __ldg(mat + (long long)(r * M + c) * N + t);
        s = fma(e.y, in[2 * c + 1], fma(e.x, in[2 * c], s));
      }
      out[r] = s;
    }
#pragma unroll
    for (int m = 0; m < M; m++) x[m][v] = make_double2(out[2 * m], out[2 * m + 1]);
  }
}

// Step i with the solver's DiffEq.
template <class S, int R, int NT>
__device__ __forceinline__ void fx_diffeq_step(const PropArgs& a, int i, int N, int T, int j, double2 (&x)[S::kM][R]) {
  constexpr int M = S::kM, P = S::kP > 0 ? S::kP : 1;
  const double2* c = a.coef + (long long)(i - 1) * 3 * a.nCoef;
#pragma unroll
  for (int v = 0; v < R; v++) {
    const int t = j + v * T;
    if (NT <= 0 && t >= N) continue;
    double2 p[3][P], xm[M];
#pragma unroll
    for (int q = 0; q < P; q++) {
      if (S::kP > 0) {
        const double2* pr = a.pump + q * a.pumpStride + (long long)(2 * i - 2) * N + t;
        p[0][q] = __ldg(pr);
        p[1][q] = __ldg(pr + N);
        p[2][q] = __ldg(pr + 2 * N);
      } else {
        p[0][q] = p[1][q] = p[2][q] = czero();
      }
    }
#pragma unroll
    for (int m = 0; m < M; m++) xm[m] = x[m][v];
    rk4_point<S>(xm, p, c);
#pragma unroll
    for (int m = 0; m < M; m++) x[m][v] = xm[m];
  }
}

template <int M, int R, int NT = 0>
__global__ void __launch_bounds__(fx_threads(NT, R), 512 / fx_threads(NT, R)) k_fx_linear(const PropArgs a) {
  const int N = NT > 0 ? NT : a.plan.N, T = NT > 0 ? NT / R : a.plan.T, j = threadIdx.x;
  fx_march<M, R, NT>(a, [&](int i, double2 (&x)[M][R]) { fx_matrix_step<M, R, NT>(a, i, N, T, j, x); });
}

template <class S, int R, int NT = 0>
__global__ void __launch_bounds__(512) k_fx_direct(const PropArgs a) {
  constexpr int M = S::kM;
  const int N = NT > 0 ? NT : a.plan.N, T = NT > 0 ? NT / R : a.plan.T, j = threadIdx.x;
  fx_march<M, R, NT>(a, [&](int i, double2 (&x)[M][R]) { fx_diffeq_step<S, R, NT>(a, i, N, T, j, x); });
}

}  // namespace nlm
