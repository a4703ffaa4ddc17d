// prop_fx_gnlse.cu -- Chi3GNLSE (solvers/Chi3GNLSE.cpp:39-92) with block fixed-point transforms (nlm_fx.cuh).
//
// The step of prop_gnlse.cu: the RK4 sum and the state's spectrum kept in the frequency domain, one row per CTA
// (k_fx_gnlse, 16 transforms a step) or two rows sharing their Raman transforms (k_fx_gnlse_pair, 12 per row and
// step).  Every convolution is one fx_pair: forward transform, factors and inverse transform in integers.  The
// products with the field, the RK4 sums and the state stay in FP64, in the CTA's slot of global scratch.
// 1024 rows of 4096 points, 109 steps: 527 -> 131 ms against the FP64 passes.
#include <vector>

#include "prop_fx.cuh"

namespace nlm {

// [a row's input] -> its spectrum x exp(+i dz/2 D) / N in XF and the field in X
template <int R, int NT>
__device__ __forceinline__ void fx_gnlse_load(const PropArgs& a, FxField<NT>& f, long long inst, bool active, double2* XF,
                                              double2* X) {
  const int N = NT > 0 ? NT : f.grid, T = f.template T<R>(), j = f.j;
  double2 x[R];
#pragma unroll
  for (int v = 0; v < R; v++) x[v] = active && a.inChannels > 0 && f.has(j + v * T) ? a.in[inst * a.inStride + j + v * T] : czero();
  auto spectrum = [&](int v, double2 s) {
    XF[j + v * T] = s;
    if (a.gridF && active && f.has(j + v * T)) a.gridF[j + v * T] = cscale(s, (double)N);
  };
  if (!a.inTime) {
#pragma unroll
    for (int v = 0; v < R; v++) {
      if (f.has(j + v * T)) x[v] = cmul(x[v], __ldg(a.half + j + v * T));
      spectrum(v, x[v]);
    }
  }
  fx_pair(f, a.fx, x, a.fx.tab + 2LL * N, a.fx.et, a.inTime != 0, true, true, spectrum);
#pragma unroll
  for (int v = 0; v < R; v++) {
    X[j + v * T] = x[v];
    if (!f.has(j + v * T)) continue;
    if (a.gridT && active) a.gridT[j + v * T] = x[v];
    if (a.ckpt && active) a.ckpt[inst * a.ckN * (long long)N + j + v * T] = x[v];
  }
}

// The end of step i: the dispersion factors on the spectrum of x + sum / 6, N (XF + A / 6), which stays in FP64 from
// step to step; then back to time.
template <int R, int NT>
__device__ __forceinline__ void fx_gnlse_end(const PropArgs& a, FxField<NT>& f, int i, long long inst, bool active,
                                             double2* XF, const double2* A, double2* X) {
  const int N = NT > 0 ? NT : f.grid, T = f.template T<R>(), j = f.j;
  const bool last = i == a.nZ - 1;
  const double2* table = last ? a.dlast : a.dstep;
  double2 x[R];
#pragma unroll
  for (int v = 0; v < R; v++) {
    const int t = j + v * T;
    x[v] = f.has(t) ? cmul(cscale(caxpy(XF[t], 1.0 / 6.0, A[t]), (double)N), __ldg(table + t)) : czero();
    XF[t] = x[v];
    if (a.gridF && active && f.has(t)) a.gridF[(long long)i * N + t] = cscale(x[v], (double)N);
  }
  const bool inv = !last || a.inTime || a.gridT != nullptr;
  fx_pair(f, a.fx, x, a.fx.tab, a.fx.et, false, inv, false, [](int, double2) {});
#pragma unroll
  for (int v = 0; v < R; v++) {
    const int t = j + v * T;
    if (!last) X[t] = x[v];
    if (!f.has(t)) continue;
    if (!last) {
      if (a.ckpt && active && i % a.ckK == 0) a.ckpt[(inst * a.ckN + i / a.ckK) * (long long)N + t] = x[v];
    }
    if (a.gridT && active) a.gridT[(long long)i * N + t] = x[v];
    if (last && active && a.out) {
      const double2 o = a.inTime ? x[v] : XF[t];
      for (int om = 0; om < a.nOut; om++) a.out[inst * a.outStride + (long long)om * N + t] = cscale(o, a.inTime ? 1.0 : (double)N);
    }
  }
}

template <int R, int NT>
__global__ void __launch_bounds__(fx_threads(NT, R), 512 / fx_threads(NT, R))
    k_fx_gnlse(const PropArgs a, double2* __restrict__ scratch) {
  extern __shared__ int4 fxsm[];
  __shared__ long long s_group;
  FxField<NT> f;
  fx_begin(f, a.fx, a.plan, fxsm);
  const int T = f.template T<R>(), j = f.j, slot = T * R;
  double2* X = scratch + (long long)blockIdx.x * 3 * slot;
  double2 *A = X + slot, *XF = X + 2 * slot;
  for (long long local = blockIdx.x; local < a.nInst; local = next_group(a, local, &s_group)) {
    const long long inst = a.instBase + local;
    fx_gnlse_load<R>(a, f, inst, true, XF, X);
    for (int i = 1; i < a.nZ; i++) {
      const double* rel = a.relInt + (long long)(i - 1) * 3;
      double2 k[R];
#pragma unroll
      for (int v = 0; v < R; v++) k[v] = czero();
#pragma unroll 1
      for (int s = 0; s < 4; s++) {
        const double fac = s == 0 ? 0.0 : (s == 3 ? 1.0 : 0.5);
        const double wgt = (s == 1 || s == 2) ? 2.0 : 1.0;
        const double ri = __ldg(rel + (s == 0 ? 0 : (s == 3 ? 2 : 1)));
        double2 y[R], u[R];
#pragma unroll
        for (int v = 0; v < R; v++) {
          y[v] = caxpy(X[j + v * T], fac, k[v]);
          u[v] = make_double2(ri * cabs2(y[v]), 0.0);
        }
        // the two convolutions through one copy of the pair: Raman, then (times the field) self-steepening
#pragma unroll 1
        for (int c = 0; c < 2; c++) {
          if (c == 1) {
#pragma unroll
            for (int v = 0; v < R; v++) u[v] = cmul(u[v], y[v]);
          }
          fx_pair(f, a.fx, u, c ? a.fx.steep : a.fx.raman, c ? a.fx.etSteep : a.fx.etRaman, true, c == 0 || s < 3, c == 1,
                  [&](int v, double2 w) { A[j + v * T] = s == 0 ? w : caxpy(A[j + v * T], wgt, w); });
        }
#pragma unroll
        for (int v = 0; v < R; v++) k[v] = u[v];
      }
      fx_gnlse_end<R>(a, f, i, inst, true, XF, A, X);
    }
    __syncthreads();
  }
}

// Two rows per CTA (rows 2q and 2q + 1): IFFT[R~ FFT[uA + i uB]] = conv(uA) + i conv(uB) for the real intensities.
template <int R, int NT>
__global__ void __launch_bounds__(fx_threads(NT, R), 512 / fx_threads(NT, R))
    k_fx_gnlse_pair(const PropArgs a, double2* __restrict__ scratch) {
  extern __shared__ int4 fxsm[];
  __shared__ long long s_group;
  FxField<NT> f;
  fx_begin(f, a.fx, a.plan, fxsm);
  const int T = NT / R, j = f.j;
  double2* slot = scratch + (long long)blockIdx.x * 9 * NT;
  auto X = [&](int r) { return slot + r * NT; };
  auto XF = [&](int r) { return slot + (2 + r) * NT; };
  auto A = [&](int r) { return slot + (4 + r) * NT; };
  auto K = [&](int r) { return slot + (6 + r) * NT; };
  double* U = reinterpret_cast<double*>(slot + 8 * NT);   // the rows' real Raman results, [row][N]
  const long long nPairs = (a.nInst + 1) / 2;
  for (long long pair = blockIdx.x; pair < nPairs; pair = next_group(a, pair, &s_group)) {
    auto active = [&](int r) { return 2 * pair + r < a.nInst; };
    auto inst = [&](int r) { return a.instBase + 2 * pair + r; };
#pragma unroll 1
    for (int r = 0; r < 2; r++) fx_gnlse_load<R>(a, f, inst(r), active(r), XF(r), X(r));
    for (int i = 1; i < a.nZ; i++) {
      const double* rel = a.relInt + (long long)(i - 1) * 3;
#pragma unroll 1
      for (int s = 0; s < 4; s++) {
        const double fac = s == 0 ? 0.0 : (s == 3 ? 1.0 : 0.5);
        const double wgt = (s == 1 || s == 2) ? 2.0 : 1.0;
        const double ri = __ldg(rel + (s == 0 ? 0 : (s == 3 ? 2 : 1)));
        const bool scaled = __double_as_longlong(ri) != 0x3ff0000000000000LL;   // 1 without an intensity profile
        // c = 0: both rows' Raman convolutions; c = 1, 2: row c - 1's product and self-steepening
#pragma unroll 1
        for (int c = 0; c < 3; c++) {
          double2 u[R];
          if (c == 0) {
#pragma unroll
            for (int v = 0; v < R; v++) {
              const int t = j + v * T;
              double2 yA = X(0)[t], yB = X(1)[t];
              if (s > 0) {   // the stage's input, kept in K's place for the product with the convolution
                yA = caxpy(yA, fac, K(0)[t]);
                yB = caxpy(yB, fac, K(1)[t]);
                K(0)[t] = yA;
                K(1)[t] = yB;
              }
              u[v] = make_double2(cabs2(yA), cabs2(yB));
              if (scaled) u[v] = cscale(u[v], ri);
            }
          } else {
            const double2* y = s == 0 ? X(c - 1) : K(c - 1);
            const double* cv = U + (c - 1) * NT;
#pragma unroll
            for (int v = 0; v < R; v++) {
              const int t = j + v * T;
              u[v] = cscale(y[t], cv[t]);
            }
          }
          double2* acc = A(c == 2);
          fx_pair(f, a.fx, u, c ? a.fx.steep : a.fx.raman, c ? a.fx.etSteep : a.fx.etRaman, true, c == 0 || s < 3, c > 0,
                  [&](int v, double2 w) { acc[j + v * T] = s == 0 ? w : caxpy(acc[j + v * T], wgt, w); });
          if (c == 0) {
#pragma unroll
            for (int v = 0; v < R; v++) {
              U[j + v * T] = u[v].x;
              U[NT + j + v * T] = u[v].y;
            }
          } else if (s < 3) {
            double2* k = K(c - 1);
#pragma unroll
            for (int v = 0; v < R; v++) k[j + v * T] = u[v];
          }
        }
      }
#pragma unroll 1
      for (int r = 0; r < 2; r++) fx_gnlse_end<R>(a, f, i, inst(r), active(r), XF(r), A(r), X(r));
    }
    __syncthreads();
  }
}

void add_kernels_fx_gnlse(std::vector<KernelEntry>& t) {
  // key = solver + 1000 log2 N, + 400: two rows per CTA
#define NLM_FX(R, LOG)                                                                                          \
  t.push_back({kKindFxGnlse, kChi3GNLSE + 1000 * LOG, R, (const void*)k_fx_gnlse<R, 1 << LOG>});              \
  t.push_back({kKindFxGnlse, kChi3GNLSE + 400 + 1000 * LOG, R, (const void*)k_fx_gnlse_pair<R, 1 << LOG>});
  NLM_FX(4, 7)
  NLM_FX(8, 8)
  NLM_FX(8, 9)
  NLM_FX(8, 10)
  NLM_FX(8, 11)
  NLM_FX(8, 12)
#undef NLM_FX
  // key + kGenKey: grids that are not powers of two
  t.push_back({kKindFxGnlse, kChi3GNLSE + kGenKey, 8, (const void*)k_fx_gnlse<8, kFxGen>});
  t.push_back({kKindFxGnlse, kChi3GNLSE + kConvKey, 8, (const void*)k_fx_gnlse<8, 0>});
}

}  // namespace nlm
