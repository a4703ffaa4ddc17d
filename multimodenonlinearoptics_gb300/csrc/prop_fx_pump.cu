// prop_fx_pump.cu -- batched row transforms (pump grids) in block fixed point, and the Chi3 pump march.
//
// k_fx_rows: one row per CTA at a time, each with its own exponent.  In FP64 the rows of a pump grid cost about 33
// instructions a point on the FP64 pipe.  Linear pump of 399 rows: 600 points 155 -> 67 us, 128 points 52 -> 37 us.
//
// k_fx_pump_chi3: the march (solvers/Chi3.cpp:41-70) on one CTA, for the
// grids that the cluster kernels do not take: those that are not powers of two (general plan or convolution form).
// The self-phase factor is FP64; 502 points x 199 rows: 90 ms with the FP64 general plan (a product per point and unit
// of the factor 251).
#include <vector>

#include "prop_fx.cuh"

namespace nlm {

// a.plan, a.fx: the transform, with a.fx.tab the tables [half, dstep][N] of modulus 1.
template <int R, int NT>
__global__ void __launch_bounds__(512) k_fx_pump_chi3(const PropArgs a, const PumpMarchArgs p) {
  extern __shared__ int4 fxsm[];
  FxField<NT> f;
  fx_begin(f, a.fx, a.plan, fxsm);
  const int N = f.grid, T = f.template T<R>(), j = f.j;
  const double invN = 1.0 / N;
  double2 x[R];
  // row 0: half a dispersion step; rows 1 ..: self-phase, a step; then half of the last step back
  for (int i = 0; i <= p.nRows; i++) {
    const int row = min(i, p.nRows - 1);
    const long long at = (long long)row * N;
    const bool back = i == p.nRows;
#pragma unroll
    for (int v = 0; v < R; v++) {
      const int t = j + v * T;
      if (!f.has(t)) {
        x[v] = czero();
      } else if (i == 0) {
        x[v] = p.env[t];
      } else if (back) {   // this thread's own points, as they are in FP64
        x[v] = cmul(p.pf[at + t], p.backP[t]);
        p.pf[at + t] = x[v];
      } else {
        const double2 r = p.rel[i - 1];
        const double a2 = cabs2(x[v]);
        x[v] = cmul(x[v], spm_factor(r.x * a2, r.y * a2));
      }
    }
    fx_pair(f, a.fx, x, a.fx.tab + (long long)(i == 0 ? 0 : 1) * N, 0, !back, true, true, [&](int v, double2 s) {
      if (f.has(j + v * T)) p.pf[at + j + v * T] = s;
    });
#pragma unroll
    for (int v = 0; v < R; v++) {
      x[v] = cscale(x[v], invN);
      if (f.has(j + v * T)) p.pt[at + j + v * T] = x[v];
    }
  }
}

// out = scale x transform of each row.
template <int R, int NT>
__global__ void __launch_bounds__(512) k_fx_rows(const double2* __restrict__ in, double2* __restrict__ out, long long rows,
                                                 const FFTPlanH plan, const FxArgs fx, int inverse, double scale) {
  extern __shared__ int4 fxsm[];
  FxField<NT> f;
  fx_begin(f, fx, plan, fxsm);
  const int N = NT > 0 ? NT : f.grid, T = f.template T<R>(), j = f.j;
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    double2 x[R];
    fxc y[R];
#pragma unroll
    for (int v = 0; v < R; v++) x[v] = f.has(j + v * T) ? in[row * N + j + v * T] : czero();
    int lift, up = 0;
    const int a = fx_enter(f, x, y, fx.A0, &lift);
#pragma unroll 1
    for (int d = 0; d < 2; d++) {   // swapped components around the forward transform: the inverse one
      if (inverse) {
#pragma unroll
        for (int v = 0; v < R; v++) y[v] = fxc{y[v].y, y[v].x};
      }
      if (d == 0) up = fx_fft(f, y, true);
    }
    fx_leave<R>(y, x, a - 1023 - fx.A0 - lift + fx.sh - up, a > 2200);
#pragma unroll
    for (int v = 0; v < R; v++)
      if (f.has(j + v * T)) out[row * N + j + v * T] = cscale(x[v], scale);
  }
}

void add_kernels_fx_pump(std::vector<KernelEntry>& t) {
  // key: kConvKey the convolution form, kGenKey the general plan
  t.push_back({kKindFxPump, kConvKey, 8, (const void*)k_fx_pump_chi3<8, 0>});
  t.push_back({kKindFxPump, kConvKey, 4, (const void*)k_fx_pump_chi3<4, 0>});
  t.push_back({kKindFxPump, kGenKey, 8, (const void*)k_fx_pump_chi3<8, kFxGen>});
  t.push_back({kKindFxPump, kGenKey, 4, (const void*)k_fx_pump_chi3<4, kFxGen>});
  // row transforms: key = log2 N, kConvKey or kGenKey
  t.push_back({kKindFxRows, 7, 4, (const void*)k_fx_rows<4, 128>});
  t.push_back({kKindFxRows, 8, 8, (const void*)k_fx_rows<8, 256>});
  t.push_back({kKindFxRows, 9, 8, (const void*)k_fx_rows<8, 512>});
  t.push_back({kKindFxRows, 10, 8, (const void*)k_fx_rows<8, 1024>});
  t.push_back({kKindFxRows, 11, 8, (const void*)k_fx_rows<8, 2048>});
  t.push_back({kKindFxRows, 12, 8, (const void*)k_fx_rows<8, 4096>});
  t.push_back({kKindFxRows, kConvKey, 8, (const void*)k_fx_rows<8, 0>});
  t.push_back({kKindFxRows, kConvKey, 4, (const void*)k_fx_rows<4, 0>});
  t.push_back({kKindFxRows, kGenKey, 8, (const void*)k_fx_rows<8, kFxGen>});
  t.push_back({kKindFxRows, kGenKey, 4, (const void*)k_fx_rows<4, kFxGen>});
}

}  // namespace nlm
