// prop_spread.cuh -- the one-point-per-thread cluster kernels (nlm_spread.cuh), templated on the
// cluster size C (4 or 8): single propagations and small batches, and the Chi3 pump march.
//
// k_pump_chi3_spread has the arithmetic of k_pump_chi3 / k_pump_chi3_cluster (solvers/Chi3.cpp:41-70);
// k_propagate_spread<S, C> that of k_propagate_cluster<S> (src/_NonlinearMedium.hpp:160-239): the same
// tables, the same order of operations per point, only the ownership of the points differs.
#pragma once
#include "nlm_spread.cuh"

namespace nlm {

// tw: the N-point Q62 table; M = N / C threads per CTA.
template <int C>
__global__ void __launch_bounds__(kMaxThreads) k_pump_chi3_spread(double2* __restrict__ pf, double2* __restrict__ pt,
                                                                  const double2* __restrict__ env,
                                                                  const double2* __restrict__ halfP,
                                                                  const double2* __restrict__ dstepP,
                                                                  const double2* __restrict__ backP,
                                                                  const double2* __restrict__ rel, int nRows, int M,
                                                                  const int4* __restrict__ tw, ExchangeWait wait) {
  extern __shared__ double2 smem[];
  cg::cluster_group cl = cg::this_cluster();
  SpreadFFT f;
  const int rank = (int)cl.block_rank();
  spread_init<C>(f, smem, tw, M, rank, wait);
  cl.sync();
  const int N = M * C;
  const int tn = rank + C * f.t;          // time-domain point of this thread
  const int fk = f.j + M * rank;          // frequency bin of this thread
  const double invN = 1.0 / N;
  const int et = -(31 - __clz(N));        // the inverse transform's 1/N
  const int4 dp = fx_factor(dstepP[fk]);
  double2 x = spread_fwd_end<C>(f, env[tn]);
  x = cmul(x, halfP[fk]);
  pf[fk] = x;
  x = cscale(spread_inv_end<C>(f, x), invN);
  pt[tn] = x;
  for (int i = 1; i < nRows; i++) {
    const double2 r = rel[i - 1];
    const double a2 = cabs2(x);
    x = cmul(x, spm_factor(r.x * a2, r.y * a2));
    // the spectrum comes with the 1/N of the field
    x = spread_pair_spec<C>(f, x, dp, et, true, [&](double2 v) { pf[(long long)i * N + fk] = cscale(v, (double)N); });
    pt[(long long)i * N + tn] = x;
  }
  // last row: undo half of the last pump dispersion step (each thread rereads its own bin)
  const long long last = (long long)(nRows - 1) * N;
  x = cmul(pf[last + fk], backP[fk]);
  pf[last + fk] = x;
  pt[last + tn] = cscale(spread_inv_end<C>(f, x), invN);
  cl.sync();
  spread_drain(f);
}

// The modes one place on, the first one last.
template <class T, int MD>
__device__ __forceinline__ void spread_turn(T (&x)[MD]) {
  const T t = x[0];
#pragma unroll
  for (int q = 0; q < MD - 1; q++) x[q] = x[q + 1];
  x[MD - 1] = t;
}

// All MD modes, one after another: time -> frequency domain and back (the ends of a march).
template <int C, int MD>
__device__ __forceinline__ void spread_fwd_all(SpreadFFT& f, double2 (&x)[MD]) {
#pragma unroll 1
  for (int m = 0; m < MD; m++) {   // mode m sits in x[0] during its turn
    x[0] = spread_fwd_end<C>(f, x[0]);
    spread_turn(x);
  }
}

template <int C, int MD>
__device__ __forceinline__ void spread_inv_all(SpreadFFT& f, double2 (&x)[MD]) {
#pragma unroll 1
  for (int m = 0; m < MD; m++) {
    x[0] = spread_inv_end<C>(f, x[0]);
    spread_turn(x);
  }
}

// All MD modes through the dispersion pair.
template <int C, int K, int MD, class Spec>
__device__ __forceinline__ void spread_pair_all(SpreadFFT& f, double2 (&x)[MD], int4 (&fac)[MD], int et, bool want,
                                                Spec spec) {
  if constexpr (K > 1) {
    spread_pair_k<C, MD>(f, x, fac, et, want, spec);
  } else {
#pragma unroll 1
    for (int m = 0; m < MD; m++) {
      x[0] = spread_pair_spec<C>(f, x[0], fac[0], et, want, [&](double2 v) { spec(m, v); });
      spread_turn(x);
      spread_turn(fac);
    }
  }
}

// One propagation per cluster (clusters take instances in turn); a.plan.N = M, a.fx.twN the N-point table.
// Point-wise work: the pump-driven solvers' RK4 matrices (a.prop) or the solver's DiffEq.  K = 1: the
// modes' transforms one after another; K = the solver's mode count: all modes in each transform
// together (the _k forms: one barrier and one exchange per transform for all of them), with K times the exchange and receive buffers.  Either way every mode
// goes through the same operations, so the results are identical.
template <class S, int C, int K = 1>
__global__ void __launch_bounds__(kMaxThreads) k_propagate_spread(const PropArgs a) {
  constexpr int MD = S::kM, P = S::kP > 0 ? S::kP : 1;
  static_assert(K == 1 || K == MD, "modes one at a time or all together");
  extern __shared__ double2 smem[];
  cg::cluster_group cl = cg::this_cluster();
  SpreadFFT f;
  const int rank = (int)cl.block_rank();
  const int M = a.plan.N;
  spread_init<C, K>(f, smem, a.fx.twN, M, rank, a.fx.wait);
  cl.sync();
  const int N = M * C;
  const int tn = rank + C * f.t;
  const int fk = f.j + M * rank;
  const long long clusterId = blockIdx.x / C, nClusters = gridDim.x / C;
  const long long ms = (long long)a.nZ * N;
  for (long long local = clusterId; local < a.nInst; local += nClusters) {
    const long long inst = a.instBase + local;
    double2 x[MD];
    const double2* row = a.in + inst * a.inStride;
#pragma unroll
    for (int m = 0; m < MD; m++) {
      int seg = -1;
      if (m == a.inputMode) seg = 0;
      else if (a.inputMode < 1 && m < a.inChannels) seg = m;
      x[m] = seg >= 0 ? row[(long long)seg * N + (a.inTime ? tn : fk)] : czero();
    }
    if (a.inTime) spread_fwd_all<C, MD>(f, x);
#pragma unroll
    for (int m = 0; m < MD; m++) x[m] = cmul(x[m], __ldg(a.half + (long long)m * N + fk));
    if (a.gridF) {
#pragma unroll
      for (int m = 0; m < MD; m++) a.gridF[m * ms + fk] = cscale(x[m], (double)N);
    }
    spread_inv_all<C, MD>(f, x);
    if (a.gridT) {
#pragma unroll
      for (int m = 0; m < MD; m++) a.gridT[m * ms + tn] = x[m];
    }
    // checkpoints for a reverse sweep: the time-domain state before steps 1, K + 1, 2 K + 1, ...
    double2* ckRow = a.ckpt ? a.ckpt + inst * a.ckN * MD * (long long)N : nullptr;
    if (ckRow && a.nZ > 1) {
#pragma unroll
      for (int m = 0; m < MD; m++) ckRow[(long long)m * N + tn] = x[m];
    }
    // What a step reads is loaded during the step before (a load from L2 takes a fifth of a step): the dispersion
    // factors once, the RK4 matrix of a single mode, or the pump rows.
    constexpr bool kAhead = MD == 1;
    constexpr int kWords = kAhead ? 2 : 1;
    int4 fac[MD];
    if (a.nZ > 1) {
#pragma unroll
      for (int m = 0; m < MD; m++) fac[m] = __ldg(a.fx.tab + (long long)m * N + fk);
    }
    double2 ahead[kWords], rows[3][P];
    auto loadMatrix = [&](int i) {
      const double2* mat = reinterpret_cast<const double2*>(a.prop) + (long long)(i - 1) * 2 * N + tn;
#pragma unroll
      for (int w = 0; w < kWords; w++) ahead[w] = __ldg(mat + (long long)w * N);
    };
    auto loadRow = [&](int row, int at) {
#pragma unroll
      for (int q = 0; q < P; q++)
        rows[at][q] = S::kP > 0 ? __ldg(a.pump + q * a.pumpStride + (long long)row * N + tn) : czero();
    };
    if (a.nZ > 1) {
      if (a.prop) {
        if (kAhead) loadMatrix(1);
      } else {
        loadRow(0, 0);
        loadRow(1, 1);
        loadRow(2, 2);
      }
    }
    for (int i = 1; i < a.nZ; i++) {
      if (kAhead && a.prop) {
        const double2 e0 = ahead[0], e1 = ahead[kWords - 1], v = x[0];
        x[0] = make_double2(fma(e0.y, v.y, e0.x * v.x), fma(e1.y, v.y, e1.x * v.x));
        if (i < a.nZ - 1) loadMatrix(i + 1);
      } else if (a.prop) {
        // the RK4 step as its per-point real (2M)x(2M) matrix, stored as pairs (row r, columns 2c and
        // 2c+1) at [step][r * M + c][N]
        constexpr int D = 2 * MD;
        const double2* mat = reinterpret_cast<const double2*>(a.prop) + (long long)(i - 1) * (D * D / 2) * N;
        double in[D], outv[D];
#pragma unroll
        for (int m = 0; m < MD; m++) {
          in[2 * m] = x[m].x;
          in[2 * m + 1] = x[m].y;
        }
#pragma unroll
        for (int r = 0; r < D; r++) {
          double acc = 0.0;
#pragma unroll
          for (int cc = 0; cc < D / 2; cc++) {
            const double2 e = __ldg(mat + (long long)(r * (D / 2) + cc) * N + tn);
            acc = fma(e.x, in[2 * cc], acc);
            acc = fma(e.y, in[2 * cc + 1], acc);
          }
          outv[r] = acc;
        }
#pragma unroll
        for (int m = 0; m < MD; m++) x[m] = make_double2(outv[2 * m], outv[2 * m + 1]);
      } else {
        const double2* c = a.coef + (long long)(i - 1) * 3 * a.nCoef;
        rk4_point<S>(x, rows, c);
        if (i < a.nZ - 1) {   // row 2i is the next step's first
#pragma unroll
          for (int q = 0; q < P; q++) rows[0][q] = rows[2][q];
          loadRow(2 * i + 1, 1);
          loadRow(2 * i + 2, 2);
        }
      }
      const bool last = i == a.nZ - 1;
      const bool wantTime = !last || a.inTime || a.gridT != nullptr;
      auto storeF = [&](int m, double2 v) {
        if (a.gridF) a.gridF[m * ms + (long long)i * N + fk] = cscale(v, (double)N);
      };
      if (wantTime) {
        if (last) {
#pragma unroll
          for (int m = 0; m < MD; m++) fac[m] = __ldg(a.fx.tab + (long long)(MD + m) * N + fk);
        }
        spread_pair_all<C, K, MD>(f, x, fac, a.fx.et, a.gridF != nullptr, storeF);
        if (a.gridT) {
#pragma unroll
          for (int m = 0; m < MD; m++) a.gridT[m * ms + (long long)i * N + tn] = x[m];
        }
      } else {
        spread_fwd_all<C, MD>(f, x);
#pragma unroll
        for (int m = 0; m < MD; m++) {
          x[m] = cmul(x[m], __ldg(a.dlast + (long long)m * N + fk));
          storeF(m, x[m]);
        }
      }
      if (ckRow && !last && i % a.ckK == 0) {
#pragma unroll
        for (int m = 0; m < MD; m++) ckRow[((long long)(i / a.ckK) * MD + m) * N + tn] = x[m];
      }
    }
    if (a.nZ == 1) {
      spread_fwd_all<C, MD>(f, x);
#pragma unroll
      for (int m = 0; m < MD; m++) {
        x[m] = cmul(x[m], __ldg(a.back + (long long)m * N + fk));
        if (a.gridF) a.gridF[m * ms + fk] = cscale(x[m], (double)N);
      }
      if (a.inTime || a.gridT) {
        spread_inv_all<C, MD>(f, x);
        if (a.gridT) {
#pragma unroll
          for (int m = 0; m < MD; m++) a.gridT[m * ms + tn] = x[m];
        }
      }
    }
    // the last row is in the time domain when the input was, else in the frequency domain
    if (a.out) {
      double2* o = a.out + inst * a.outStride;
      const double sc = a.inTime ? 1.0 : (double)N;
      for (int om = 0; om < a.nOut; om++) {
#pragma unroll
        for (int m = 0; m < MD; m++)
          if (m == a.outModes[om]) o[(long long)om * N + (a.inTime ? tn : fk)] = cscale(x[m], sc);
      }
    }
  }
  cl.sync();
  spread_drain(f);
}

}  // namespace nlm
