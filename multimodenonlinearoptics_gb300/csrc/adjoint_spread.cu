// adjoint_spread.cu -- the Chi2PDC reverse sweep (adjoint.cu) with each propagation on a cluster of four
// CTAs holding one point per thread (nlm_spread.cuh): the reverse of the forwards that run on the
// spread kernels (few rows on grids of 128 to 1024 points), whose checkpoints it reads.  Same steps as
// adjoint_cluster.cu: per segment between checkpoints the states are recomputed into per-cluster scratch
// (K > 1), then the reverse steps run: the dispersion pair as spread transforms, the transposed RK4 step
// point-wise in the time-domain ownership (the marching form with every state stored: P^T per point,
// the stage-factor gradients in a parallel launch afterwards).  The state and gradient of a point are
// read and written by the thread that owns the point in the time domain.
#include <vector>

#include "nlm_adjoint_pdc.cuh"
#include "nlm_spread.cuh"

namespace nlm {

// The transpose of step i's dispersion: forward transform, conjugate factors, inverse transform; the last step's
// gradient starts in the frequency domain.
__device__ __forceinline__ double2 spread_adjoint_dispersion(const PropArgs& a, SpreadFFT& f, double2 g, int i, int fk) {
  if (i < a.nZ - 1) return spread_pair(f, g, fx_conj(__ldg(a.fx.tab + fk)), a.fx.et);
  return spread_inv_end(f, cmulc(g, __ldg(a.dlast + fk)));
}

// a.plan.N = M (N / 4 threads per CTA); a.fx.twN: the N-point table.  d.seg: [cluster][K][N] when d.K > 1.
__global__ void __launch_bounds__(kMaxThreads) k_adjoint_pdc_spread(const PropArgs a, const AdjArgs d) {
  extern __shared__ double2 smem[];
  cg::cluster_group cl = cg::this_cluster();
  SpreadFFT f;
  const int rank = (int)cl.block_rank();
  const int M = a.plan.N;
  spread_init(f, smem, a.fx.twN, M, rank, a.fx.wait);
  cl.sync();
  const int N = M * kSpreadC;
  const int tn = rank + kSpreadC * f.t, fk = f.j + M * rank;
  const int K = d.K;
  const long long clusterId = blockIdx.x / kSpreadC, nClusters = gridDim.x / kSpreadC;
  double2* seg = K > 1 ? d.seg + clusterId * (long long)K * N : nullptr;
  for (long long local = clusterId; local < a.nInst; local += nClusters) {
    const long long inst = a.instBase + local;
    const double2* ck = d.ckpt + inst * (long long)d.nCk * N;
    double2 g = cscale(d.gout[inst * (long long)N + fk], (double)N);
    int segEnd = a.nZ - 1;
    while (segEnd >= 1) {
      const int jseg = (segEnd - 1) / K, s0 = jseg * K;
      const double2* states = ck + (long long)s0 * N;   // K = 1: checkpoint i-1 is the state s_{i-1}
      if (K > 1) {
        // states s_{s0} .. s_{segEnd-1} into seg[0 ..]
        double2 x = ck[(long long)jseg * N + tn];
        seg[tn] = x;
        for (int i = s0 + 1; i < segEnd; i++) {
          x = pdc_step_point(a, N, i, tn, x);
          x = spread_pair(f, x, __ldg(a.fx.tab + fk), a.fx.et);
          seg[(long long)(i - s0) * N + tn] = x;
        }
        states = seg;
      }
      for (int i = segEnd; i > s0; i--) {
        g = spread_adjoint_dispersion(a, f, g, i, fk);
        if (d.gp) {   // marching form: P^T per point, the stage-factor gradients afterwards in parallel
          g = pdc_march_point(a, d, N, i, tn, inst, g, true);
          continue;
        }
        const double2* c = a.coef + (long long)(i - 1) * 3 * a.nCoef;
        const double2* prev = states + (long long)(i - 1 - s0) * N;
        g = pdc_reverse_point(a, d, N, i, tn, c[0], c[1], c[2], prev[tn], g, true);
      }
      segEnd = s0;
    }
    // gradient of the input spectrum: s_0 = IFFT(half X_in)
    g = spread_fwd_end(f, g);
    d.gin[inst * (long long)N + fk] = cmulc(g, __ldg(a.half + fk));
  }
  cl.sync();
  spread_drain(f);
}

// Pipelined form for checkpoint intervals K > 1 on clusters of eight CTAs (two groups of four, as in
// k_adjoint_pdc_cluster_pipe): ranks 4..7 recompute the states of segment j-1 from its checkpoint into
// one half of STG while ranks 0..3 reverse segment j from the other half.  The groups' transforms only
// wait for their own four CTAs; one barrier of the whole cluster ends each segment iteration and hands the
// halves over.  d.seg: [cluster][2][K][N].
__global__ void __launch_bounds__(kMaxThreads) k_adjoint_pdc_spread_pipe(const PropArgs a, const AdjArgs d) {
  extern __shared__ double2 smem[];
  cg::cluster_group cl = cg::this_cluster();
  const int crank = (int)cl.block_rank();
  const int role = crank / kSpreadC;   // 0: reverse sweep, 1: recomputation
  SpreadFFT f;
  const int M = a.plan.N;
  spread_init(f, smem, a.fx.twN, M, crank - role * kSpreadC, a.fx.wait);
  f.base = role * kSpreadC;
  cl.sync();
  const int N = M * kSpreadC;
  const int tn = f.rank + kSpreadC * f.t, fk = f.j + M * f.rank;
  const int K = d.K;
  const long long clusterId = blockIdx.x / (2 * kSpreadC), nClusters = gridDim.x / (2 * kSpreadC);
  const long long bufStride = (long long)K * N;
  double2* STG = d.seg + clusterId * 2 * bufStride;
  const int nSeg = (a.nZ - 2) / K + 1;
  for (long long local = clusterId; local < a.nInst; local += nClusters) {
    const long long inst = a.instBase + local;
    const double2* ck = d.ckpt + inst * (long long)d.nCk * N;
    double2 g = czero();
    if (role == 0) g = cscale(d.gout[inst * (long long)N + fk], (double)N);
    for (int it = 0; it <= nSeg; it++) {
      if (role == 1) {
        if (it < nSeg) {
          const int jseg = nSeg - 1 - it, s0 = jseg * K, segEnd = min(s0 + K, a.nZ - 1);
          double2* stg = STG + (long long)(it & 1) * bufStride;
          double2 x = ck[(long long)jseg * N + tn];
          stg[tn] = x;
          for (int q = 1; q <= K; q++) {
            const int i = s0 + q;
            if (i < segEnd) {
              x = pdc_step_point(a, N, i, tn, x);
              x = spread_pair(f, x, __ldg(a.fx.tab + fk), a.fx.et);
              stg[(long long)q * N + tn] = x;
            }
          }
        }
      } else {
        if (it >= 1) {
          const int jseg = nSeg - it, s0 = jseg * K, segEnd = min(s0 + K, a.nZ - 1);
          const double2* stg = STG + (long long)((it - 1) & 1) * bufStride;
          for (int q = 0; q < K; q++) {
            const int i = segEnd - q;
            if (i > s0) {
              const double2* prev = stg + (long long)(i - 1 - s0) * N;
              g = spread_adjoint_dispersion(a, f, g, i, fk);
              const double2* c = a.coef + (long long)(i - 1) * 3 * a.nCoef;
              g = pdc_reverse_point(a, d, N, i, tn, c[0], c[1], c[2], prev[tn], g, true);
            }
          }
        }
      }
      cl.sync();
    }
    if (role == 0) {
      g = spread_fwd_end(f, g);
      d.gin[inst * (long long)N + fk] = cmulc(g, __ldg(a.half + fk));
    }
  }
  cl.sync();
  spread_drain(f);
}

// Stage-factor gradient groups beside the pipelined sweep, on clusters of 4 (2 + G) CTAs, for
// checkpoint intervals K > 1 with the RK4 propagator matrices built.  In k_adjoint_pdc_spread_pipe the
// reverse group also runs the transposed stages of every step (about 90 FP64 operations per point),
// so the recomputing group, whose step is 4 FMAs, waits at every shared barrier.  Here:
//   ranks 4..7 (group 1) recompute the states of segment j-1 into STG, as there;
//   ranks 0..3 (group 0) reverse segment j: the dispersion pair, then P^T per point (4 FMAs), storing
//     the gradient after each step's RK4 in GP;
//   ranks 8.. (groups 2 .. 1 + G) compute the stage-factor gradients of segment j+1, reversed in the
//     previous iteration, from its states (STG) and stored gradients (GP).  Group 2 + s takes the steps
//     q = s mod G of the segment (q = 0 .. K-1).
// G = 2 (sixteen CTAs) halves the stage groups' work; G = 1 (twelve) is the form for GPUs without 16-CTA
// clusters.  STG holds three segments (written by group 1 at iteration it, read by group 0 at it+1 and by the
// stage groups at it+2) and GP two; one barrier of the whole cluster ends each iteration.  After the last
// iteration all groups share the stage-factor gradients of segment 0, by steps.
// d.seg: [cluster][3 + 2][K][N].
template <int G>
__global__ void __launch_bounds__(kMaxThreads) k_adjoint_pdc_spread_stage(const PropArgs a, const AdjArgs d) {
  constexpr int kGroups = 2 + G;
  extern __shared__ double2 smem[];
  cg::cluster_group cl = cg::this_cluster();
  const int crank = (int)cl.block_rank();
  const int role = crank / kSpreadC;   // 0: reverse sweep, 1: recomputation, 2..: stage-factor gradients
  const int lr = crank - role * kSpreadC;
  const int M = a.plan.N;
  const int N = M * kSpreadC;
  SpreadFFT f;
  if (role < 2) {
    spread_init(f, smem, a.fx.twN, M, lr, a.fx.wait);
    f.base = role * kSpreadC;
  }
  cl.sync();
  const int tn = lr + kSpreadC * spread_time_index((int)threadIdx.x, M), fk = (int)threadIdx.x + M * lr;
  const int pc = lr * M + (int)threadIdx.x;   // the point of this thread's stage-factor gradients
  const int K = d.K;
  const long long clusterId = blockIdx.x / (kGroups * kSpreadC), nClusters = gridDim.x / (kGroups * kSpreadC);
  const long long bufStride = (long long)K * N;
  double2* STG = d.seg + clusterId * 5 * bufStride;
  double2* GP = STG + 3 * bufStride;
  const int nSeg = (a.nZ - 2) / K + 1;
  // a stage group's step in flight: its forward stages, state and gradient (step 0: none)
  PdcStages st{};
  double2 sx = czero(), sg = czero();
  int si = 0;
  auto stageLoad = [&](const double2* stg, const double2* gps, int i, int s0) {
    sx = stg[(long long)(i - 1 - s0) * N + pc];
    sg = gps[(long long)(i - 1 - s0) * N + pc];
    const double2* c = a.coef + (long long)(i - 1) * 3 * a.nCoef;
    st = pdc_stages(a, N, i, pc, c[0], c[1], c[2], sx);
    si = i;
  };
  auto stageFinish = [&]() {
    if (si == 0) return;
    double2 ga0, ga1, ga2;
    pdc_stages_reverse(st, sx, sg, ga0, ga1, ga2);
    pdc_store_ga(d, N, si, pc, ga0, ga1, ga2);
    si = 0;
  };
  for (long long local = clusterId; local < a.nInst; local += nClusters) {
    const long long inst = a.instBase + local;
    const double2* ck = d.ckpt + inst * (long long)d.nCk * N;
    double2 g = czero();
    if (role == 0) g = cscale(d.gout[inst * (long long)N + fk], (double)N);
    for (int it = 0; it <= nSeg; it++) {
      if (role == 1) {
        if (it < nSeg) {
          const int jseg = nSeg - 1 - it, s0 = jseg * K, segEnd = min(s0 + K, a.nZ - 1);
          double2* stg = STG + (long long)(it % 3) * bufStride;
          double2 x = ck[(long long)jseg * N + tn];
          stg[tn] = x;
          for (int q = 1; q <= K; q++) {
            const int i = s0 + q;
            if (i < segEnd) {
              x = pdc_step_point(a, N, i, tn, x);
              x = spread_pair(f, x, __ldg(a.fx.tab + fk), a.fx.et);
              stg[(long long)q * N + tn] = x;
            }
          }
        }
      } else if (role == 0) {
        if (it >= 1) {
          const int jseg = nSeg - it, s0 = jseg * K, segEnd = min(s0 + K, a.nZ - 1);
          double2* gps = GP + (long long)(it & 1) * bufStride;
          for (int q = 0; q < K; q++) {
            const int i = segEnd - q;
            if (i > s0) {
              g = spread_adjoint_dispersion(a, f, g, i, fk);
              gps[(long long)(i - 1 - s0) * N + tn] = g;
              g = pdc_transpose_point(a, N, i, tn, g);
            }
          }
        }
      } else {
        if (it >= 2) {
          const int sub = role - 2;
          const int jseg = nSeg - it + 1, s0 = jseg * K, segEnd = min(s0 + K, a.nZ - 1);
          const double2* stg = STG + (long long)((it - 2) % 3) * bufStride;
          const double2* gps = GP + (long long)((it - 1) & 1) * bufStride;
          for (int q = 0; q < K; q++) {
            stageFinish();   // the step loaded in an earlier slot
            const int i = s0 + 1 + q;
            if (q % G == sub && i <= segEnd) stageLoad(stg, gps, i, s0);
          }
          stageFinish();
        }
      }
      cl.sync();
    }
    if (role == 0) {
      g = spread_fwd_end(f, g);
      d.gin[inst * (long long)N + fk] = cmulc(g, __ldg(a.half + fk));
    }
    // segment 0 (reversed in the last iteration): its steps shared by all groups
    {
      const int segEnd = min(K, a.nZ - 1);
      const double2* stg = STG + (long long)((nSeg - 1) % 3) * bufStride;
      const double2* gps = GP + (long long)(nSeg & 1) * bufStride;
      for (int i = 1 + role; i <= segEnd; i += kGroups) {
        stageLoad(stg, gps, i, 0);
        stageFinish();
      }
    }
    cl.sync();
  }
  if (role < 2) spread_drain(f);
}

void add_kernels_adjoint_spread(std::vector<KernelEntry>& t) {
  // key + 300: one propagation per cluster of four CTAs; key + 200: pipelined on eight; R = 1 point
  // per thread
  t.push_back({kKindAdjoint, kChi2PDC + 300, 1, (const void*)k_adjoint_pdc_spread});
  t.push_back({kKindAdjoint, kChi2PDC + 200, 1, (const void*)k_adjoint_pdc_spread_pipe});
  // key + 500 / + 600: stage-factor gradients in one / two groups of their own, on twelve / sixteen
  // CTAs (checkpoints with the propagator matrices)
  t.push_back({kKindAdjoint, kChi2PDC + 500, 1, (const void*)k_adjoint_pdc_spread_stage<1>});
  t.push_back({kKindAdjoint, kChi2PDC + 600, 1, (const void*)k_adjoint_pdc_spread_stage<2>});
}

}  // namespace nlm
