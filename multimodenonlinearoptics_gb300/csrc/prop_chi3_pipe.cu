// prop_chi3_pipe.cu -- the Chi3 pump march and one signal propagation in one cluster of eight CTAs.
//
// Ranks 0..3 march the pump with the arithmetic of k_pump_chi3_spread (solvers/Chi3.cpp:41-70); ranks
// 4..7 propagate the signal with that of k_propagate_spread<FChi3, 4> (src/_NonlinearMedium.hpp:160-239,
// the solver's DiffEq at every step), one phase behind the pump.  The signal's step i reads pump rows
// 2i-2, 2i-1 and 2i of the time-domain grid at its own points; the pump writes rows 2p-1 and 2p in
// phase p, and the cluster barrier that ends the phase orders those writes before the signal's reads
// (barrier.cluster arrive has release and wait acquire semantics at cluster scope).  Each march alone
// is a chain of latency-bound transforms on four SMs; side by side the signal's march costs about
// nothing beyond the pump's.  The groups' exchanges wait for their own four CTAs only, so the phase
// barrier is the one place where they meet: nZ of them after the opening one, in both groups
// (pump: one after each row pair and two at the end; signal: one before each step and one at the end).
// The pump group runs the operations of k_pump_chi3_spread in the same order; the two kernels' grids
// agree to rounding (the compiler may pair multiply-adds differently in each).
#include "nlm_launch.h"
#include "prop_spread.cuh"

namespace nlm {

__global__ void __launch_bounds__(kMaxThreads) k_chi3_pump_signal_spread(const PropArgs a, const PumpMarchArgs p) {
  extern __shared__ double2 smem[];
  cg::cluster_group cl = cg::this_cluster();
  const int crank = (int)cl.block_rank();
  const int role = crank / kSpreadC;   // 0: pump march, 1: signal
  SpreadFFT f;
  const int M = a.plan.N;
  spread_init(f, smem, a.fx.twN, M, crank - role * kSpreadC, a.fx.wait);
  f.base = role * kSpreadC;
  const int N = M * kSpreadC;
  const int tn = f.rank + kSpreadC * f.t, fk = f.j + M * f.rank;
  const int nZ = a.nZ;
  cl.sync();   // every CTA of the cluster has started before the first exchange writes to its memory
  const int et = -(31 - __clz(N));   // the inverse transforms' 1/N
  if (role == 0) {
    const double invN = 1.0 / N;
    const int4 dp = fx_factor(p.dstepP[fk]);
    double2 x = spread_fwd_end(f, p.env[tn]);
    x = cmul(x, p.halfP[fk]);
    p.pf[fk] = x;
    x = cscale(spread_inv_end(f, x), invN);
    p.pt[tn] = x;
    for (int i = 1; i < p.nRows; i++) {
      const double2 r = p.rel[i - 1];
      const double a2 = cabs2(x);
      x = cmul(x, spm_factor(r.x * a2, r.y * a2));
      x = spread_pair_spec(f, x, dp, et, true, [&](double2 v) { p.pf[(long long)i * N + fk] = cscale(v, (double)N); });
      if (i < p.nRows - 1) p.pt[(long long)i * N + tn] = x;
      if ((i & 1) == 0 && i < p.nRows - 1) cl.sync();   // rows up to i are in place for step i / 2
    }
    // last row: undo half of the last pump dispersion step (each thread rereads its own bin)
    const long long last = (long long)(p.nRows - 1) * N;
    x = cmul(p.pf[last + fk], p.backP[fk]);
    p.pf[last + fk] = x;
    p.pt[last + tn] = cscale(spread_inv_end(f, x), invN);
    cl.sync();
    cl.sync();
    spread_drain(f);
    return;
  }
  const long long inst = a.instBase;
  double2 x = a.in[inst * a.inStride + (a.inTime ? tn : fk)];
  if (a.inTime) x = spread_fwd_end(f, x);
  x = cmul(x, __ldg(a.half + fk));
  if (a.gridF) a.gridF[fk] = cscale(x, (double)N);
  x = spread_inv_end(f, x);
  if (a.gridT) a.gridT[tn] = x;
  // step i: the DiffEq with pump rows 2i-2 .. 2i (plain loads: the pump group writes them during this
  // launch), then the dispersion step
  for (int i = 1; i < nZ; i++) {
    cl.sync();   // pump rows up to 2i are in place
    const double2* c = a.coef + (long long)(i - 1) * 3 * a.nCoef;
    const double2* pr = a.pump + (long long)(2 * i - 2) * N + tn;
    double2 pp[3][1] = {{pr[0]}, {pr[N]}, {pr[2 * N]}};
    double2 xm[1] = {x};
    rk4_point<FChi3>(xm, pp, c);
    const bool last = i == nZ - 1;
    auto storeF = [&](double2 v) {
      if (a.gridF) a.gridF[(long long)i * N + fk] = cscale(v, (double)N);
    };
    if (!last || a.inTime || a.gridT != nullptr) {
      x = spread_pair_spec(f, xm[0], __ldg(a.fx.tab + (last ? N : 0) + fk), a.fx.et, a.gridF != nullptr, storeF);
      if (a.gridT) a.gridT[(long long)i * N + tn] = x;
    } else {
      x = cmul(spread_fwd_end(f, xm[0]), __ldg(a.dlast + fk));
      storeF(x);
    }
  }
  cl.sync();
  spread_drain(f);
}

cudaError_t launch_chi3_pump_signal_spread(const PropArgs& a, const PumpMarchArgs& p, cudaStream_t s, int* regs) {
  const int M = a.plan.N, N = M * kSpreadC;
  if (M < 32 || M > kMaxThreads || (M & (M - 1)) != 0 || a.nZ < 2 || p.nRows != 2 * a.nZ - 1 || a.nInst != 1 ||
      a.inStride < N)
    return cudaErrorInvalidValue;
  const void* fn = (const void*)k_chi3_pump_signal_spread;
  size_t smem = 0;
  cudaFuncAttributes fa;
  cudaError_t e = exclusive_smem(fn, (size_t)spread_smem_per_point(kSpreadC) * M * sizeof(double2), &smem, &fa);
  if (e != cudaSuccess) return e;
  if (smem == 0) return cudaErrorInvalidValue;
  if (regs) *regs = fa.numRegs;
  PropArgs ac = a;
  PumpMarchArgs pc = p;
  void* args[] = {(void*)&ac, (void*)&pc};
  return launch_clustered(fn, 2 * kSpreadC, M, smem, s, 2 * kSpreadC, args);
}

}  // namespace nlm
