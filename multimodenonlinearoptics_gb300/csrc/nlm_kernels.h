// nlm_kernels.h -- launch interface between the host engine (engine.h) and the kernels.
// Plain C++ (no device code): included by both nvcc and g++ translation units.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace nlm {

constexpr int kMaxModes = 4;
constexpr int kMaxPumps = 2;
constexpr int kMaxCoefs = 8;
constexpr int kMaxFFT = 8192;   // largest grid of the fused kernels
constexpr int kTablePad = 16;   // zeroed values after every per-point device table (padded ownership reads)

// Plan of an N-point transform held by T threads of R points each.  gen == 0: N a power of two and
// T = N / R, radix-8/4/2 passes on the register ownership (nlm_device.cuh, fft_regs).  gen == 1: any N,
// T = ceil(N / R) (thread j owns the points j + v T that are below N), passes of any radix through
// shared memory (fft_general).
struct FFTPlanH {
  int N, T, nPass;
  int radix[16];
  int gen;
  int R;   // points per thread the plan was made for
};

// How a cluster kernel waits for an exchange between its CTAs (nlm_spread.cuh).
constexpr int kExchangePolls = 1 << 16;
struct ExchangeWait {
  int* err;    // host memory, raised when an exchange does not arrive
  int polls;   // polls before a wait gives up
};

// Block fixed-point transforms (nlm_fx.cuh): the twiddles and dispersion tables as Q62 integers, each complex
// value as balanced 32-bit halves {re high, re low, im high, im low} with value (h 2^32 + l) 2^(et - 62).
struct FxArgs {
  const int4* tw;    // the plan's twiddles, pass by pass (one-CTA kernels)
  // grids with a prime factor above 7: the convolution form on L points (0: none), its chirp exp(-pi i t^2 / N) and the
  // transform of the conjugate chirp over L, relative to a power of two that sh carries
  int L;
  const int4* chirp;
  const int4* conv;
  const int4* root;  // exp(-2 pi i q / r) of the odd radices (fx_root_at)
  const int4* twN;   // exp(-2 pi i m / N), m < N (cluster kernels with one point per thread)
  const int4* tab;   // [dispStep, last, half][mode][N], each with its 1/N
  int et;            // exponent of the tables: 2^et is at least their largest modulus
  const int4* raman; // Chi3GNLSE: Raman response and self-steepening factors (1/N folded in), their exponents
  const int4* steep;
  int etRaman, etSteep;
  int A0;            // log2 bound of the field's 2-norm on entry
  int sh;            // places a transform shifts right in all
  ExchangeWait wait; // cluster kernels
  int ls;            // places the table product after a forward transform is shifted left
};

// Places a pass of radix r shifts its values right, in a block fixed-point transform whose 2-norm stands `level`
// half bits above its entry: the fewest that keep it within kFxPeak half bits after the pass (each pass grows the
// norm by sqrt(r)).  The higher the norm stands, the less a rounding weighs.  Updates level.
constexpr int kFxPeak = 4;
constexpr int kFxA0 = 60;   // log2 bound of the 2-norm on entry
__host__ __device__ constexpr int fx_log2(int r) { return r >= 16 ? 4 : r >= 8 ? 3 : r >= 4 ? 2 : r >= 2 ? 1 : 0; }
__host__ __device__ constexpr int fx_pass_shift(int level, int r) {
  return level + fx_log2(r) <= kFxPeak ? 0 : (level + fx_log2(r) - kFxPeak + 1) / 2;
}
// The same on the general plan, whose radices are not all powers of two, in sixteenths of a bit: a pass of radix r adds
// log2(r) / 2 bits (rounded up), and the norm stays within 2 bits of its entry.  The first pass never shifts.
__host__ __device__ constexpr int fx_gen_growth(int r) {
  return r == 2 ? 8 : r == 3 ? 13 : r == 4 ? 16 : r == 5 ? 19 : r == 7 ? 23 : 24;
}
__host__ __device__ constexpr int fx_gen_shift(int level, int r) {
  return level + fx_gen_growth(r) <= 32 ? 0 : (level + fx_gen_growth(r) - 32 + 15) / 16;
}

// v / 2^r (0 <= r <= 62) rounded to nearest, ties to even.  r is mostly 1 to 3, where every 2^r-th value is a tie: ties
// upwards would move the mean of every field by 2^-r / 2 in every forward transform.  (From r = 32 on, where ties are
// one value in 2^32, the bit that breaks them is another one.)
__host__ __device__ inline long long fx_align(long long v, int r) {
  const int one = r > 0;
  const int odd = (int)((unsigned)v >> (r < 31 ? r : 31)) & one;
  return (v + (((1LL << r) >> 1) - one) + odd) >> r;
}

// Shared memory of a CTA of the block fixed-point kernels: the twiddles, two exchange buffers of
// fx_buffer(N) values and one pair of words per warp (at most 16).
__host__ __device__ constexpr int fx_buffer(int N) { return N + N / 8; }
constexpr size_t fx_smem(int N) { return (size_t)(N + 2 * fx_buffer(N)) * 16 + 16 * 8; }

// Arguments of every propagation kernel (batched impulses, dense rows, one full grid).
struct PropArgs {
  FFTPlanH plan;          // mirrors nlm::FFTPlan
  int R;                  // points per thread per mode
  int nModes;             // signal modes
  int nZ;                 // nZSteps
  long long nInst;        // independent propagations in this launch
  long long instBase;     // global index of the launch's first propagation
  int ipc;                // propagations per CTA
  unsigned long long* work;  // zeroed work counter for dynamic scheduling of the groups; null: static
  // input description
  int inKind;             // 0: impulses (Green's function), 1: dense rows
  int inTime;             // inputs and outputs in the time domain
  const double2* in;      // dense rows
  long long inStride;     // complex elements between rows
  int inChannels;         // number of N-blocks per row
  int inputMode;          // mode receiving a single N-block
  int impModes[kMaxModes];// impulses: input mode of impulse group im = inst / (2N)
  // output description (last row of the selected modes)
  int nOut;
  int outModes[kMaxModes];
  double2* out;
  long long outStride;
  // point-wise tables (device)
  const double2* tw;      // N twiddles exp(-2 pi i m / N)
  const double2* dstep;   // [mode][N] dispStep / N
  const double2* dlast;   // [mode][N] dispStep * exp(-i dz/2 D) / N
  const double2* half;    // [mode][N] exp(+i dz/2 D) / N
  const double2* back;    // [mode][N] exp(-i dz/2 D) / N
  const double* prop;     // linear propagator [(nZ-1)][(2M)^2][N]
  const double2* pump;    // pumpTime [pump][nZStepsP][N]
  long long pumpStride;   // nZStepsP * N
  int nPumps;
  const double2* coef;    // [(nZ-1)][3][nCoef]
  int nCoef;
  // full grids of a single propagation (runSignalSimulation); null otherwise
  double2* gridF;         // [mode][nZ][N]
  double2* gridT;
  // checkpoints of the forward states for the adjoint: state s_i (time domain, all modes) is stored
  // at ckpt[((inst * ckN) + i / ckK) * nModes + m][N] when i % ckK == 0 and i < nZ - 1
  double2* ckpt;
  int ckK, ckN;
  // Chi3GNLSE adjoint forward on clusters: the stage inputs y_s and convolutions u2_s of every step
  // (time domain) at stages[((inst * (nZ - 1) + i - 1) * 8 + {s, 4 + s})][N]; null otherwise
  double2* stages;
  // Chi3GNLSE tables
  const double2* raman;   // ramanResponse / N
  const double2* steep;   // (nlStep0 + nlStep1 * omega) / N
  const double* relInt;   // [(nZ-1)][3] relative intensity at i-1, i-1/2, i
  FxArgs fx;              // block fixed-point transforms
};

// Arguments of the reverse (adjoint) sweep.
struct AdjArgs {
  const double2* gout;   // [nInst][N]: dL/dRe X + i dL/dIm X of the output spectrum
  const double2* ckpt;   // forward checkpoints (PropArgs::ckpt layout)
  int K, nCk;            // checkpoint interval and count
  double2* seg;          // scratch [slot][K][N] for the recomputed states of one segment (K > 1)
  double2* ga;           // [(nZ-1)][3][N] accumulated gradients of the stage factors a_s = c_s P_s
  double2* gin;          // [nInst][N]: gradient with respect to the input spectrum
  int single;            // 1: a single instance, whose stage-factor gradients are stored without atomics
  // marching form (checkpoint interval 1 with the propagator matrices): the gradient after every
  // step's RK4, [nInst][nZ-1][N], for k_adj_stage_grads; null otherwise
  double2* gp;
};

// Registry of the propagation kernels.  The host engine launches them generically with
// cudaLaunchKernel(fn, grid, block, {&PropArgs[, &scratch]}, smem, stream).
enum KernelKind : int {
  kKindDirect = 0,     // k_propagate_direct<Solver, R>      key = solver id
  kKindLinear = 1,     // k_propagate_linear<M, R>           key = number of modes M
  kKindGnlse = 2,      // k_propagate_gnlse<R>               key = solver id (Chi3GNLSE); extra arg: scratch
  kKindBuildProp = 3,  // k_build_propagator<Solver>         key = solver id, R = 0
  kKindAdjoint = 4,    // k_adjoint_pdc<R>                   key = solver id; args (PropArgs, AdjArgs)
  kKindRagged = 5,     // k_propagate_ragged<Solver, R>      key = solver id; args (items, nItems, work)
  kKindLinearFF = 6,   // k_propagate_linear_ff<R, SMALL>    key = M + 10 SMALL; args (PropArgs, FFTables)
  kKindCluster = 7,    // k_propagate_cluster<Solver, C>     key = solver id, R = C; cluster launch
  kKindSpreadFused = 8, // k_propagate_spread<Solver, C, M>  key as kKindCluster (R = 1): modes transformed together
  kKindFxLinear = 9,   // k_fx_linear<M, R, N>               key = modes + 1000 log2 N; args (PropArgs)
  kKindFxDirect = 10,  // k_fx_direct<Solver, R>             key = solver id; args (PropArgs)
  kKindFxGnlse = 11,   // k_fx_gnlse<R, N>                   key = solver id (+ 400: pairs) + 1000 log2 N; extra arg: scratch
  kKindFxRows = 13,    // k_fx_rows<R, N>                    key = log2 N, kConvKey or kGenKey
  kKindFxPump = 12     // k_fx_pump_chi3<R, N>               key = kConvKey, kGenKey; args (PropArgs, PumpMarchArgs)
};

// Float-float copies (float4 {re.hi, re.lo, im.hi, im.lo} per complex value) of the tables of a
// single-mode linear propagation, for the double-float kernel on the FP32 pipes.
struct FFTables {
  const float4* tw;      // N twiddles
  const float4* dstep;   // [N]
  const float4* dlast;
  const float4* half;
  const float4* back;
  const float4* prop;    // [(nZ-1)][2][N]: pairs (M00, M01) and (M10, M11)
};
struct KernelEntry {
  int kind;
  int key;
  int R;
  const void* fn;
};
// All registered kernels (filled on first call).
const KernelEntry* kernel_table(int* count);
cudaError_t launch_fft_rows(const double2* in, double2* out, long long rows, const FFTPlanH& plan,
                            const double2* tw, bool inverse, double scale, const double2* postMul,
                            cudaStream_t s);
cudaError_t launch_pump_linear(const double2* freq0, const double* disp, double dzp, int nRows, int N,
                               double2* pumpFreq, cudaStream_t s);
cudaError_t launch_scale_rows(double2* a, const double* scale, int nRows, int N, cudaStream_t s);
// stage-factor gradients of every step and point from the marching form's stored gradients (rows
// summed): d.ga = sum over rows of the stage chain at (state before the step, gradient after it)
cudaError_t launch_adj_stage_grads(const PropArgs& a, const AdjArgs& d, int N, long long rows, cudaStream_t s);
cudaError_t launch_pump_chi3(double2* pumpFreq, double2* pumpTime, const double2* env, const double2* halfP,
                             const double2* dstepP, const double2* backP, const double2* rel, int nRows,
                             const FFTPlanH& plan, const double2* tw, cudaStream_t s);
// the same march over a 4-CTA cluster; localPlan is the (N/4)-point plan with four points per thread
cudaError_t launch_pump_chi3_cluster(double2* pumpFreq, double2* pumpTime, const double2* env, const double2* halfP,
                                     const double2* dstepP, const double2* backP, const double2* rel, int nRows,
                                     const FFTPlanH& localPlan, const double2* tw, cudaStream_t s);
// Shared memory of a CTA of the one-point-per-thread cluster kernels (prop_spread.cu) of C CTAs, in
// double2 values per point of the CTA: M-point twiddles, two exchange buffers, two halves of C receive
// rows.
constexpr long long spread_smem_per_point(int C) { return 3 + 2LL * C; }
// The same for the kernels that transform their K modes together (kKindSpreadFused): twiddles, two
// K-field exchange buffers, two halves of C x K receive rows.
constexpr long long spread_smem_per_point_k(int C, int K) { return 1 + 2LL * K + 2LL * C * K; }
constexpr long long kSpreadSmemPerPoint = spread_smem_per_point(4);
// Registry key offset of the instantiations for the general plan (FFTPlanH::gen == 1): grids that are
// not powers of two (kKindDirect, kKindLinear, kKindGnlse).
constexpr int kGenKey = 2000;
// and (kKindRagged) of the block fixed-point kernels
constexpr int kFxRaggedKey = 1000;
// and of their convolution form, where it needs a kernel of its own (kKindFxDirect's runtime-size kernels serve it too)
constexpr int kConvKey = 3000;
// Registry key offset (kKindCluster) of the one-point-per-thread kernels on eight CTAs, and on sixteen.
constexpr int kSpreadWideKey = 800;
constexpr int kSpreadW16Key = 900;

// Chi3 pump march on a 4-CTA cluster with one point per thread (prop_spread.cu); N = 4 M, M a power of
// two from 32 to 1024.
cudaError_t launch_pump_chi3_spread(double2* pumpFreq, double2* pumpTime, const double2* env, const double2* halfP,
                                    const double2* dstepP, const double2* backP, const double2* rel, int nRows, int N,
                                    const int4* tw, ExchangeWait wait, cudaStream_t s);

// The Chi3 pump march's grids and per-point tables (k_pump_chi3_spread's arguments).
struct PumpMarchArgs {
  double2* pf;            // [nRows][N] frequency-domain grid
  double2* pt;            // [nRows][N] time-domain grid
  const double2* env;     // [N] time-domain envelope
  const double2* halfP;   // [N] half a dispersion step
  const double2* dstepP;  // [N] a dispersion step, 1/N folded in
  const double2* backP;   // [N] half a step back (the last row)
  const double2* rel;     // [nRows] nonlinear step factors
  int nRows;
};

// The Chi3 pump march and one signal propagation (a: the signal's launch, a.pump = p.pt, a.nInst = 1)
// pipelined on one cluster of eight CTAs (prop_chi3_pipe.cu); N = 4 M, M a power of two from 32 to
// 1024, p.nRows = 2 a.nZ - 1.  regs (optional): the kernel's registers per thread.
cudaError_t launch_chi3_pump_signal_spread(const PropArgs& a, const PumpMarchArgs& p, cudaStream_t s,
                                           int* regs = nullptr);
cudaError_t launch_green_epilogue(const double2* raw, long long rawStride, int N, int nIn, int nOut,
                                  const double2* blockScale, const uint8_t* blockShift, double2* C,
                                  double2* S, cudaStream_t s);
cudaError_t launch_pump_from(const double2* otherSignalFreq, int otherRows, double ratio, double otherDz,
                             const double* dispPump, const double* otherDispSign, double dzp, double beta1Delay,
                             const double* omega, int nRowsP, int N, double z, double otherZ, double2* pumpFreq,
                             cudaStream_t s);
cudaError_t launch_cgemm_compose(const double2* Ci, const double2* Si, const double2* C, const double2* S,
                                 int rows, int inner, int cols, double2* Cout, double2* Sout, cudaStream_t s);
// dst[k] = float-float split of src[k] for k < n (segments of several arrays in one launch)
struct SplitSeg {
  const double2* src;
  float4* dst;
  long long n;
};
cudaError_t launch_split_ff(const SplitSeg* segs, int nSegs, cudaStream_t s);
cudaError_t launch_fp64_peak(double* out, int iters, int blocks, int threads, cudaStream_t s);
cudaError_t launch_fp64_mma_peak(double* out, int iters, int blocks, int threads, cudaStream_t s);
// Green's-function consumers (greens_quadrature.cu): quadrature-basis Z and the a-basis block matrix
cudaError_t launch_quadrature_z(const double2* C, const double2* S, long long rows, long long cols, double* Z,
                                cudaStream_t s);
cudaError_t launch_abasis_z(const double2* C, const double2* S, long long rows, long long cols, double2* Za,
                            cudaStream_t s);
// Post-processing of the adjoint of Chi2PDC (adjoint.cu)
cudaError_t launch_adj_pump_rows(const double2* ga, const double2* coef, const double* prof, int nZ, int N,
                                 double2* gP, cudaStream_t s);
cudaError_t launch_adj_pump_reduce(const double2* fgP, const double* disp, double dzp, int nRowsP, int N,
                                   double2* gF0, cudaStream_t s);
cudaError_t launch_adj_coef_reduce(const double2* ga, const double2* pump, int nZ, int N, double2* gc,
                                   cudaStream_t s);

}  // namespace nlm
