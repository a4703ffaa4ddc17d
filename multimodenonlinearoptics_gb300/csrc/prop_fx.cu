// prop_fx.cu -- instantiations of the block fixed-point kernels of the pump-driven solvers.
#include <vector>

#include "prop_fx.cuh"

namespace nlm {

void add_kernels_fx(std::vector<KernelEntry>& t) {
  // key = modes + 1000 * log2 N
#define NLM_FX(M, R, LOG) t.push_back({kKindFxLinear, M + 1000 * LOG, R, (const void*)k_fx_linear<M, R, 1 << LOG>});
  NLM_FX(1, 4, 7)
  NLM_FX(1, 8, 8)
  NLM_FX(1, 8, 9)
  NLM_FX(1, 8, 10)
  NLM_FX(1, 8, 11)
  NLM_FX(1, 8, 12)
  NLM_FX(2, 4, 7)
  NLM_FX(2, 4, 8)
  NLM_FX(2, 4, 9)
  NLM_FX(2, 4, 10)
  NLM_FX(2, 4, 11)
  NLM_FX(2, 8, 12)
#undef NLM_FX
  // + 500: half the points per thread, for launches that leave schedulers idle (engine.h, fxFew)
#define NLM_FX(M, R, LOG) t.push_back({kKindFxLinear, M + 500 + 1000 * LOG, R, (const void*)k_fx_linear<M, R, 1 << LOG>});
  NLM_FX(1, 2, 7)
  NLM_FX(1, 4, 8)
  NLM_FX(1, 4, 9)
  NLM_FX(1, 4, 10)
  NLM_FX(1, 4, 11)
  NLM_FX(2, 2, 7)
  NLM_FX(2, 2, 8)
  NLM_FX(2, 2, 9)
#undef NLM_FX
  // key + kGenKey: grids that are not powers of two
  t.push_back({kKindFxLinear, 1 + kGenKey, 8, (const void*)k_fx_linear<1, 8, kFxGen>});
  t.push_back({kKindFxLinear, 2 + kGenKey, 4, (const void*)k_fx_linear<2, 4, kFxGen>});
  t.push_back({kKindFxLinear, 2 + kGenKey, 8, (const void*)k_fx_linear<2, 8, kFxGen>});
  // four modes: one kernel for every size (its fields fill the registers whatever the offsets are)
  for (int log = 7; log <= 11; log++) t.push_back({kKindFxLinear, 4 + 1000 * log, 4, (const void*)k_fx_linear<4, 4>});
  // key + kConvKey: the convolution form
  t.push_back({kKindFxLinear, 1 + kConvKey, 8, (const void*)k_fx_linear<1, 8>});
  t.push_back({kKindFxLinear, 1 + kConvKey, 4, (const void*)k_fx_linear<1, 4>});
  t.push_back({kKindFxLinear, 2 + kConvKey, 8, (const void*)k_fx_linear<2, 8>});
  t.push_back({kKindFxLinear, 2 + kConvKey, 4, (const void*)k_fx_linear<2, 4>});
  t.push_back({kKindFxLinear, 4 + kConvKey, 4, (const void*)k_fx_linear<4, 4>});
}

}  // namespace nlm
