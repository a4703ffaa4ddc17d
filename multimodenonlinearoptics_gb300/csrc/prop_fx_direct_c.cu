// prop_fx_direct_c.cu -- block fixed-point kernels of the fully nonlinear solvers (see prop_fx_direct_a.cu).
#include <vector>

#include "prop_fx.cuh"

namespace nlm {

void add_kernels_fx_direct_c(std::vector<KernelEntry>& t) {
#define NLM_FX(S, id, R) t.push_back({kKindFxDirect, id, R, (const void*)k_fx_direct<S, R>});
#define NLM_FXG(S, id, R) t.push_back({kKindFxDirect, id + kGenKey, R, (const void*)k_fx_direct<S, R, kFxGen>});
  NLM_FX(FChi2SHG, kChi2SHG, 4)
  NLM_FXG(FChi2SHG, kChi2SHG, 4)
  NLM_FX(FChi2SHG, kChi2SHG, 8)
  NLM_FXG(FChi2SHG, kChi2SHG, 8)
  NLM_FX(FChi2ASHG, kChi2ASHG, 4)
  NLM_FXG(FChi2ASHG, kChi2ASHG, 4)
  NLM_FX(FChi2ASHG, kChi2ASHG, 8)
  NLM_FXG(FChi2ASHG, kChi2ASHG, 8)
  NLM_FX(FChi2SHGXPM, kChi2SHGXPM, 4)
  NLM_FXG(FChi2SHGXPM, kChi2SHGXPM, 4)
  NLM_FX(FChi2SHGXPM, kChi2SHGXPM, 8)
  NLM_FXG(FChi2SHGXPM, kChi2SHGXPM, 8)
  NLM_FX(FChi2SHGOPA, kChi2SHGOPA, 4)
  NLM_FXG(FChi2SHGOPA, kChi2SHGOPA, 4)
  NLM_FX(FChi2DSFG, kChi2DSFG, 4)
  NLM_FXG(FChi2DSFG, kChi2DSFG, 4)
#undef NLM_FX
#undef NLM_FXG
}

}  // namespace nlm
