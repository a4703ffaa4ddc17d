// prop_fx_direct_a.cu -- block fixed-point kernels with the DiffEq of the pump-driven solvers (prop_fx.cuh).
// One mode: eight points per thread from 256 points, four at 128.  Two modes: four points per thread up to 2048
// points, eight at 4096.  Four modes: four points per thread up to 2048 points.
#include <vector>

#include "prop_fx.cuh"

namespace nlm {

void add_kernels_fx_direct_a(std::vector<KernelEntry>& t) {
#define NLM_FX(S, id, R) t.push_back({kKindFxDirect, id, R, (const void*)k_fx_direct<S, R>});
#define NLM_FXG(S, id, R) t.push_back({kKindFxDirect, id + kGenKey, R, (const void*)k_fx_direct<S, R, kFxGen>});
  NLM_FX(FChi3, kChi3, 8)
  NLM_FXG(FChi3, kChi3, 8)
  NLM_FX(FChi3, kChi3, 4)
  NLM_FX(FChi2PDC, kChi2PDC, 8)
  NLM_FXG(FChi2PDC, kChi2PDC, 8)
  NLM_FX(FChi2PDC, kChi2PDC, 4)
  NLM_FX(FChi2SFG, kChi2SFG, 4)
  NLM_FXG(FChi2SFG, kChi2SFG, 4)
  NLM_FX(FChi2SFG, kChi2SFG, 8)
  NLM_FXG(FChi2SFG, kChi2SFG, 8)
  NLM_FX(FChi2AFC, kChi2AFC, 4)
  NLM_FXG(FChi2AFC, kChi2AFC, 4)
  NLM_FX(FChi2AFC, kChi2AFC, 8)
  NLM_FXG(FChi2AFC, kChi2AFC, 8)
  NLM_FX(FChi2SFGPDC, kChi2SFGPDC, 4)
  NLM_FXG(FChi2SFGPDC, kChi2SFGPDC, 4)
  NLM_FX(FChi2SFGPDC, kChi2SFGPDC, 8)
  NLM_FXG(FChi2SFGPDC, kChi2SFGPDC, 8)
#undef NLM_FX
#undef NLM_FXG
}

}  // namespace nlm
