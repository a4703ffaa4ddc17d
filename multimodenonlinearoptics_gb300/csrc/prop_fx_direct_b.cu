// prop_fx_direct_b.cu -- further block fixed-point kernels with the solvers' DiffEq (see prop_fx_direct_a.cu).
#include <vector>

#include "prop_fx.cuh"

namespace nlm {

void add_kernels_fx_direct_b(std::vector<KernelEntry>& t) {
#define NLM_FX(S, id, R) t.push_back({kKindFxDirect, id, R, (const void*)k_fx_direct<S, R>});
#define NLM_FXG(S, id, R) t.push_back({kKindFxDirect, id + kGenKey, R, (const void*)k_fx_direct<S, R, kFxGen>});
  NLM_FX(FChi2PDCII, kChi2PDCII, 4)
  NLM_FXG(FChi2PDCII, kChi2PDCII, 4)
  NLM_FX(FChi2PDCII, kChi2PDCII, 8)
  NLM_FXG(FChi2PDCII, kChi2PDCII, 8)
  NLM_FX(FChi2SFGOPA, kChi2SFGOPA, 4)
  NLM_FXG(FChi2SFGOPA, kChi2SFGOPA, 4)
  NLM_FX(FChi2SFGOPA, kChi2SFGOPA, 8)
  NLM_FXG(FChi2SFGOPA, kChi2SFGOPA, 8)
  NLM_FX(FChi2SFGXPM, kChi2SFGXPM, 4)
  NLM_FXG(FChi2SFGXPM, kChi2SFGXPM, 4)
  NLM_FX(FChi2SFGXPM, kChi2SFGXPM, 8)
  NLM_FXG(FChi2SFGXPM, kChi2SFGXPM, 8)
  NLM_FX(FChi2SFGII, kChi2SFGII, 4)
  NLM_FXG(FChi2SFGII, kChi2SFGII, 4)
#undef NLM_FX
#undef NLM_FXG
}

}  // namespace nlm
