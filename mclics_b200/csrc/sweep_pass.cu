// Colour passes: which set of kernels (sweep_pass_kernels.cu) a model's options need.
#include "sweep_fused.cuh"

namespace mcl {

template <int POT, bool FLIP, bool CHIRAL, bool FIELD>
cudaError_t launch_pass_gp(const ModelDev &m, const FusedArgs &a, const FusedLaunch &l);

// The sets of options there are: a dipole field brings its flips with it, and pears always flip.
template <int POT, bool CHIRAL>
static cudaError_t by_options(const ModelDev &m, const FusedArgs &a, const FusedLaunch &l) {
  if (l.flip) return l.field ? launch_pass_gp<POT, true, CHIRAL, true>(m, a, l) : cudaErrorInvalidValue;
  return l.field ? launch_pass_gp<POT, false, CHIRAL, true>(m, a, l) : launch_pass_gp<POT, false, CHIRAL, false>(m, a, l);
}

cudaError_t launch_pass_ll(const ModelDev &m, const FusedArgs &a, const FusedLaunch &l) {
  return l.chiral ? cudaErrorInvalidValue : by_options<POT_LL, false>(m, a, l);
}

cudaError_t launch_pass_ghrl(const ModelDev &m, const FusedArgs &a, const FusedLaunch &l) {
  return l.chiral ? by_options<POT_GHRL, true>(m, a, l) : by_options<POT_GHRL, false>(m, a, l);
}

cudaError_t launch_pass_pear(const ModelDev &m, const FusedArgs &a, const FusedLaunch &l) {
  if (!l.flip || l.chiral) return cudaErrorInvalidValue;
  return l.field ? launch_pass_gp<POT_PEAR, true, false, true>(m, a, l)
                 : launch_pass_gp<POT_PEAR, true, false, false>(m, a, l);
}

}  // namespace mcl
