// Resident-sweep kernels of one potential (instantiations split across files so they compile in parallel).
#include "sweep_resident.cuh"

namespace mcl {

cudaError_t launch_resident_ghrl_chiral(const ModelDev &m, const ResidentArgs &a, const ResidentLaunch &l) {
  if (l.flip == false && l.field == false) return launch_resident_gp<POT_GHRL, false, true, false>(m, a, l);
  if (l.flip == false && l.field == true) return launch_resident_gp<POT_GHRL, false, true, true>(m, a, l);
  if (l.flip == true && l.field == true) return launch_resident_gp<POT_GHRL, true, true, true>(m, a, l);
  return cudaErrorInvalidValue;  // the combinations the colour passes have, and no others
}

}  // namespace mcl
