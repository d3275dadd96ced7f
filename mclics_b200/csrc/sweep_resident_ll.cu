// Resident-sweep kernels of one potential (instantiations split across files so they compile in parallel).
#include "sweep_resident.cuh"

namespace mcl {

cudaError_t launch_resident_ll(const ModelDev &m, const ResidentArgs &a, const ResidentLaunch &l) {
  if (l.flip == false && l.field == false) return launch_resident_gp<POT_LL, false, false, false>(m, a, l);
  if (l.flip == false && l.field == true) return launch_resident_gp<POT_LL, false, false, true>(m, a, l);
  if (l.flip == true && l.field == true) return launch_resident_gp<POT_LL, true, false, true>(m, a, l);
  return cudaErrorInvalidValue;  // the combinations the colour passes have, and no others
}

}  // namespace mcl
