// Colour-pass kernels of one potential with one set of options, 24 of them. Compiled once per set (build.py): the
// compiler's time grows faster than the number of kernels in a file (the chiral GHRL ones: 689 s in one file, 39, 45 and
// 79 s in three).
#include "sweep_pass.cuh"

namespace mcl {

template cudaError_t launch_pass_gp<PASS_POT, PASS_FLIP, PASS_CHIRAL, PASS_FIELD>(const ModelDev &, const FusedArgs &,
                                                                                  const FusedLaunch &);

}  // namespace mcl
