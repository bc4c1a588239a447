// metropolis_exp_group_f64.cu -- the FP64 instances of the exp group kernels (metropolis_exp_group.cuh).
#include "metropolis_exp_group.cuh"

namespace klft {

cudaError_t launch_exp_group_f64(int nd, int G, bool defect, const GroupLaunch &l) {
  return launch_exp_group_t<double>(nd, G, defect, l);
}

}  // namespace klft
