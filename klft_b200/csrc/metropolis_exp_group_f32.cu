// metropolis_exp_group_f32.cu -- the FP32 instances of the exp group kernels (metropolis_exp_group.cuh).
#include "metropolis_exp_group.cuh"

namespace klft {

cudaError_t launch_exp_group_f32(int nd, int G, bool defect, const GroupLaunch &l) {
  return launch_exp_group_t<float>(nd, G, defect, l);
}

}  // namespace klft
