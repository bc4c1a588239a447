// metropolis_group_u1.cu -- the U(1) instances of the group kernels (metropolis_group.cuh).
#include "metropolis_group.cuh"

namespace klft {

cudaError_t launch_group_u1(int nd, int dtype, int G, bool defect, const GroupLaunch &l) {
  return launch_group_nc<1>(nd, dtype, G, defect, l);
}

}  // namespace klft
