// metropolis_group_su3.cu -- the SU(3) instances of the group kernels (metropolis_group.cuh).
#include "metropolis_group.cuh"

namespace klft {

cudaError_t launch_group_su3(int nd, int dtype, int G, bool defect, const GroupLaunch &l) {
  return launch_group_nc<3>(nd, dtype, G, defect, l);
}

}  // namespace klft
