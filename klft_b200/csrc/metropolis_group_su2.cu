// metropolis_group_su2.cu -- the SU(2) instances of the group kernels (metropolis_group.cuh).
#include "metropolis_group.cuh"

namespace klft {

cudaError_t launch_group_su2(int nd, int dtype, int G, bool defect, const GroupLaunch &l) {
  return launch_group_nc<2>(nd, dtype, G, defect, l);
}

}  // namespace klft
