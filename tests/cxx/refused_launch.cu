// A launch with more threads than a block can have is refused by the runtime; launch_after
// reports it once, and the launch after it is an ordinary one.
#include <cstdio>

#include "pdl.cuh"

__global__ void set_one(int *p) { *p = 1; }

int main() {
  int *p = nullptr, v = 0;
  if (cudaMalloc(&p, sizeof(int)) != cudaSuccess) return 2;
  for (bool dependent : {false, true}) {
    const cudaError_t refused = klft::launch_after(dependent, set_one, dim3(1), dim3(4096), 0, nullptr, p);
    const cudaError_t after = cudaGetLastError();
    std::printf("%d %d\n", (int)refused, (int)after);
    if (refused == cudaSuccess || after != cudaSuccess) return 1;
  }
  if (klft::launch_after(false, set_one, dim3(1), dim3(1), 0, nullptr, p) != cudaSuccess) return 3;
  if (cudaMemcpy(&v, p, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return 4;
  return v == 1 ? 0 : 5;
}
