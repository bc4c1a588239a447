// Sweeps of FP32 U(1) and SU(2) links by the site pass and by the group pass, in a build of
// their own: with -fmad=false the compiler contracts nothing, so what it leaves as it is in
// the library is what the source fixes.
#include "metropolis_group.cuh"

namespace klft {

template <int NC, int ND>
__global__ void __launch_bounds__(128) site_pass(Links<NC, float> U, Geom g, int val, MetroArgs a, uint32_t sweep) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < g.Vh) site_update_ref<NC, ND, float, false>(U, g, pass_site(g, t, val, ND), a, sweep, Defect{});
}

template <int NC, int ND>
__global__ void __launch_bounds__(GROUP_THREADS) group_pass(Links<NC, float> U, Geom g, int val, MetroArgs a, uint32_t sweep) {
  __shared__ GroupShared<NC, ND, float, 8> sh[GROUP_THREADS / 8];
  const long long t = ((long long)blockIdx.x * GROUP_THREADS + threadIdx.x) / 8;
  group_site_update<NC, ND, float, false, 8>(sh, U, g, t, val, a, sweep, Defect{});
}

template <int NC, int ND> cudaError_t sweeps(const int *L, float *host, const MetroArgs &a, int n, bool group) {
  Geom g{};
  g.nd = ND;
  g.V = g.Vh = 1;
  g.open_mu = -1;
  int stride = 1;
  for (int d = 0; d < 4; ++d) {
    g.L[d] = d < ND ? L[d] : 1;
    g.H[d] = d < ND ? L[d] / 2 : 1;
    g.hs[d] = stride;
    stride *= g.H[d];
    g.Vh *= g.H[d];
    if (d < ND) g.V *= L[d];
  }
  const size_t bytes = (size_t)g.V * ND * NC * sizeof(cx<float>);
  cx<float> *p = nullptr;
  cudaError_t e = cudaMalloc(&p, bytes);
  if (e != cudaSuccess) return e;
  e = cudaMemcpy(p, host, bytes, cudaMemcpyHostToDevice);
  const Links<NC, float> U{p, g.V};
  for (int k = 0; k < n && e == cudaSuccess; ++k)
    for (int val = 0; val < 1 << ND; ++val) {
      if (group) group_pass<NC, ND><<<(unsigned)group_blocks(g.Vh, 8), GROUP_THREADS>>>(U, g, val, a, (uint32_t)k);
      else site_pass<NC, ND><<<(unsigned)((g.Vh + 127) / 128), 128>>>(U, g, val, a, (uint32_t)k);
    }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(host, p, bytes, cudaMemcpyDeviceToHost);
  cudaFree(p);
  return e;
}

}  // namespace klft

// links: [mu][row-0 entry][class][half site] complex, updated in place
extern "C" int pinned_sweeps(int nc, const int *L, float *links, double beta, double delta, int nhits, int nsweeps,
                             unsigned long long seed, unsigned long long chain, int group) {
  const klft::MetroArgs a{beta, delta, 0.0, nhits, 0, seed, chain};
  return (int)(nc == 1 ? klft::sweeps<1, 3>(L, links, a, nsweeps, group) : klft::sweeps<2, 4>(L, links, a, nsweeps, group));
}
