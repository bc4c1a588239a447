// chains.cuh -- the chain table of a multi-chain launch (batch.cu).
#pragma once
#include "common.cuh"
#include "kernels.cuh"

namespace klft {

constexpr int BATCH_MAX = 64;

struct ChainDesc {
  void *links;
  uint32_t *ctr;  // the chain's counters ([0] = sweep)
  Geom g;
  MetroArgs a;
  Defect df;
  int index;        // chain id in the batch
  int block_begin;  // first CTA of this chain in the launch
};

struct ChainTable {
  int n;
  int nchains_total;
  int block;  // threads per CTA of the launch (<= 128)
  ChainDesc c[BATCH_MAX];
};

KLFT_D int find_chain(const ChainTable &tab) {
  int lo = 0, hi = tab.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tab.c[mid].block_begin <= (int)blockIdx.x) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// One pass by groups of lanes, of one lattice or of many chains.
struct GroupLaunch {
  // one lattice
  void *links = nullptr;
  const Geom *g = nullptr;
  const MetroArgs *a = nullptr;
  const Defect *df = nullptr;
  const uint32_t *d_sweep = nullptr;
  // many chains
  const ChainTable *tab = nullptr;
  int blocks = 0;
  const uint32_t *slot = nullptr;
  int val = 0;
  unsigned long long *nacc = nullptr;
  cudaStream_t st = nullptr;
};
cudaError_t launch_exp_group_f32(int nd, int G, bool defect, const GroupLaunch &l);
cudaError_t launch_exp_group_f64(int nd, int G, bool defect, const GroupLaunch &l);

}  // namespace klft
