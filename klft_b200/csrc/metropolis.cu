// metropolis.cu -- one pass of the Metropolis sweep on one lattice.
//
// Reference proposals: sweep_Metropolis (Metropolis.hpp:118-178) visits the
// 2^Nd parity classes in the reference's order (class val has parity bit
// (val >> (Nd-1-d)) & 1 in dimension d, IndexHelper.hpp:84-93); the host
// enqueues one launch per class.  Sites of one class share no staple link, so
// a pass is race free.  exp(i eps H) proposals: 2 Nd link passes (mu, parity)
// of one thread per link (metropolis_site.cuh).  The per-site and per-link
// updates are in metropolis_site.cuh.  Passes too small to fill the device so go
// to groups of lanes (metropolis_group.cuh, metropolis_exp_group.cuh).
#include "metropolis_group.cuh"

namespace klft {

template <int NC, int ND, typename T, bool DF>
__global__ void __launch_bounds__(128, MinBlocks<T>::v)
    metropolis_ref_kernel(Links<NC, T> U, Geom g, int val, MetroArgs a, const uint32_t *__restrict__ d_sweep,
                          unsigned long long *__restrict__ d_nacc, Defect df) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int nacc = 0;
  if (t < g.Vh) nacc = site_update_ref<NC, ND, T, DF>(U, g, pass_site(g, t, val, ND), a, *d_sweep, df);
  add_accepts(nacc, d_nacc);
}

// link pass val = 2 MU + p: U_MU(x) of the V/2 sites of parity p (one
// instance per direction, so the staple's site steps are compiled)
template <int ND, typename T, bool DF, int MU>
__global__ void __launch_bounds__(128, MinBlocks<T>::v)
    metropolis_exp_kernel(Links<3, T> U, Geom g, int val, MetroArgs a, const uint32_t *__restrict__ d_sweep,
                          unsigned long long *__restrict__ d_nacc, Defect df) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int nacc = 0;
  bool ok = false;
  const Site x = link_pass_site(g, t, val & 1, ND, ok);
  if (ok && t < link_pass_threads(g, ND)) nacc = link_update_exp<ND, T, DF, MU>(U, g, x, MU, a, *d_sweep, df);
  add_accepts(nacc, d_nacc);
}

template <int NC, int ND, typename T, bool DF>
static cudaError_t launch_tdf(const Links<NC, T> &U, const Geom &g, int val, const MetroArgs &a,
                              const uint32_t *d_sweep, unsigned long long *d_nacc, const Defect &df, int block,
                              cudaStream_t st) {
  const unsigned grid = (unsigned)((g.Vh + block - 1) / block);
  if constexpr (NC == 3) {
    if (a.proposal == PROPOSAL_EXP) {
      const unsigned lgrid = (unsigned)((link_pass_threads(g, ND) + block - 1) / block);
      switch (val >> 1) {
        case 0: metropolis_exp_kernel<ND, T, DF, 0><<<lgrid, block, 0, st>>>(U, g, val, a, d_sweep, d_nacc, df); break;
        case 1: metropolis_exp_kernel<ND, T, DF, 1><<<lgrid, block, 0, st>>>(U, g, val, a, d_sweep, d_nacc, df); break;
        case 2:
          if constexpr (ND > 2)
            metropolis_exp_kernel<ND, T, DF, (ND > 2 ? 2 : 0)><<<lgrid, block, 0, st>>>(U, g, val, a, d_sweep, d_nacc,
                                                                                       df);
          break;
        default:
          if constexpr (ND > 3)
            metropolis_exp_kernel<ND, T, DF, (ND > 3 ? 3 : 0)><<<lgrid, block, 0, st>>>(U, g, val, a, d_sweep, d_nacc,
                                                                                       df);
          break;
      }
      return cudaGetLastError();
    }
  }
  metropolis_ref_kernel<NC, ND, T, DF><<<grid, block, 0, st>>>(U, g, val, a, d_sweep, d_nacc, df);
  return cudaGetLastError();
}

template <int NC, int ND, typename T>
static cudaError_t launch_t(void *links, const Geom &g, int val, const MetroArgs &a, const uint32_t *d_sweep,
                            unsigned long long *d_nacc, const Defect &df, int block, cudaStream_t st) {
  Links<NC, T> U{(cx<T> *)links, g.V};
  if (block != 32 && block != 64 && block != 128) block = 128;  // the kernels are built for <= 128 threads
  if (df.active) return launch_tdf<NC, ND, T, true>(U, g, val, a, d_sweep, d_nacc, df, block, st);
  return launch_tdf<NC, ND, T, false>(U, g, val, a, d_sweep, d_nacc, df, block, st);
}

template <int NC, typename T>
static cudaError_t launch_nd(int nd, void *links, const Geom &g, int val, const MetroArgs &a,
                             const uint32_t *d_sweep, unsigned long long *d_nacc, const Defect &df, int block,
                             cudaStream_t st) {
  switch (nd) {
    case 2: return launch_t<NC, 2, T>(links, g, val, a, d_sweep, d_nacc, df, block, st);
    case 3: return launch_t<NC, 3, T>(links, g, val, a, d_sweep, d_nacc, df, block, st);
    case 4: return launch_t<NC, 4, T>(links, g, val, a, d_sweep, d_nacc, df, block, st);
  }
  return cudaErrorInvalidValue;
}

// More lanes shorten a site's chain of proposals but repeat its serial part in every
// lane and form proposals that are not used, so fewer lanes pay as the sites fill
// the device, and one thread per site once they do.  us per sweep (4-D, nHits 10) by
// lanes, at 256, 1200, 2058, 4096, 8192 and 20736 sites a pass (V / 16):
//   U(1) FP64   1: 511 527 529 530 529 561    32: 165 194 243 414 714 1780
//               16: 190 202 206 281 505 1094   8: 212 216 220 237 319 868
//   U(1) FP32   1: 464 480 476 470 480 528     8: 141 145 147 161 252 549
//               4: 183 184 186 195 226 520
//   SU(2) FP64  1: 824 842 857 842 836 981    32: 218 376 390 752 1469 3620
//               16: 255 309 392 776 1228 2759
//   SU(2) FP32  1: 505 529 530 530 529 617     8: 180 192 194 283 543 1036
//               16: 177 192 206 318 603 1514
// and SU(3) at 256, 1200, 4096, 8192, 20736 (at the chain's own acceptance of 1 %; a
// cold start, which accepts nothing, takes half as long):
//   SU(3) FP64  1: 1611 1656 1685 1733 2232   32: 443 644 1627 3016 7295
//                8: 706 764 989 1697 3883
//   SU(3) FP32  1: 1486 1502 1517 1527 1855   32: 322 456 1038 1992 5099
//                8: 536 572 781 1224 2402
int group_lanes(int nc, int dtype, bool defect, long long sites) {
  const bool f64 = dtype == 0;
  if (nc == 3) return sites <= 1500 ? 32 : (sites <= (f64 ? 8200 : 12000) ? 8 : 1);
  if (defect && !f64) return 1;  // no FP32 form for U(1), SU(2) with a defect
  if (nc == 2) return f64 ? (sites <= 1000 ? 32 : (sites <= 5500 ? 16 : 1)) : (sites <= 7500 ? 8 : 1);
  if (f64) return sites <= 1300 ? 32 : (sites <= 2500 ? 16 : (sites <= 9000 ? 8 : 1));
  return sites <= 6000 ? 8 : (sites <= 16000 ? 4 : 1);
}

// The chain of a link's accepted products is repeated in every lane, so groups pay
// while the links leave the device idle.  us per sweep (4-D, nHits 10) by lanes, at
// 128, 2048, 3200, 4800 and 9600 links a pass (V / 2):
//   FP64  1: 169 184 185 184 185   4: 106 109 119 131 220   16: 78 106 183 252 424
//   FP32  1: 132 134 133 132 134   4:  90  93 102 108 166   16: 63  78 103 163 253
// (3-D, 840 links: FP64 127, 73, 66; FP32 91, 60, 52.)  FP32 links with a defect keep
// one thread: their staple's contraction, and with it the chain's bits, differ here.
int exp_group_lanes(int dtype, bool defect, long long links) {
  if (defect && dtype == 1) return 1;
  return links <= 2500 ? 16 : (links <= 6500 ? 4 : 1);
}

int pass_lanes(int nc, int dtype, int proposal, bool defect, const Geom &g) {
  if (nc == 3 && proposal == PROPOSAL_EXP) return exp_group_lanes(dtype, defect, g.V / 2);
  return group_lanes(nc, dtype, defect, g.Vh);
}

cudaError_t launch_metropolis_pass(int nc, int dtype, void *links, const Geom &g, int val, const MetroArgs &a,
                                   const uint32_t *d_sweep, unsigned long long *d_nacc, const Defect &df, int block,
                                   cudaStream_t st) {
  const bool exp = nc == 3 && a.proposal == PROPOSAL_EXP;
  const int lanes = pass_lanes(nc, dtype, a.proposal, df.active != 0, g);
  if (lanes > 1) {
    MetroArgs b = a;
    // the FP64 exp(i eps H) proposal reads its Gaussians from the host-built table
    if (exp && dtype == 0 && !(b.bm = bm_table())) return cudaErrorMemoryAllocation;
    GroupLaunch l;
    l.links = links;
    l.g = &g;
    l.a = &b;
    l.df = &df;
    l.d_sweep = d_sweep;
    l.val = val;
    l.nacc = d_nacc;
    l.st = st;
    if (exp) return dtype == 0 ? launch_exp_group_f64(g.nd, lanes, df.active != 0, l) : launch_exp_group_f32(g.nd, lanes, df.active != 0, l);
    if (nc == 1) return launch_group_u1(g.nd, dtype, lanes, df.active != 0, l);
    if (nc == 2) return launch_group_su2(g.nd, dtype, lanes, df.active != 0, l);
    return launch_group_su3(g.nd, dtype, lanes, df.active != 0, l);
  }
  if (dtype == 0) {
    if (nc == 3 && a.proposal == 1) {
      // the FP64 exp(i eps H) proposal reads its Gaussians from the host-built table
      MetroArgs b = a;
      if (!(b.bm = bm_table())) return cudaErrorMemoryAllocation;
      return launch_nd<3, double>(g.nd, links, g, val, b, d_sweep, d_nacc, df, block, st);
    }
    switch (nc) {
      case 1: return launch_nd<1, double>(g.nd, links, g, val, a, d_sweep, d_nacc, df, block, st);
      case 2: return launch_nd<2, double>(g.nd, links, g, val, a, d_sweep, d_nacc, df, block, st);
      case 3: return launch_nd<3, double>(g.nd, links, g, val, a, d_sweep, d_nacc, df, block, st);
    }
  } else {
    switch (nc) {
      case 1: return launch_nd<1, float>(g.nd, links, g, val, a, d_sweep, d_nacc, df, block, st);
      case 2: return launch_nd<2, float>(g.nd, links, g, val, a, d_sweep, d_nacc, df, block, st);
      case 3: return launch_nd<3, float>(g.nd, links, g, val, a, d_sweep, d_nacc, df, block, st);
    }
  }
  return cudaErrorInvalidValue;
}

__global__ void advance_kernel(uint32_t *c) { c[0] += 1u; }

cudaError_t launch_advance(uint32_t *d_counter, cudaStream_t st) {
  advance_kernel<<<1, 1, 0, st>>>(d_counter);
  return cudaGetLastError();
}

}  // namespace klft
