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
#include <math.h>

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
// The hits of a site enter where their places outgrow its window of the stream, and where
// few of them leave the second wave of SU(2) FP64's CTAs nothing to hide.  us per sweep
// over one thread's, 4-D, by nHits:
//   U(1) FP32   7168 sites   13: 0.44 (4 lanes) 0.49 (8)   20: 0.89 0.75   30: 1.19 0.86   60: 1.51 1.05
//              12,800 sites  13: 0.59 0.83   20: 1.06 1.18
//   U(1) FP64   4608 sites   20: 0.59 (16) 0.61 (8)   60: 0.69 0.85   300: 0.70 0.85
//               7168 sites   20: 0.99 0.74   60: 1.07 1.04   300: 1.08 1.08
//   SU(2) FP32  3136 sites   30: 0.84 (8)   60: 0.95   300: 1.02;   4608 sites  0.97 1.09 1.20
//   SU(2) FP64  4096 sites    1: 1.44 (16)   4: 1.14   10: 0.91   13: 0.94   30: 1.04
// Waves: 3552 sites of SU(2) FP64 with 16 lanes, 7104 of SU(2) FP32 with 8.
static int group_lanes12(int nc, bool f64, const PassWork &w) {
  const long long sites = w.sites;
  const long long hits = (long long)w.nd * w.nhits_max;  // of a site
  if (nc == 2 && f64) {
    if (sites <= 1000) return 32;
    return sites <= 3552 || (sites <= 5500 && w.nhits_min >= 8 && w.nhits_max <= 13) ? 16 : 1;
  }
  if (nc == 2) return sites <= (hits <= 150 ? 7104 : 3200) ? 8 : 1;
  if (f64) {
    if (sites <= 1300) return 32;
    if (hits > 130) return sites <= 5900 ? 16 : 1;
    return sites <= 2500 ? 16 : (sites <= 9000 ? 8 : 1);
  }
  if (hits <= 60) return sites <= 6000 ? 8 : (sites <= 16000 ? 4 : 1);
  return sites <= (hits <= 130 ? 9300 : 5500) ? 8 : 1;
}

// SU(3): a hit that lowers the action ends the chunk of proposals, so the groups win by
// the rejected hits, and how many there are follows beta.  x = beta sqrt(2 (Nd - 1)), a
// link's coupling to the sum of its staples when these are in no order, says where:
// about 0.85 of the hits accepted at x = 1.2, 0.43 at 5, 0.23 at 7, 0.12 at 10, 0.05 at
// 12, below 0.03 from 14 on.  us per sweep over one thread's, 4-D, nHits 10 (one thread:
// FP64 1970-2010, 1700 at x = 14.7; FP32 1610-1650, 1500), equilibrium:
//   sites  lanes   x = 1.2   4.9   7.3   9.8   12.2  14.0  14.7
//   576    32 FP64    0.76  0.62  0.51  0.41  0.33  0.36  0.32   FP32 0.57 ..  0.22
//   1152   32 FP64    0.94  0.73  0.60  0.48  0.39  0.44  0.40   FP32 0.86 ..  0.29
//   1152   8  FP64    1.00  0.85  0.72  0.60  0.49  0.56  0.57   FP32 0.85 ..  0.42
//   2304   8  FP64    1.01  0.87  0.75  0.62  0.51  0.58  0.60   FP32 0.86 ..  0.43
//   4608   8  FP64    1.27  1.07  0.91  0.75  0.63  0.70  0.60
//   4608   8  FP32    1.28  1.03  0.86  0.71  0.59  0.57  0.46
//   6656   8  FP64    2.36  1.90  1.54  1.23  0.98  0.95  0.81
//   6656   8  FP32    1.31  1.06  0.89  0.74  0.62  0.54  0.44
//   8192   8  FP64    2.47  1.98  1.63  1.32  1.06  1.02  0.87
//   8192   8  FP32    2.24  1.74  1.39  1.12  0.92  0.78  0.66
// The steps are waves of CTAs: FP64 2368, 4736 sites at two and four CTAs per SM (592,
// 1184 with 32 lanes), FP32 three and six (4736 in 2-D and 3-D).  Past the first full
// wave one hit a link is too few (FP64 6656 sites, nHits 1: 1.10 at x = 14.7).
static int group_lanes3(bool f64, const PassWork &w) {
  const long long sites = w.sites;
  const double x = w.beta_min * sqrt(2.0 * (w.nd - 1));
  const bool second = w.nhits_min >= 8;  // enough hits for a second wave
  if (f64) {
    if (sites <= 592 || (sites <= 1184 && x >= 3.0) || (sites <= 1500 && x >= 12.0)) return 32;
    const long long most = x >= 14.0 && second ? 8200 : (x >= 12.0 && second ? 6700 : (x >= 7.3 ? 4736 : (x >= 4.5 ? 2368 : 0)));
    return sites <= most ? 8 : 1;
  }
  if (sites <= 1184 || (sites <= 1500 && x >= 3.0)) return 32;
  const long long most = x >= 14.0 && second ? 12000
                         : x >= 12.0 && second ? 8200
                         : x >= 12.0 || (w.nd == 4 && x >= 7.0) ? 7104
                         : x >= 7.0 ? 4736
                         : x >= 4.5 ? 3552 : 2368;
  return sites <= most ? 8 : 1;
}

int group_lanes(int nc, int dtype, bool defect, const PassWork &w) {
  if (nc == 3) return group_lanes3(dtype == 0, w);
  if (defect && dtype == 1) return 1;  // no FP32 form for U(1), SU(2) with a defect
  return group_lanes12(nc, dtype == 0, w);
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

int pass_lanes(int nc, int dtype, const MetroArgs &a, bool defect, const Geom &g) {
  if (nc == 3 && a.proposal == PROPOSAL_EXP) return exp_group_lanes(dtype, defect, g.V / 2);
  PassWork w;
  w.add(g, a);
  return group_lanes(nc, dtype, defect, w);
}

cudaError_t launch_metropolis_pass(int nc, int dtype, void *links, const Geom &g, int val, const MetroArgs &a,
                                   const uint32_t *d_sweep, unsigned long long *d_nacc, const Defect &df, int block,
                                   cudaStream_t st) {
  const bool exp = nc == 3 && a.proposal == PROPOSAL_EXP;
  const int lanes = pass_lanes(nc, dtype, a, df.active != 0, g);
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
