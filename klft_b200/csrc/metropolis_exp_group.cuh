// metropolis_exp_group.cuh -- the SU(3) exp(i eps H) link update by a group of G
// lanes, for link passes with too few links to fill the device with one thread each.
//
// link_update_exp runs a link's staple and its hits in one thread: 15 us a pass
// whatever the size up to some 10^4 links.  The proposals sit at fixed places of the
// stream, so here each lane forms one of them (and its accept uniform) before the
// wait for the pass before (programmatic dependent launch), the staple's terms are
// shared out as well, and only the chain of accepted products is left to every lane:
// a pass of 8^4 takes 10 us in FP32 (134 -> 78 us per sweep).
// Operations on a link and their order are those of link_update_exp; so is the chain.
#pragma once
#include "chains.cuh"
#include "metropolis_site.cuh"
#include "pdl.cuh"

namespace klft {

template <int ND, typename T, int G> struct ExpGroupShared {
  static constexpr int NTERM = 2 * (ND - 1);
  Mat<3, T> X[G];         // the proposals of a chunk of G hits
  Mat<3, T> term[NTERM];  // the staple's terms: forward, then backward
  double u[G];            // accept uniforms
  float lg[G];            // their logarithms
};

// Term q of the staple of U_mu(x), as staple_su3_2row_ct (FP32, no defect) or
// staple_ct (FP64) form it.
template <int ND, typename T, bool DF>
KLFT_D Mat<3, T> staple_term(const Links<3, T> &U, const Geom &g, const Site &x, int mu, int q, const Defect &df) {
  const bool fwd = q < ND - 1;
  int nu = fwd ? q : q - (ND - 1);
  nu += nu >= mu;
  const Site xpmu = site_up(g, x, mu);
  Mat<3, T> f;
  if constexpr (!DF && sizeof(T) == 4) {
    Mat<3, T> t;
    if (fwd) {
      mul_rows01(U.load_rows01(site_lin(g, x), nu), U.load(site_lin(g, site_up(g, x, nu)), mu), t);
      complete_row2(t);
      mul_nd_rows01(U.load_rows01(site_lin(g, xpmu), nu), t, f);
    } else {
      const long long ln = site_lin(g, site_dn(g, x, nu));
      mul_rows01(U.load_rows01(ln, mu), U.load(site_lin(g, site_dn(g, xpmu, nu)), nu), t);
      complete_row2(t);
      mul_dn_rows01(t, U.load(ln, nu), f);
    }
    complete_row2(f);
  } else if (fwd) {
    const Mat<3, T> t = mul_nd(load_link<3, T, DF>(U, g, xpmu, nu, df),
                               load_link<3, T, DF>(U, g, site_up(g, x, nu), mu, df));
    f = mul_nd(t, load_link<3, T, DF>(U, g, x, nu, df));
  } else {
    const Site xmnu = site_dn(g, x, nu);
    const Mat<3, T> t = mul_dd(load_link<3, T, DF>(U, g, site_dn(g, xpmu, nu), nu, df),
                               load_link<3, T, DF>(U, g, xmnu, mu, df));
    f = mul(t, load_link<3, T, DF>(U, g, xmnu, nu, df));
  }
  return f;
}

// Link pass val = 2 mu + p: the t-th link by the calling thread's group.  Every
// thread of the CTA calls it and passes the wait.  Accepted hits, in one lane.
template <int ND, typename T, bool DF, int G>
KLFT_D int exp_group_update(ExpGroupShared<ND, T, G> *shared, const Links<3, T> &U, const Geom &g, long long t, int val,
                            const MetroArgs &a, uint32_t sweep, const Defect &df) {
  ExpGroupShared<ND, T, G> &sh = shared[threadIdx.x / G];
  const int mu = val >> 1, gl = (int)(threadIdx.x & (unsigned)(G - 1));
  const unsigned mask = G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << (threadIdx.x & 31u & ~(unsigned)(G - 1));
  bool ok = false;
  const Site x = link_pass_site(g, t, val & 1, ND, ok);
  ok = ok && t < link_pass_threads(g, ND) && !open_link(g, x, mu);
  const ExpHitStream hs{(uint32_t)a.seed, (uint32_t)(a.seed >> 32) ^ (uint32_t)a.chain, site_lex(g, x), sweep, a.bm};
  const T half_eps = (T)(0.5 * a.eps);
  const uint32_t h0 = (uint32_t)(mu * a.nhits);
  auto chunk = [&](int first) {
    if (first + gl < a.nhits) {
      const uint32_t h = h0 + (uint32_t)(first + gl);
      sh.X[gl] = exp_proposal<T>(hs, h, half_eps);
      uint32_t w[4];
      hs.accept_block(h, w);
      const double u = accept_word(w, h);
      sh.u[gl] = u;
      sh.lg[gl] = __logf((float)u);
    }
  };
  if (ok) chunk(0);
  grid_dependency_wait();
  grid_launch_dependents();
  int nacc = 0;
  if (ok) {
    const long long lx = site_lin(g, x);
    const T bnc = (T)a.beta / T(3);
    const T cdef = DF && df.active && in_defect(g, df, x, mu) ? (T)defect_c(df) : T(1);
    const Mat<3, T> U0 = U.load(lx, mu);
    for (int q = gl; q < ExpGroupShared<ND, T, G>::NTERM; q += G) sh.term[q] = staple_term<ND, T, DF>(U, g, x, mu, q, df);
    __syncwarp(mask);
    Mat<3, T> S = mzero<3, T>();
#pragma unroll 1
    for (int q = 0; q < ExpGroupShared<ND, T, G>::NTERM; ++q) madd(S, sh.term[q]);
    const Mat<3, T> M0 = mul(U0, S);
    Mat<3, T> A = mident<3, T>();
    T trO = retr_diag(M0);
#pragma unroll 1
    for (int first = 0; first < a.nhits; first += G) {
      if (first) {
        __syncwarp(mask);
        chunk(first);
        __syncwarp(mask);
      }
      const int n = a.nhits - first < G ? a.nhits - first : G;
#pragma unroll 1
      for (int k = 0; k < n; ++k) {
        const Mat<3, T> Y = first + k == 0 ? sh.X[k] : mul(sh.X[k], A);
        const T tY = retr_mul(Y, M0);
        const T dS = -bnc * (tY - trO) * cdef;
        // u < exp(-dS) from ln u <= 0 in FP32 (absolute error below 2e-5); within 1e-4, and
        // for a NaN, the comparison of exp_hit
        const float d = (float)dS + sh.lg[k];
        bool accept = d < 0.f;
        if (__builtin_expect(!(fabsf(d) > 1e-4f), 0)) accept = dS < T(0) || sh.u[k] < (double)exp(-dS);
        if (accept) {
          A = Y;
          trO = tY;
          ++nacc;
        }
      }
    }
    if (nacc && gl == 0) U.store(lx, mu, restore(mul(A, U0)));
  }
  return gl == 0 ? nacc : 0;
}

template <int ND, typename T, bool DF, int G>
__global__ void __launch_bounds__(GROUP_THREADS)
    exp_group_kernel(Links<3, T> U, Geom g, int val, MetroArgs a, const uint32_t *__restrict__ d_sweep,
                     unsigned long long *__restrict__ d_nacc, Defect df) {
  __shared__ ExpGroupShared<ND, T, G> sh[GROUP_THREADS / G];
  const long long t = ((long long)blockIdx.x * GROUP_THREADS + threadIdx.x) / G;
  add_accepts(exp_group_update<ND, T, DF, G>(sh, U, g, t, val, a, *d_sweep, df), d_nacc);
}

template <int ND, typename T, bool DF, int G>
__global__ void __launch_bounds__(GROUP_THREADS)
    multi_exp_group_kernel(const __grid_constant__ ChainTable tab, int val, unsigned long long *nacc_slots,
                           const uint32_t *__restrict__ slot) {
  __shared__ ExpGroupShared<ND, T, G> sh[GROUP_THREADS / G];
  const ChainDesc &c = tab.c[find_chain(tab)];
  const long long t = ((long long)(blockIdx.x - c.block_begin) * GROUP_THREADS + threadIdx.x) / G;
  const Links<3, T> U{(cx<T> *)c.links, c.g.V};
  add_accepts(exp_group_update<ND, T, DF, G>(sh, U, c.g, t, val, c.a, *c.ctr, c.df),
              nacc_slots + (size_t)(*slot) * tab.nchains_total + c.index);
}

// The passes of a sweep after its first start before the pass before them has ended.
template <int ND, typename T, bool DF, int G> static cudaError_t launch_exp_group_t(const GroupLaunch &l) {
  if (l.tab)
    return launch_after(l.val > 0, multi_exp_group_kernel<ND, T, DF, G>, dim3(l.blocks), dim3(GROUP_THREADS), 0, l.st,
                        *l.tab, l.val, l.nacc, l.slot);
  const Geom &g = *l.g;
  return launch_after(l.val > 0, exp_group_kernel<ND, T, DF, G>,
                      dim3((unsigned)group_blocks(link_pass_threads(g, ND), G)), dim3(GROUP_THREADS), 0, l.st,
                      Links<3, T>{(cx<T> *)l.links, g.V}, g, l.val, *l.a, l.d_sweep, l.nacc, *l.df);
}
template <int ND, typename T> static cudaError_t launch_exp_group_nd(int G, bool defect, const GroupLaunch &l) {
  if constexpr (sizeof(T) == 4) {
    if (defect) return cudaErrorInvalidValue;  // exp_group_lanes gives 1
  } else if (defect)
    return G == 16 ? launch_exp_group_t<ND, T, true, 16>(l) : launch_exp_group_t<ND, T, true, 4>(l);
  return G == 16 ? launch_exp_group_t<ND, T, false, 16>(l) : launch_exp_group_t<ND, T, false, 4>(l);
}
template <typename T> static cudaError_t launch_exp_group_t(int nd, int G, bool defect, const GroupLaunch &l) {
  if (nd == 2) return launch_exp_group_nd<2, T>(G, defect, l);
  if (nd == 3) return launch_exp_group_nd<3, T>(G, defect, l);
  return launch_exp_group_nd<4, T>(G, defect, l);
}

}  // namespace klft
