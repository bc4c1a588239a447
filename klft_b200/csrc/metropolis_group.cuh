// metropolis_group.cuh -- the reference-proposal update of one site by a group of
// G lanes, for passes with too few sites to fill the device with one thread each.
//
// site_update_ref runs a site's Nd links and their hits one after another in one
// thread: Nd * nhits proposals (Philox rounds, sine and cosine, norms), each on
// the chain of the one before, and Nd staples whose loads wait for each other.  A
// class of 8^4 has 256 sites, so that chain is the whole pass.  Only two things
// in it are sequential: the accept decisions and the place in the site's stream
// they leave it at.  The lanes of a group share the rest:
//
//  * U(1), SU(2): the lanes form the uniforms of a window of the stream and the
//    proposal that would start at each place in it; a hit then takes the one at
//    its place.  Most are not used (a hit moves on by 1-2 or 3-4 places).  In
//    FP64 the staples' products are shared out as for SU(3) (group_hits); in FP32
//    the links around the site are brought into L1 by all lanes at once, then
//    every lane forms the staples (group_link_f32).  Every lane runs the hits.
//  * SU(3), where a few per cent of the hits are accepted: lane j forms the
//    proposal and the action change of the j-th hit from here, as if every hit
//    before it were rejected with its uniform drawn; the group keeps the hits
//    before the first exception, applies that one and goes on from there.  The
//    products of neighbour links in the staples of all directions are shared out
//    as well (StapleParts in FP64, StapleTerms in FP32): links of one class are
//    not neighbours, so only U_nu(x) itself changes while the site is updated.
//
// None of the proposals read links, so the first ones come before the wait for
// the pass before (programmatic dependent launch).  Operations on a link and
// their order are those of site_update_ref; the chain is the same.
#pragma once
#include "chains.cuh"
#include "metropolis_site.cuh"
#include "pdl.cuh"

namespace klft {

template <int G> KLFT_D unsigned group_mask() {
  if constexpr (G == 32) return 0xffffffffu;
  else return ((1u << G) - 1u) << (threadIdx.x & 31u & ~(unsigned)(G - 1));
}

// ------------------------------------------------------------------ U(1), SU(2)
// Window of stream places in shared memory, per group.
template <int NC, typename T, int G> struct DrawTable {
  static constexpr int K = RefDraws<NC>::n;
  // 40 hits move on by 40-80 or 120-160 places: one window, or two, holds a site's
  static constexpr int W = NC == 1 ? 96 : 160;
  static constexpr int N = W + K + 2;  // a hit looks up to K + 1 places past its own
  cx<T> prop[N][NC];  // row 0 of the proposal starting at each place
  double u[N];
  float lg[N];  // ln u (NaN for u = 0)
};

// HitDraws for a group: the same uniforms and proposals, from the group's table.
template <int NC, typename T, int G> struct TableDraws {
  using Table = DrawTable<NC, T, G>;
  static constexpr int K = Table::K;
  Table &tab;
  const SiteStream st;
  const double delta;
  long long left;       // hits that may still come
  const int gl;         // lane in the group
  const unsigned mask;  // the group's lanes
  int wn = 0, i = 0;    // window: places [base, base + wn) of the stream; the next hit's place
  uint32_t base = 0;
  cx<T> r[NC], ra[NC], rb[NC];  // row 0 of this hit's proposal, of the two that can come next
  float lg = 0.f, la = 0.f, lb = 0.f;

  KLFT_D TableDraws(Table &t, const SiteStream &s, double delta_, long long hits)
      : tab(t), st(s), delta(delta_), left(hits), gl((int)(threadIdx.x & (unsigned)(G - 1))), mask(group_mask<G>()) {}

  // the window from the next hit's place on
  KLFT_D void fill() {
    __syncwarp(mask);
    const uint32_t pos = base + (uint32_t)i;
    base = pos & ~1u;
    i = (int)(pos & 1u);
    const long long need = (left * (K + 1) + i + 1) & ~1ll;
    wn = need < Table::W ? (int)need : Table::W;
    for (int b = gl; 2 * b < wn; b += G) {
      double u0, u1;
      st.block((base >> 1) + (uint32_t)b, u0, u1);
      tab.u[2 * b] = u0;
      tab.u[2 * b + 1] = u1;
      tab.lg[2 * b] = u0 > 0.0 ? __logf((float)u0) : __int_as_float(0x7fc00000);
      tab.lg[2 * b + 1] = u1 > 0.0 ? __logf((float)u1) : __int_as_float(0x7fc00000);
    }
    __syncwarp(mask);
    for (int p = gl; p + K < wn; p += G) {
      const Mat<NC, T> m = propose<T>(&tab.u[p], delta, (const Mat<NC, T> *)nullptr);
#pragma unroll
      for (int j = 0; j < NC; ++j) tab.prop[p][j] = m.e[0][j];
    }
    __syncwarp(mask);
  }

  // the number of hits, up to `hits` (>= 1), that the window surely holds
  KLFT_D int ready(int hits) {
    if (i + K >= wn) fill();
    const int sure = (wn - i) / (K + 1);
    const int m = hits < sure ? hits : (sure > 1 ? sure : 1);
    left -= m;
#pragma unroll
    for (int j = 0; j < NC; ++j) r[j] = tab.prop[i][j];
    lg = tab.lg[i + K];
    return m;
  }
  KLFT_D Mat<NC, T> propose_next() {
    // both places the next hit can be at, loaded beside this hit's arithmetic
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      ra[j] = tab.prop[i + K][j];
      rb[j] = tab.prop[i + K + 1][j];
    }
    la = tab.lg[i + 2 * K];
    lb = tab.lg[i + 2 * K + 1];
    Mat<NC, T> m;
#pragma unroll
    for (int j = 0; j < NC; ++j) m.e[0][j] = r[j];
    if constexpr (NC == 2) su2_row1(m);
    return m;
  }
  // u < exp(-dS) from ln u <= 0 in FP32 (absolute error below 2e-5); within 1e-4, and
  // for u = 0 or a NaN, the accurate comparison of accept_uniform
  KLFT_D bool accept(T dS) const {
    const float t = (float)dS + lg;
    if (__builtin_expect(!(fabsf(t) > 1e-4f), 0)) return dS < T(0) || tab.u[i + K] < (double)exp(-dS);
    return t < 0.f;
  }
  KLFT_D void advance(bool drawn) {
    i += drawn ? K + 1 : K;
#pragma unroll
    for (int j = 0; j < NC; ++j) r[j] = drawn ? rb[j] : ra[j];
    lg = drawn ? lb : la;
  }
};

// One lane's share of the links that the staples of site x read, into L1.
template <int NC, int ND, typename T, int G>
KLFT_D void touch_neighbours(const Links<NC, T> &U, const Geom &g, const Site &x, int gl) {
  // q = (mu, nu): U_mu(x-nu) always, U_nu(x+mu) and U_nu(x+mu-nu) for nu != mu
  for (int q = gl; q < ND * ND; q += G) {
    const int mu = q / ND, nu = q - mu * ND;
    const Site xp = site_up(g, x, mu);
    const long long lin[3] = {site_lin(g, site_dn(g, x, nu)), site_lin(g, xp), site_lin(g, site_dn(g, xp, nu))};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (k > 0 && mu == nu) break;
      const cx<T> *p = U.p + (long long)(k == 0 ? mu : nu) * Links<NC, T>::P * U.V + lin[k];
#pragma unroll
      for (int c = 0; c < Links<NC, T>::P; ++c) {
        float d;  // the value is not used: nothing waits for the load
        asm volatile("ld.global.ca.f32 %0, [%1];" : "=f"(d) : "l"(p + c * U.V) : "memory");
      }
    }
  }
}

// ------------------------------------------------------------------ U(1), SU(2) in FP64
// The hits of a link with staple S, as in link_update_ref; Uo: the link, updated when
// any is accepted.
template <int NC, typename Draws>
KLFT_D int group_hits(const Mat<NC, double> &S, Mat<NC, double> &Uo, const MetroArgs &a, bool dlink, const Defect &df,
                      Draws &rng, double bnc) {
  const Mat<NC, double> U0 = Uo, M0 = mul(S, U0);
  const double cdef = dlink ? defect_c(df) : 1.0;
  Mat<NC, double> A = mident<NC, double>();
  double trO = retr_diag(M0);
  int nacc = 0;
#pragma unroll 1
  for (int hit = 0; hit < a.nhits;) {
    const int m = rng.ready(a.nhits - hit);
    hit += m;
#pragma unroll 1
    for (int k = 0; k < m; ++k) {
      const Mat<NC, double> Y = mul(A, rng.propose_next());
      const double tY = retr_mul(Y, M0);
      const double dS = -bnc * (tY - trO) * cdef;
      const bool accept = rng.accept(dS);  // ln u <= 0: also of dS < 0
      rng.advance(!(dS < 0.0));
      if (accept) {
        A = Y;
        trO = tY;
        ++nacc;
      }
    }
  }
  if (nacc) Uo = restore(mul(U0, A));
  return nacc;
}

// ------------------------------------------------------------------ U(1), SU(2) in FP32
// The hits of link_update_f32 for a group.  Every lane runs them on the link and the
// staple as it loaded them, so lane 0 stores the new link between two barriers: no lane
// then reads it half way, and the next direction's staple sees it.
template <int NC, int ND, int MU, typename Draws>
KLFT_D int group_link_f32(const Links<NC, float> &U, const Geom &g, const Site &x, const MetroArgs &a, Draws &rng) {
  if constexpr (MU < ND) {
    if (open_link(g, x, MU)) return 0;
    const long long lx = site_lin(g, x);
    Hits32<NC> h(staple_f32<NC, ND, MU>(U, g, x), row0(U.load(lx, MU)), (float)a.beta / (float)NC);
#pragma unroll 1
    for (int hit = 0; hit < a.nhits;) {
      const int m = rng.ready(a.nhits - hit);
      hit += m;
#pragma unroll 1
      for (int k = 0; k < m; ++k) {
        const float dS = h.propose(row0(rng.propose_next()));
        const bool accept = rng.accept(dS);  // ln u <= 0: also of dS < 0
        rng.advance(!(dS < 0.f));
        if (accept) h.accept();
      }
    }
    if (h.nacc) {
      const Mat<NC, float> m = h.template link<MU == 0>();
      __syncwarp(rng.mask);
      if (rng.gl == 0) U.store(lx, MU, m);
      __syncwarp(rng.mask);
    }
    return h.nacc;
  }
  return 0;
}

// ------------------------------------------------------------------ staples shared out
// FP64 (every element of a link is stored): the links of a site and the products of its
// neighbours' links, per group.
template <int NC, int ND, typename T> struct StapleParts {
  Mat<NC, T> own[ND];
  // [mu][forward nu, backward nu]: U_nu(x+mu) U_mu(x+nu)^+, the whole backward term
  Mat<NC, T> part[2 * ND * (ND - 1)];

  template <bool DF, int G>
  KLFT_D void load(const Links<NC, T> &U, const Geom &g, const Site &x, long long lx, const Defect &df, int gl) {
    for (int d = gl; d < ND; d += G) own[d] = U.load(lx, d);
    for (int q = gl; q < 2 * ND * (ND - 1); q += G) {
      const int mu = q / (2 * (ND - 1)), r = q - mu * 2 * (ND - 1);  // r: forward, then backward nu
      const bool fwd = r < ND - 1;
      int nu = fwd ? r : r - (ND - 1);
      nu += nu >= mu;
      const Site xpmu = site_up(g, x, mu), xmnu = site_dn(g, x, nu);
      // forward A B^+ = U_nu(x+mu) U_mu(x+nu)^+, backward D^+ E^+ G with
      // D = U_nu(x+mu-nu), E = U_mu(x-nu), G = U_nu(x-nu)
      const Mat<NC, T> a1 = load_link<NC, T, DF>(U, g, fwd ? xpmu : site_dn(g, xpmu, nu), nu, df);
      const Mat<NC, T> a2 = load_link<NC, T, DF>(U, g, fwd ? site_up(g, x, nu) : xmnu, mu, df);
      Mat<NC, T> t = mul_nd(fwd ? a1 : dagger(a1), a2);
      if (!fwd) t = mul(t, load_link<NC, T, DF>(U, g, xmnu, nu, df));
      part[q] = t;
    }
  }

  // staple(): all forward terms, then all backward ones
  template <bool DF> KLFT_D Mat<NC, T> staple(int mu, bool own0_in_defect, const Defect &df) const {
    Mat<NC, T> S = mzero<NC, T>();
    const Mat<NC, T> *p = part + mu * 2 * (ND - 1);
#pragma unroll 1
    for (int k = 0; k < ND - 1; ++k) {
      const int nu = k + (k >= mu);
      Mat<NC, T> c = own[nu];
      if constexpr (DF) {
        if (nu == 0 && own0_in_defect) c = mscale(c, (T)defect_c(df));
      }
      madd(S, mul_nd(p[k], c));
    }
#pragma unroll 1
    for (int k = 0; k < ND - 1; ++k) madd(S, p[ND - 1 + k]);
    return S;
  }
};

// SU(3) in FP32: the same products, each formed as staple() forms it, so that the
// compiler contracts them as it does there (StapleParts gave other last bits: one accept
// decision in 10^7 on disordered links).  The last product of a forward term, which
// reads a link of the site, is one lane's.  With a defect the form of the shared
// products differed once more, so there each lane forms a whole term of one link's
// staple.  us per sweep at nHits 10, beta = 6, without a defect 8^4 210, 16^4 549; with
// whole terms 298, 594; one thread per site 1500 in both.
template <int ND> struct StapleTerms {
  static constexpr int NT = 2 * (ND - 1);  // terms of a link: forward nu, then backward nu
  Mat<3, float> part[ND * NT];             // [mu][term]; with a defect the terms of one link
  Mat<3, float> fwd[ND - 1];

  // first product of forward term r, or all of backward term r
  template <bool DF>
  static KLFT_D Mat<3, float> product(const Links<3, float> &U, const Geom &g, const Site &x, int mu, int r, int nu,
                                      const Defect &df) {
    const Site xpmu = site_up(g, x, mu);
    if (r < ND - 1)
      return mul_nd(load_link<3, float, DF>(U, g, xpmu, nu, df),
                    load_link<3, float, DF>(U, g, site_up(g, x, nu), mu, df));
    const Site xmnu = site_dn(g, x, nu);
    const Mat<3, float> t = mul_dd(load_link<3, float, DF>(U, g, site_dn(g, xpmu, nu), nu, df),
                                   load_link<3, float, DF>(U, g, xmnu, mu, df));
    return mul(t, load_link<3, float, DF>(U, g, xmnu, nu, df));
  }
  static KLFT_D int nu_of(int mu, int r) {
    const int nu = r < ND - 1 ? r : r - (ND - 1);
    return nu + (nu >= mu);
  }

  template <bool DF, int G>
  KLFT_D void load(const Links<3, float> &U, const Geom &g, const Site &x, const Defect &df, int gl) {
    if constexpr (DF) touch_neighbours<3, ND, float, G>(U, g, x, gl);
    else
      for (int q = gl; q < ND * NT; q += G) {
        const int mu = q / NT, r = q - mu * NT;
        part[q] = product<DF>(U, g, x, mu, r, nu_of(mu, r), df);
      }
  }

  template <bool DF, int G>
  KLFT_D Mat<3, float> staple(const Links<3, float> &U, const Geom &g, const Site &x, int mu, const Defect &df, int gl,
                              unsigned mask) {
    const Mat<3, float> *p = part;
    if constexpr (DF) {
      for (int r = gl; r < NT; r += G) {
        const int nu = nu_of(mu, r);
        Mat<3, float> t = product<DF>(U, g, x, mu, r, nu, df);
        if (r < ND - 1) t = mul_nd(t, load_link<3, float, DF>(U, g, x, nu, df));
        part[r] = t;
      }
    } else {
      p += mu * NT;
      if (gl < ND - 1) fwd[gl] = mul_nd(p[gl], load_link<3, float, DF>(U, g, x, nu_of(mu, gl), df));
    }
    __syncwarp(mask);
    Mat<3, float> S = mzero<3, float>();
#pragma unroll 1
    for (int k = 0; k < ND - 1; ++k) madd(S, DF ? p[k] : fwd[k]);
#pragma unroll 1
    for (int k = ND - 1; k < NT; ++k) madd(S, p[k]);
    return S;
  }
};

// The links of site x in the order mu = 0 .. Nd-1; hits(S, U, dlink) updates one link
// and returns its accepted hits, the same in every lane.
template <int ND, bool DF, int G, typename Hits>
KLFT_D int group_links(StapleTerms<ND> &sh, const Links<3, float> &U, const Geom &g, const Site &x, const Defect &df,
                       Hits &&hits) {
  const long long lx = site_lin(g, x);
  const int gl = (int)(threadIdx.x & (unsigned)(G - 1));
  const unsigned mask = group_mask<G>();
  sh.template load<DF, G>(U, g, x, df, gl);
  __syncwarp(mask);
  const bool own0 = DF && df.active && in_defect(g, df, x, 0);
  int nacc = 0;
#pragma unroll 1
  for (int mu = 0; mu < ND; ++mu) {
    if (open_link(g, x, mu)) continue;
    const Mat<3, float> S = sh.template staple<DF, G>(U, g, x, mu, df, gl, mask);
    Mat<3, float> V = U.load(lx, mu);
    const int n = hits(S, V, mu == 0 && own0);
    __syncwarp(mask);  // every lane has read the link and the terms
    if (n && gl == 0) U.store(lx, mu, V);
    __syncwarp(mask);
    nacc += n;
  }
  return nacc;
}

// The same from shared parts.
template <int ND, bool DF, int G, int NC, typename T, typename Hits>
KLFT_D int group_links(StapleParts<NC, ND, T> &sh, const Links<NC, T> &U, const Geom &g, const Site &x,
                       const Defect &df, Hits &&hits) {
  const long long lx = site_lin(g, x);
  const int gl = (int)(threadIdx.x & (unsigned)(G - 1));
  const unsigned mask = group_mask<G>();
  sh.template load<DF, G>(U, g, x, lx, df, gl);
  __syncwarp(mask);
  const bool own0 = DF && df.active && in_defect(g, df, x, 0);
  int nacc = 0;
#pragma unroll 1
  for (int mu = 0; mu < ND; ++mu) {
    if (open_link(g, x, mu)) continue;
    Mat<NC, T> V = sh.own[mu];
    const int n = hits(sh.template staple<DF>(mu, own0, df), V, mu == 0 && own0);
    if (n) {
      __syncwarp(mask);
      if (gl == 0) {
        U.store(lx, mu, V);
        sh.own[mu] = V;
      }
      __syncwarp(mask);
    }
    nacc += n;
  }
  return nacc;
}

// ------------------------------------------------------------------ SU(3)
// The hits of a site's links, one per lane.
template <typename T, int G> struct LaneHits3 {
  const MetroArgs &a;
  const SiteStream st;
  const int gl;         // lane in the group
  const unsigned mask;  // the group's lanes
  uint32_t pos = 0;     // place of the next hit in the stream
  // this lane's hit of the chunk: proposal, the uniform after it, uniforms it took
  Mat<3, T> rr;
  double uacc = 0.0;
  uint32_t used = 12u;
  int ci = G;  // the chunk's next hit (G: none left)

  KLFT_D LaneHits3(const MetroArgs &args, const SiteStream &stream)
      : a(args), st(stream), gl((int)(threadIdx.x & (unsigned)(G - 1))), mask(group_mask<G>()) {}

  // lane j: the proposal of the j-th hit from pos if no place is skipped
  KLFT_D void chunk() {
    HitDraws<3> d(st);
    d.pos = pos + 13u * (uint32_t)gl;
    if (d.pos & 1u) {
      double u0;
      st.block(d.pos >> 1, u0, d.carry);
    }
    rr = d.template propose_next<T>(a.delta, uacc);
    used = d.used;
    ci = 0;
  }

  // the hits of a link; Uo: the link, updated; the number accepted
  KLFT_D int hits(const Mat<3, T> &S, Mat<3, T> &Uo, T bnc, bool dlink, T cdef) {
    int nacc = 0;
    Mat<3, T> M = mul(S, Uo);
    T trO = retr_diag(M);
    int hit = 0;
    while (hit < a.nhits) {
      if (ci == G) chunk();
      const int n = a.nhits - hit < G - ci ? a.nhits - hit : G - ci;
      const bool mine = gl >= ci && gl < ci + n;
      bool down = false, accept = false;
      if (mine) {
        T dS = -bnc * (retr_mul(rr, M) - trO);
        if (dlink) dS *= cdef;
        down = dS < T(0);
        accept = down || accept_uniform(dS, uacc);
      }
      const unsigned ev = __ballot_sync(mask, mine && (accept || down || used != 12u));
      if (!ev) {
        hit += n;
        ci += n;
        pos += 13u * (uint32_t)n;
        continue;
      }
      const int src = __ffs((int)ev) - 1;  // lane of the warp
      const int f = src & (G - 1);
      const bool fdown = __shfl_sync(mask, down, src), facc = __shfl_sync(mask, accept, src);
      const uint32_t fused = __shfl_sync(mask, used, src);
      pos += 13u * (uint32_t)(f - ci);
      hit += f - ci + 1;
      if (facc) {
        Mat<3, T> r;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            r.e[i][j].re = __shfl_sync(mask, rr.e[i][j].re, src);
            r.e[i][j].im = __shfl_sync(mask, rr.e[i][j].im, src);
          }
        Uo = restore(mul(Uo, r));
        M = mul(S, Uo);
        trO = retr_diag(M);
        ++nacc;
      }
      const uint32_t step = fused + (fdown ? 0u : 1u);
      pos += step;
      ci = step == 13u ? f + 1 : G;  // the chunk's later proposals hold unless the place moved
    }
    return nacc;
  }
};

// ------------------------------------------------------------------ one site
// Whether the staples are formed from shared parts.  In FP32 U(1) and SU(2) they
// are not: every lane forms the staple as site_update_ref does (staple_f32), from
// links already in L1.
template <int NC, typename T> struct SharedStaples { static constexpr bool v = NC == 3 || sizeof(T) == 8; };

template <int NC, int ND, typename T, int G> struct GroupShared {
  DrawTable<NC, T, G> table;
  StapleParts<NC, SharedStaples<NC, T>::v ? ND : 1, T> parts;
};
template <int ND, int G> struct GroupShared<3, ND, double, G> { StapleParts<3, ND, double> parts; };
template <int ND, int G> struct GroupShared<3, ND, float, G> { StapleTerms<ND> parts; };

// Site t (if t < Vh) of class val by the calling thread's group; sh: one entry per
// group of the CTA.  Every thread of the CTA calls it and passes the wait.  The
// sweep counter is read before it: a pass launched as a programmatic dependent
// has only passes of its own sweep before it that may still run.  Accepted hits,
// counted in one lane of the group.
template <int NC, int ND, typename T, bool DF, int G>
KLFT_D int group_site_update(GroupShared<NC, ND, T, G> *shared, const Links<NC, T> &U, const Geom &g, long long t, int val, const MetroArgs &a, uint32_t sweep, const Defect &df) {
  const bool ok = t < g.Vh;
  const Site x = pass_site(g, ok ? t : 0, val, ND);
  const SiteStream st(a.seed, a.chain, site_lex(g, x), sweep, KIND_METROPOLIS);
  GroupShared<NC, ND, T, G> &sh = shared[threadIdx.x / G];
  const int gl = (int)(threadIdx.x & (unsigned)(G - 1));
  const T bnc = (T)a.beta / (T)NC;
  int n = 0;
  if constexpr (NC == 3) {
    LaneHits3<T, G> lanes(a, st);
    if (ok) lanes.chunk();
    grid_dependency_wait();
    grid_launch_dependents();
    if (ok)
      n = group_links<ND, DF, G>(sh.parts, U, g, x, df, [&](const Mat<3, T> &S, Mat<3, T> &V, bool dlink) {
        return lanes.hits(S, V, bnc, dlink, dlink ? (T)defect_c(df) : T(1));
      });
  } else {
    TableDraws<NC, T, G> rng(sh.table, st, a.delta, (long long)ND * a.nhits);
    if (ok) rng.fill();
    grid_dependency_wait();
    grid_launch_dependents();
    if (ok) {
      if constexpr (SharedStaples<NC, T>::v) {
        n = group_links<ND, DF, G>(sh.parts, U, g, x, df, [&](const Mat<NC, T> &S, Mat<NC, T> &V, bool dlink) {
          return group_hits<NC>(S, V, a, dlink, df, rng, bnc);
        });
      } else {
        // every lane: the same links and decisions
        static_assert(!DF, "FP32 U(1), SU(2): lattices without a defect");
        touch_neighbours<NC, ND, T, G>(U, g, x, gl);
        __syncwarp(rng.mask);
        n = group_link_f32<NC, ND, 0>(U, g, x, a, rng);
        n += group_link_f32<NC, ND, 1>(U, g, x, a, rng);
        n += group_link_f32<NC, ND, 2>(U, g, x, a, rng);
        n += group_link_f32<NC, ND, 3>(U, g, x, a, rng);
      }
    }
  }
  return gl == 0 ? n : 0;
}

// ------------------------------------------------------------------ kernels
// the reference-proposal pass of one lattice
template <int NC, int ND, typename T, bool DF, int G>
__global__ void __launch_bounds__(GROUP_THREADS)
    metropolis_group_kernel(Links<NC, T> U, Geom g, int val, MetroArgs a, const uint32_t *__restrict__ d_sweep,
                            unsigned long long *__restrict__ d_nacc, Defect df) {
  __shared__ GroupShared<NC, ND, T, G> sh[GROUP_THREADS / G];
  const long long t = ((long long)blockIdx.x * GROUP_THREADS + threadIdx.x) / G;
  add_accepts(group_site_update<NC, ND, T, DF, G>(sh, U, g, t, val, a, *d_sweep, df), d_nacc);
}

// the same pass of many chains (multi_pass_kernel)
template <int NC, int ND, typename T, bool DF, int G>
__global__ void __launch_bounds__(GROUP_THREADS)
    multi_group_kernel(const __grid_constant__ ChainTable tab, int val, unsigned long long *nacc_slots,
                       const uint32_t *__restrict__ slot) {
  __shared__ GroupShared<NC, ND, T, G> sh[GROUP_THREADS / G];
  const ChainDesc &c = tab.c[find_chain(tab)];
  const long long t = ((long long)(blockIdx.x - c.block_begin) * GROUP_THREADS + threadIdx.x) / G;
  const Links<NC, T> U{(cx<T> *)c.links, c.g.V};
  add_accepts(group_site_update<NC, ND, T, DF, G>(sh, U, c.g, t, val, c.a, *c.ctr, c.df),
              nacc_slots + (size_t)(*slot) * tab.nchains_total + c.index);
}

// The passes of a sweep after its first start before the kernel before them in the
// stream, a pass of the same sweep, has ended.
template <int NC, int ND, typename T, bool DF, int G> static cudaError_t launch_group_t(const GroupLaunch &l) {
  if (l.tab) {
    return launch_after(l.val > 0, multi_group_kernel<NC, ND, T, DF, G>, dim3(l.blocks), dim3(GROUP_THREADS), 0, l.st,
                        *l.tab, l.val, l.nacc, l.slot);
  }
  const Geom &g = *l.g;
  return launch_after(l.val > 0, metropolis_group_kernel<NC, ND, T, DF, G>, dim3((unsigned)group_blocks(g.Vh, G)),
                      dim3(GROUP_THREADS), 0, l.st, Links<NC, T>{(cx<T> *)l.links, g.V}, g, l.val, *l.a, l.d_sweep,
                      l.nacc, *l.df);
}

template <int NC, int ND, typename T, bool DF> static cudaError_t launch_group_df(int G, const GroupLaunch &l) {
  // the widths group_lanes gives
  if constexpr (NC == 3) return G == 32 ? launch_group_t<NC, ND, T, DF, 32>(l) : launch_group_t<NC, ND, T, DF, 8>(l);
  else if constexpr (sizeof(T) == 4)
    return NC == 1 && G == 4 ? launch_group_t<NC, ND, T, DF, (NC == 1 ? 4 : 8)>(l) : launch_group_t<NC, ND, T, DF, 8>(l);
  else if constexpr (NC == 1)
    return G == 32 ? launch_group_t<NC, ND, T, DF, 32>(l)
                   : (G == 16 ? launch_group_t<NC, ND, T, DF, 16>(l) : launch_group_t<NC, ND, T, DF, 8>(l));
  else return G == 32 ? launch_group_t<NC, ND, T, DF, 32>(l) : launch_group_t<NC, ND, T, DF, 16>(l);
}

template <int NC, int ND, typename T> static cudaError_t launch_group_nd(int G, bool defect, const GroupLaunch &l) {
  if constexpr (SharedStaples<NC, T>::v) {
    if (defect) return launch_group_df<NC, ND, T, true>(G, l);
  } else {
    if (defect) return cudaErrorInvalidValue;  // group_lanes gives 1
  }
  return launch_group_df<NC, ND, T, false>(G, l);
}

template <int NC> static cudaError_t launch_group_nc(int nd, int dtype, int G, bool defect, const GroupLaunch &l) {
  if (dtype == 0) {
    if (nd == 2) return launch_group_nd<NC, 2, double>(G, defect, l);
    if (nd == 3) return launch_group_nd<NC, 3, double>(G, defect, l);
    return launch_group_nd<NC, 4, double>(G, defect, l);
  }
  if (nd == 2) return launch_group_nd<NC, 2, float>(G, defect, l);
  if (nd == 3) return launch_group_nd<NC, 3, float>(G, defect, l);
  return launch_group_nd<NC, 4, float>(G, defect, l);
}

// per group, each in its own translation unit
cudaError_t launch_group_u1(int nd, int dtype, int G, bool defect, const GroupLaunch &l);
cudaError_t launch_group_su2(int nd, int dtype, int G, bool defect, const GroupLaunch &l);
cudaError_t launch_group_su3(int nd, int dtype, int G, bool defect, const GroupLaunch &l);

}  // namespace klft
