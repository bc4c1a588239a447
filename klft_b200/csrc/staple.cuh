// staple.cuh -- the staple of a link, GaugeField.hpp:187-237 (3D :389-433,
// 2D :579-618) with the PTBC defect factors of PTBCGaugeField.hpp:232-277:
//   S = sum_{nu != mu} U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+
//     + sum_{nu != mu} U_nu(x+mu-nu)^+ U_mu(x-nu)^+ U_nu(x-nu)
// accumulated in the reference's order (all forward terms, then all backward).
#pragma once
#include "common.cuh"

namespace klft {

// DF = false compiles the defect handling out (lattices without a PTBC defect).
template <int NC, typename T, bool DF>
KLFT_D Mat<NC, T> load_link(const Links<NC, T> &U, const Geom &g, const Site &s, int mu, const Defect &df) {
  Mat<NC, T> m = U.load(site_lin(g, s), mu);
  if constexpr (DF) {
    if (df.active && in_defect(g, df, s, mu)) m = mscale(m, (T)defect_c(df));
  }
  return m;
}

// The nu loops stay rolled: the update kernels are instruction-fetch bound when
// the 4(Nd-1) products are all inlined next to the proposal code.
template <int NC, int ND, typename T, bool DF = false>
KLFT_D Mat<NC, T> staple(const Links<NC, T> &U, const Geom &g, const Site &x, int mu, const Defect &df) {
  Mat<NC, T> S = mzero<NC, T>();
  const Site xpmu = site_up(g, x, mu);
#pragma unroll 1
  for (int nu = 0; nu < ND; ++nu) {
    if (nu == mu) continue;
    const Site xpnu = site_up(g, x, nu);
    const Mat<NC, T> t = mul_nd(load_link<NC, T, DF>(U,g, xpmu, nu, df), load_link<NC, T, DF>(U,g, xpnu, mu, df));
    madd(S, mul_nd(t, load_link<NC, T, DF>(U,g, x, nu, df)));
  }
#pragma unroll 1
  for (int nu = 0; nu < ND; ++nu) {
    if (nu == mu) continue;
    const Site xpmu_mnu = site_dn(g, xpmu, nu);
    const Site xmnu = site_dn(g, x, nu);
    const Mat<NC, T> t = mul_dd(load_link<NC, T, DF>(U,g, xpmu_mnu, nu, df), load_link<NC, T, DF>(U,g, xmnu, mu, df));
    madd(S, mul(t, load_link<NC, T, DF>(U,g, xmnu, nu, df)));
  }
  return S;
}

// SU(3) with links stored as two FP32 rows (the mixed form, no defect): every
// staple term is a product of three SU(3) links and so itself in SU(3), which
// lets most of its third rows come from the first two (row 2 = conj(row 0 x
// row 1)) instead of from products:
//   forward  A B^+ C^+ = A (C B)^+,  backward  D^+ E^+ G = (E D)^+ G,
// with C B and E D formed on their first two rows (C and E need no third row),
// completed, and each term formed on its first two rows and completed.  Same
// terms in the same order as staple(); rounding differs at FP32 level.
template <typename T> KLFT_D void complete_row2(Mat<3, T> &m) {
  m.e[2][0] = conj(m.e[0][1] * m.e[1][2] - m.e[0][2] * m.e[1][1]);
  m.e[2][1] = conj(m.e[0][2] * m.e[1][0] - m.e[0][0] * m.e[1][2]);
  m.e[2][2] = conj(m.e[0][0] * m.e[1][1] - m.e[0][1] * m.e[1][0]);
}
// rows 0, 1 of a b (a's third row is not read)
template <typename T> KLFT_D void mul_rows01(const Mat<3, T> &a, const Mat<3, T> &b, Mat<3, T> &c) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) c.e[i][j] = a.e[i][0] * b.e[0][j] + a.e[i][1] * b.e[1][j] + a.e[i][2] * b.e[2][j];
}
// rows 0, 1 of a b^+
template <typename T> KLFT_D void mul_nd_rows01(const Mat<3, T> &a, const Mat<3, T> &b, Mat<3, T> &c) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      c.e[i][j] = a.e[i][0] * conj(b.e[j][0]) + a.e[i][1] * conj(b.e[j][1]) + a.e[i][2] * conj(b.e[j][2]);
}
// rows 0, 1 of a^+ b
template <typename T> KLFT_D void mul_dn_rows01(const Mat<3, T> &a, const Mat<3, T> &b, Mat<3, T> &c) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      c.e[i][j] = conj(a.e[0][i]) * b.e[0][j] + conj(a.e[1][i]) * b.e[1][j] + conj(a.e[2][i]) * b.e[2][j];
}

// The two-row staple with mu fixed at compile time and the nu loops unrolled:
// each link pass compiles its own site steps and can issue the loads of
// several terms ahead of their products.  1.62 -> 1.50 ms per SU(3) 32^4 sweep
// against a run-time mu (1.56 with the nu loops rolled).
template <int ND, int MU>
KLFT_D Mat<3, float> staple_su3_2row_ct(const Links<3, float> &U, const Geom &g, const Site &x) {
  Mat<3, float> S = mzero<3, float>();
  const int lin = (int)site_lin(g, x), pmu = lin + step_up(g, x, MU);
#pragma unroll
  for (int nu = 0; nu < ND; ++nu) {
    if (nu == MU) continue;
    Mat<3, float> cb, f;
    mul_rows01(U.load_rows01(lin, nu), U.load(lin + step_up(g, x, nu), MU), cb);
    complete_row2(cb);
    mul_nd_rows01(U.load_rows01(pmu, nu), cb, f);
    complete_row2(f);
    madd(S, f);
  }
#pragma unroll
  for (int nu = 0; nu < ND; ++nu) {
    if (nu == MU) continue;
    const int dn = step_dn(g, x, nu);
    Mat<3, float> ed, f;
    mul_rows01(U.load_rows01(lin + dn, MU), U.load(pmu + dn, nu), ed);
    complete_row2(ed);
    mul_dn_rows01(ed, U.load(lin + dn, nu), f);
    complete_row2(f);
    madd(S, f);
  }
  return S;
}

// The same staple with mu fixed at compile time and the nu loops unrolled: the
// same products in the same order, but every site step and index folds to a few
// integer operations.  For kernels without proposal code (the HMC force), where
// the unrolled products fit the instruction cache.
// DF: the PTBC defect factors as in staple() (only links of direction 0 can
// carry one, which the compiled direction makes visible to the compiler).
template <int NC, int ND, int MU, typename T, bool DF = false>
KLFT_D Mat<NC, T> staple_ct(const Links<NC, T> &U, const Geom &g, const Site &x, const Defect &df = Defect{}) {
  Mat<NC, T> S = mzero<NC, T>();
  if constexpr (!DF && (NC == 3 || sizeof(T) == 8)) {
    // neighbours as sums of two steps.  Not in FP32 for U(1) and SU(2): the compiler
    // contracts their sums of two products in another order then, and the chain's
    // last bits (HMC's dH, Metropolis decisions) with them.
    const int lin = (int)site_lin(g, x), pmu = lin + step_up(g, x, MU);
#pragma unroll
    for (int nu = 0; nu < ND; ++nu) {
      if (nu == MU) continue;
      const Mat<NC, T> t = mul_nd(U.load(pmu, nu), U.load(lin + step_up(g, x, nu), MU));
      madd(S, mul_nd(t, U.load(lin, nu)));
    }
#pragma unroll
    for (int nu = 0; nu < ND; ++nu) {
      if (nu == MU) continue;
      const int dn = step_dn(g, x, nu);
      const Mat<NC, T> t = mul_dd(U.load(pmu + dn, nu), U.load(lin + dn, MU));
      madd(S, mul(t, U.load(lin + dn, nu)));
    }
    return S;
  }
  const Site xpmu = site_up(g, x, MU);
#pragma unroll
  for (int nu = 0; nu < ND; ++nu) {
    if (nu == MU) continue;
    const Site xpnu = site_up(g, x, nu);
    const Mat<NC, T> t = mul_nd(load_link<NC, T, DF>(U, g, xpmu, nu, df), load_link<NC, T, DF>(U, g, xpnu, MU, df));
    madd(S, mul_nd(t, load_link<NC, T, DF>(U, g, x, nu, df)));
  }
#pragma unroll
  for (int nu = 0; nu < ND; ++nu) {
    if (nu == MU) continue;
    const Site xpmu_mnu = site_dn(g, xpmu, nu);
    const Site xmnu = site_dn(g, x, nu);
    const Mat<NC, T> t =
        mul_dd(load_link<NC, T, DF>(U, g, xpmu_mnu, nu, df), load_link<NC, T, DF>(U, g, xmnu, MU, df));
    madd(S, mul(t, load_link<NC, T, DF>(U, g, xmnu, nu, df)));
  }
  return S;
}

// ------------------------------------------------------------------ U(1), SU(2) in FP32
// Products with their FMAs written out, on what is stored of a link: row 0, of which an
// SU(2) element's row 1 is (-conj(v1), conj(v0)).
KLFT_D float mad2(float a, float b, float c, float d) { return fmaf(a, b, __fmul_rn(c, d)); }  // a b + c d

template <int NC> struct Row0 { cx<float> v[NC]; };  // SU(2): row 0 of the matrix
template <int NC> KLFT_D Row0<NC> row0(const Mat<NC, float> &m) {
  Row0<NC> r;
#pragma unroll
  for (int j = 0; j < NC; ++j) r.v[j] = m.e[0][j];
  return r;
}
// a b
KLFT_D Row0<1> f32_mul(const Row0<1> &x, const Row0<1> &y) {
  const cx<float> a = x.v[0], b = y.v[0];
  return {{mk<float>(mad2(a.re, b.re, -a.im, b.im), mad2(a.im, b.re, a.re, b.im))}};
}
KLFT_D float su2_re00(const Row0<2> &x, const Row0<2> &y) {
  const cx<float> a = x.v[0], b = x.v[1], c = y.v[0], d = y.v[1];
  return __fadd_rn(mad2(a.re, c.re, -a.im, c.im), mad2(b.re, -d.re, -b.im, d.im));
}
KLFT_D Row0<2> f32_mul(const Row0<2> &x, const Row0<2> &y) {
  const cx<float> a = x.v[0], b = x.v[1], c = y.v[0], d = y.v[1];
  return {{mk<float>(su2_re00(x, y), __fadd_rn(mad2(a.im, c.re, a.re, c.im), mad2(b.re, d.im, b.im, -d.re))),
           mk<float>(__fadd_rn(mad2(a.re, d.re, -a.im, d.im), mad2(b.re, c.re, b.im, c.im)),
                     __fadd_rn(mad2(a.im, d.re, a.re, d.im), mad2(b.im, c.re, b.re, -c.im)))}};
}
// a b^+
KLFT_D Row0<1> f32_mul_nd(const Row0<1> &x, const Row0<1> &y) {
  const cx<float> a = x.v[0], b = y.v[0];
  return {{mk<float>(mad2(a.re, b.re, a.im, b.im), mad2(a.im, b.re, a.re, -b.im))}};
}
KLFT_D Row0<2> f32_mul_nd(const Row0<2> &x, const Row0<2> &y) {
  const cx<float> a = x.v[0], b = x.v[1], c = y.v[0], d = y.v[1];
  return {{mk<float>(__fadd_rn(mad2(a.re, c.re, a.im, c.im), mad2(b.re, d.re, b.im, d.im)),
                     __fadd_rn(mad2(a.im, c.re, a.re, -c.im), mad2(b.im, d.re, b.re, -d.im))),
           mk<float>(__fadd_rn(mad2(a.im, d.im, a.re, -d.re), mad2(b.re, c.re, -b.im, c.im)),
                     __fadd_rn(mad2(a.im, -d.re, a.re, -d.im), mad2(b.im, c.re, b.re, c.im)))}};
}
// a^+ b^+
KLFT_D Row0<1> f32_mul_dd(const Row0<1> &x, const Row0<1> &y) {
  const cx<float> a = x.v[0], b = y.v[0];
  return {{mk<float>(mad2(a.re, b.re, a.im, -b.im), mad2(-a.im, b.re, a.re, -b.im))}};
}
KLFT_D Row0<2> f32_mul_dd(const Row0<2> &x, const Row0<2> &y) {
  const cx<float> a = x.v[0], b = x.v[1], c = y.v[0], d = y.v[1];
  return {{mk<float>(__fadd_rn(mad2(a.re, c.re, a.im, -c.im), mad2(-b.re, d.re, b.im, -d.im)),
                     __fadd_rn(mad2(-a.im, c.re, a.re, -c.im), mad2(b.re, d.im, -b.im, d.re))),
           mk<float>(__fadd_rn(mad2(a.re, -d.re, a.im, -d.im), mad2(b.im, c.im, -b.re, c.re)),
                     __fadd_rn(mad2(-a.im, -d.re, a.re, -d.im), mad2(-b.im, c.re, -b.re, c.im)))}};
}
template <int NC> KLFT_D void f32_add(Row0<NC> &s, const Row0<NC> &a) {
#pragma unroll
  for (int j = 0; j < NC; ++j) s.v[j] = mk<float>(__fadd_rn(s.v[j].re, a.v[j].re), __fadd_rn(s.v[j].im, a.v[j].im));
}
// The staple of U_mu(x), mu = MU, without a defect: the terms of staple_ct.  The forms
// are those nvcc 12.9 chose for staple_ct in the Metropolis passes, the same in every
// direction and dimension: found one product and component at a time on fields whose
// other terms cancel exactly, so that the sum left is zero or a rounding error.
template <int NC, int ND, int MU> KLFT_D Row0<NC> staple_f32(const Links<NC, float> &U, const Geom &g, const Site &x) {
  auto link = [&](const Site &s, int mu) { return row0(U.load(site_lin(g, s), mu)); };
  Row0<NC> S = row0(mzero<NC, float>());
  const Site xpmu = site_up(g, x, MU);
#pragma unroll
  for (int nu = 0; nu < ND; ++nu) {
    if (nu == MU) continue;
    f32_add(S, f32_mul_nd(f32_mul_nd(link(xpmu, nu), link(site_up(g, x, nu), MU)), link(x, nu)));
  }
#pragma unroll
  for (int nu = 0; nu < ND; ++nu) {
    if (nu == MU) continue;
    const Site xmnu = site_dn(g, x, nu);
    f32_add(S, f32_mul(f32_mul_dd(link(site_dn(g, xpmu, nu), nu), link(xmnu, MU)), link(xmnu, nu)));
  }
  return S;
}

// staple_ct for a run-time mu (uniform across a warp in the callers)
template <int NC, int ND, typename T>
KLFT_D Mat<NC, T> staple_dispatch(const Links<NC, T> &U, const Geom &g, const Site &x, int mu) {
  if (mu == 0) return staple_ct<NC, ND, 0, T>(U, g, x);
  if (mu == 1) return staple_ct<NC, ND, 1, T>(U, g, x);
  if constexpr (ND > 2) {
    if (mu == 2) return staple_ct<NC, ND, 2, T>(U, g, x);
  }
  if constexpr (ND > 3) return staple_ct<NC, ND, 3, T>(U, g, x);
  return staple_ct<NC, ND, ND - 1, T>(U, g, x);
}

// Site of a class-blocked index lin = sub * Vh + hidx in 32-bit arithmetic
// (lattices with Vh < 2^31).
KLFT_D Site site_from_lin32(const Geom &g, unsigned lin) {
  Site s;
  const unsigned vh = (unsigned)g.Vh;
  const unsigned sub = lin / vh;
  unsigned hidx = lin - sub * vh;
#pragma unroll
  for (int d = 0; d < 4; ++d) {
    const unsigned hd = (unsigned)g.H[d];
    const unsigned q = hidx / hd;
    s.set_b(d, (int)((sub >> d) & 1u));
    s.set_h(d, (int)(hidx - q * hd));
    hidx = q;
  }
  return s;
}

}  // namespace klft
