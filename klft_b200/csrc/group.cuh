// group.cuh -- group-specific device math: Metropolis proposals, Haar-random
// links, and the Lie-algebra maps used by HMC (the SU(3) exponential is in
// expprop.cuh).
#pragma once
#include "common.cuh"
#include "expprop.cuh"

namespace klft {

constexpr double KPI = 3.141592653589793;
constexpr double K2PI = 6.283185307179586;

enum Proposal : int { PROPOSAL_REFERENCE = 0, PROPOSAL_EXP = 1 };

// ------------------------------------------------------------------ proposals
// The proposals read RefDraws<NC>::n consecutive uniforms of the site's stream (SU(3):
// 12 unless a drawn vector has norm zero); the accept uniform, when drawn, follows.
template <int NC> struct RefDraws { static constexpr int n = NC == 1 ? 1 : (NC == 2 ? 3 : 12); };

// U(1): exp(i phi), phi uniform in [-delta*pi, delta*pi]   (SUN.hpp:163-171)
template <typename T> KLFT_D Mat<1, T> propose(const double *u, double delta, const Mat<1, T> *) {
  const double phi = drand_u(-delta * KPI, delta * KPI, u[0]);
  Mat<1, T> r;
  r.e[0][0] = mk<T>((T)cos(phi), (T)sin(phi));
  return r;
}
// SU(2): cos(a) + i sin(a) n.sigma  (SUN.hpp:174-189)
template <typename T> KLFT_D Mat<2, T> propose(const double *w, double delta, const Mat<2, T> *) {
  const T alpha = (T)drand_u(0.0, delta * 2 * KPI, w[0]);
  const T u = (T)drand_u(-1.0, 1.0, w[1]);
  const T theta = (T)drand_u(0.0, 2.0 * KPI, w[2]);
  const T salpha = sin(alpha);
  const T su = sqrt(fma(-u, u, T(1)));
  const T n1 = su * sin(theta);
  const T n2 = su * cos(theta);
  Mat<2, T> r;
  r.e[0][0] = mk<T>(cos(alpha), u * salpha);
  r.e[0][1] = mk<T>(n1 * salpha, n2 * salpha);
  su2_row1(r);
  return r;
}
// SU(3): reference Gram-Schmidt proposal (SUN.hpp:192-251); the exp(i eps H)
// proposal has its own fixed-position stream (expprop.cuh).  The reference draws
// a vector again while its norm is zero.  next() gives the uniforms in order;
// false: a first draw had norm zero (the caller then redraws in stream order).
template <typename T, typename Next> KLFT_D bool su3_vec(Next &next, double delta, T v[6], T &norm) {
#pragma unroll
  for (int i = 0; i < 6; ++i) v[i] = (T)drand_u(0.0, delta, next());
  norm = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3] + v[4] * v[4] + v[5] * v[5]);
  return T(1) != (T(1) + norm);
}
template <typename T> KLFT_D void su3_row1(const T v[6], T norm, cx<T> z1[3]) {
  const T fact = T(1) / norm;
  z1[0] = fact * mk<T>(v[0], v[1]);
  z1[1] = fact * mk<T>(v[2], v[3]);
  z1[2] = fact * mk<T>(v[4], v[5]);
}
// z2 orthogonal to z1, its norm before normalisation returned
template <typename T> KLFT_D T su3_row2(const T v[6], T n, const cx<T> z1[3], cx<T> z2[3]) {
  su3_row1(v, n, z2);
  const cx<T> z = conj(z1[0]) * z2[0] + conj(z1[1]) * z2[1] + conj(z1[2]) * z2[2];
  z2[0] -= z * z1[0];
  z2[1] -= z * z1[1];
  z2[2] -= z * z1[2];
  return sqrt(z2[0].re * z2[0].re + z2[0].im * z2[0].im + z2[1].re * z2[1].re + z2[1].im * z2[1].im +
              z2[2].re * z2[2].re + z2[2].im * z2[2].im);
}
template <typename T> KLFT_D Mat<3, T> su3_rows(const cx<T> z1[3], const cx<T> z2in[3], T norm) {
  const T fact = T(1) / norm;
  cx<T> z2[3], z3[3];
  z2[0] = z2in[0] * fact;
  z2[1] = z2in[1] * fact;
  z2[2] = z2in[2] * fact;
  z3[0] = conj((z1[1] * z2[2]) - (z1[2] * z2[1]));
  z3[1] = conj((z1[2] * z2[0]) - (z1[0] * z2[2]));
  z3[2] = conj((z1[0] * z2[1]) - (z1[1] * z2[0]));
  Mat<3, T> r;
#pragma unroll
  for (int j = 0; j < 3; ++j) { r.e[0][j] = z1[j]; r.e[1][j] = z2[j]; r.e[2][j] = z3[j]; }
  return r;
}
template <typename T, typename Next> KLFT_D bool su3_propose(Next &next, double delta, Mat<3, T> &r) {
  T v[6], norm;
  cx<T> z1[3], z2[3];
  bool ok = su3_vec<T>(next, delta, v, norm);
  su3_row1(v, norm, z1);
  ok = su3_vec<T>(next, delta, v, norm) && ok;
  norm = su3_row2(v, norm, z1, z2);
  ok = ok && T(1) != (T(1) + norm);
  r = su3_rows(z1, z2, norm);
  return ok;
}
// The reference's redraws, in stream order (probability near 1e-16 per hit).
// They are bounded here (the host rejects delta <= 0, for which they never end).
template <typename T> __device__ __noinline__ void su3_propose_redraw(Stream &g, double delta, Mat<3, T> &r) {
  auto next = [&] { return g.next(); };
  T v[6], norm = T(0);
  cx<T> z1[3], z2[3];
  for (int tries = 0; tries < 64; ++tries)
    if (su3_vec<T>(next, delta, v, norm)) break;
  su3_row1(v, norm, z1);
  for (int outer = 0; outer < 64; ++outer) {
    for (int tries = 0; tries < 64; ++tries)
      if (su3_vec<T>(next, delta, v, norm)) break;
    norm = su3_row2(v, norm, z1, z2);
    if (T(1) != (T(1) + norm)) break;
  }
  r = su3_rows(z1, z2, norm);
}

// ------------------------------------------------------------------ hot start
template <typename T> KLFT_D Mat<1, T> haar(Stream &g, const Mat<1, T> *) {
  const double phi = g.drand(-KPI, KPI);
  Mat<1, T> m;
  m.e[0][0] = mk<T>((T)cos(phi), (T)sin(phi));
  return m;
}
template <typename T> KLFT_D Mat<2, T> haar(Stream &g, const Mat<2, T> *) {
  double q[4];
  g.gauss2(q[0], q[1]);
  g.gauss2(q[2], q[3]);
  const double n = sqrt(q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
#pragma unroll
  for (int k = 0; k < 4; ++k) q[k] /= n;
  Mat<2, T> m;
  m.e[0][0] = mk<T>((T)q[0], (T)q[3]);
  m.e[0][1] = mk<T>((T)q[2], (T)q[1]);
  m.e[1][0] = mk<T>((T)-q[2], (T)q[1]);
  m.e[1][1] = mk<T>((T)q[0], (T)-q[3]);
  return m;
}
template <typename T> KLFT_D Mat<3, T> haar(Stream &g, const Mat<3, T> *) {
  cx<double> r0[3], r1[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) { double a, b; g.gauss2(a, b); r0[j] = mk(a, b); }
#pragma unroll
  for (int j = 0; j < 3; ++j) { double a, b; g.gauss2(a, b); r1[j] = mk(a, b); }
  const double n0 = sqrt(r0[0].re * r0[0].re + r0[0].im * r0[0].im + r0[1].re * r0[1].re + r0[1].im * r0[1].im +
                         r0[2].re * r0[2].re + r0[2].im * r0[2].im);
#pragma unroll
  for (int j = 0; j < 3; ++j) r0[j] = cdiv(r0[j], n0);
  // products in the compiler's contraction (restore_plain)
  auto p = [](cx<double> x, cx<double> y) { return cmul_plain(x, y); };
  const cx<double> z = p(conj(r0[0]), r1[0]) + p(conj(r0[1]), r1[1]) + p(conj(r0[2]), r1[2]);
#pragma unroll
  for (int j = 0; j < 3; ++j) r1[j] -= p(z, r0[j]);
  const double n1 = sqrt(r1[0].re * r1[0].re + r1[0].im * r1[0].im + r1[1].re * r1[1].re + r1[1].im * r1[1].im +
                         r1[2].re * r1[2].re + r1[2].im * r1[2].im);
#pragma unroll
  for (int j = 0; j < 3; ++j) r1[j] = cdiv(r1[j], n1);
  cx<double> r2[3];
  r2[0] = conj(p(r0[1], r1[2]) - p(r0[2], r1[1]));
  r2[1] = conj(p(r0[2], r1[0]) - p(r0[0], r1[2]));
  r2[2] = conj(p(r0[0], r1[1]) - p(r0[1], r1[0]));
  Mat<3, T> m;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    m.e[0][j] = mk<T>((T)r0[j].re, (T)r0[j].im);
    m.e[1][j] = mk<T>((T)r1[j].re, (T)r1[j].im);
    m.e[2][j] = mk<T>((T)r2[j].re, (T)r2[j].im);
  }
  return m;
}

// ------------------------------------------------------------------ Lie algebra (HMC)
template <int N> struct Alg { static constexpr int n = N == 1 ? 1 : (N == 2 ? 3 : 8); };

// Adj(M): U(1) Im M (AdjointGroup.hpp:114-117); SU(2) (2 Im M01, 2 Re M01, 2 Im M00)
// (AdjointGroup.hpp:13-19); SU(3) Im Tr(lambda_a M), the same projection with the
// Gell-Mann generators.
template <typename T> KLFT_D void adjoint(const Mat<1, T> &M, T *v) { v[0] = M.e[0][0].im; }
template <typename T> KLFT_D void adjoint(const Mat<2, T> &M, T *v) {
  v[0] = T(2) * M.e[0][1].im;
  v[1] = T(2) * M.e[0][1].re;
  v[2] = T(2) * M.e[0][0].im;
}
template <typename T> KLFT_D void adjoint(const Mat<3, T> &M, T *v) {
  const T r3 = T(1) / sqrt(T(3));
  v[0] = M.e[1][0].im + M.e[0][1].im;            // lambda_1
  v[1] = -M.e[1][0].re + M.e[0][1].re;           // lambda_2
  v[2] = M.e[0][0].im - M.e[1][1].im;            // lambda_3
  v[3] = M.e[2][0].im + M.e[0][2].im;            // lambda_4
  v[4] = -M.e[2][0].re + M.e[0][2].re;           // lambda_5
  v[5] = M.e[2][1].im + M.e[1][2].im;            // lambda_6
  v[6] = -M.e[2][1].re + M.e[1][2].re;           // lambda_7
  v[7] = (M.e[0][0].im + M.e[1][1].im - T(2) * M.e[2][2].im) * r3;  // lambda_8
}

// exp map U <- exp(t P) U: U(1) e^{i t p} (AdjointGroup.hpp:170-173); SU(2)
// cos|a| + i sin|a| n.sigma, a = t p (AdjointGroup.hpp:98-105, with exp(0) = 1);
// SU(3) exp(i t sum_a p_a lambda_a).
template <typename T> KLFT_D Mat<1, T> expmap(const T *p, T t, const Mat<1, T> *) {
  Mat<1, T> m;
  m.e[0][0] = mk<T>(cos(t * p[0]), sin(t * p[0]));
  return m;
}
template <typename T> KLFT_D Mat<2, T> expmap(const T *p, T t, const Mat<2, T> *) {
  const T a0 = t * p[0], a1 = t * p[1], a2 = t * p[2];
  const T alpha = sqrt(a0 * a0 + a1 * a1 + a2 * a2);
  if (alpha == T(0)) return mident<2, T>();
  const T n0 = a0 / alpha, n1 = a1 / alpha, n2 = a2 / alpha;
  const T sa = sin(alpha), ca = cos(alpha);
  Mat<2, T> m;
  m.e[0][0] = mk<T>(ca, n2 * sa);
  m.e[0][1] = mk<T>(n1 * sa, n0 * sa);
  m.e[1][0] = mk<T>(-n1 * sa, n0 * sa);
  m.e[1][1] = mk<T>(ca, -n2 * sa);
  return m;
}
template <typename T> KLFT_D Mat<3, T> expmap(const T *p, T t, const Mat<3, T> *) {
  const XMat<T> x = expi_gellmann<T>(p, t);
  Mat<3, T> m;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) m.e[i][j] = mk<T>(x.re[i][j], x.im[i][j]);
  return m;
}

}  // namespace klft
