// Device potentials of the synthetic interactions (inline, shared by the kernels).
#pragma once

#include "common.cuh"
#include "devlayout.hpp"
#include "kernels.hpp"

namespace ccx {

namespace pot {
constexpr double kPi = 3.14159265358979;
constexpr double kHbarc = 197.326968;

__device__ inline double pauli_dot(int m1, int m2, int m3, int m4) {
  if (m1 == m3 && m2 == m4) return (double)(m1 * m2);
  if (m1 == m4 && m2 == m3 && m1 != m2) return 2.0;
  return 0.0;
}
__device__ inline double kd(int a, int b) { return a == b ? 1.0 : 0.0; }

// vmom_minnesota, chiral_module_andreas_with_delta.f90:8980-9111, at squared momentum
// transfer q2 and the spin and isospin factors delta_m, delta_t, sigma.sigma, tau.tau
__device__ inline double minnesota_at(const DevPotential &P, double q2, double dm, double dt, double ss, double tt,
                                      double volume) {
  double v0r, v0t, v0s, kr, kt, ks;
  if (P.f32_literals) {
    v0r = (double)200.0f; v0t = (double)178.0f; v0s = (double)91.85f;
    kr = (double)1.487f; kt = (double)0.639f; ks = (double)0.465f;
  } else {
    v0r = 200.0; v0t = 178.0; v0s = 91.85; kr = 1.487; kt = 0.639; ks = 0.465;
  }
  const double pi15 = kPi * sqrt(kPi);  // x^1.5 as x sqrt(x): no pow on the FP64 pipe
  double vr = v0r * pi15 * exp(-q2 / (4.0 * kr)) / (kr * sqrt(kr));
  double vt = -v0t * pi15 * exp(-q2 / (4.0 * kt)) / (kt * sqrt(kt));
  double vs = -v0s * pi15 * exp(-q2 / (4.0 * ks)) / (ks * sqrt(ks));
  vr = vr * (3.0 * dm * dt - tt * dm - ss * dt - tt * ss) / 8.0;
  vs = vs * (3.0 * dm * dt + tt * dm - 3.0 * ss * dt - tt * ss) / 16.0;
  vt = vt * (3.0 * dm * dt - 3.0 * tt * dm + ss * dt - tt * ss) / 16.0;
  return ((vs + vr) + vt) / volume;
}
__device__ inline double minnesota(const DevOrbits &O, const DevPotential &P, int p, int q, int r, int s) {
  if (O.nx[p] + O.nx[q] != O.nx[r] + O.nx[s] || O.ny[p] + O.ny[q] != O.ny[r] + O.ny[s] ||
      O.nz[p] + O.nz[q] != O.nz[r] + O.nz[s] || O.tz[p] + O.tz[q] != O.tz[r] + O.tz[s])
    return 0.0;
  const double q0 = 0.5 * (O.kx[p] - O.kx[q]) - 0.5 * (O.kx[r] - O.kx[s]);
  const double q1 = 0.5 * (O.ky[p] - O.ky[q]) - 0.5 * (O.ky[r] - O.ky[s]);
  const double q2v = 0.5 * (O.kz[p] - O.kz[q]) - 0.5 * (O.kz[r] - O.kz[s]);
  const double q2 = (q0 * q0 + q1 * q1) + q2v * q2v;
  const int m1 = O.sz[p], m2 = O.sz[q], m3 = O.sz[r], m4 = O.sz[s];
  const int t1 = O.tz[p], t2 = O.tz[q], t3 = O.tz[r], t4 = O.tz[s];
  const double dm = kd(m1, m3) * kd(m2, m4), dt = kd(t1, t3) * kd(t2, t4);
  return minnesota_at(P, q2, dm, dt, pauli_dot(m1, m2, m3, m4), pauli_dot(t1, t2, t3, t4), O.volume);
}

constexpr double kLambda6 = 8.303765625e15;  // (450 MeV)^6 of the regulator exp(-(p/450)^6)

// nucleon mass of a pair's isospin projection (the relativity factor's mass)
__device__ inline double pair_mass(int t1, int t2) {
  const int tsum = (t1 + t2) / 2;
  return tsum < 0 ? 9.38272046000000046e+02 : (tsum == 0 ? 9.38918267117927371e+02 : 9.39565379000000007e+02);
}

__device__ inline cplx wsig(int ma, int mb, const double w[3]) {
  const int ia = ma > 0 ? 0 : 1, ib = mb > 0 ? 0 : 1;
  if (ia == 0 && ib == 0) return cplx(w[2], 0.0);
  if (ia == 1 && ib == 1) return cplx(-w[2], 0.0);
  if (ia == 0) return cplx(w[0], -w[1]);
  return cplx(w[0], w[1]);
}

// OPE + LO/NLO contacts in the operator form of chiral_pot (:5879-6301), regulated
// by freg (:3336-3351, n=3, Lambda=450 MeV), times hbarc^3/volume
__device__ inline cplx chiral_like(const DevOrbits &O, const DevPotential &P, int p, int q, int r, int s) {
  if (O.nx[p] + O.nx[q] != O.nx[r] + O.nx[s] || O.ny[p] + O.ny[q] != O.ny[r] + O.ny[s] ||
      O.nz[p] + O.nz[q] != O.nz[r] + O.nz[s] || O.tz[p] + O.tz[q] != O.tz[r] + O.tz[s])
    return cplx(0.0, 0.0);
  const double k1[3] = {O.kx[p] * kHbarc, O.ky[p] * kHbarc, O.kz[p] * kHbarc};
  const double k2[3] = {O.kx[q] * kHbarc, O.ky[q] * kHbarc, O.kz[q] * kHbarc};
  const double k3[3] = {O.kx[r] * kHbarc, O.ky[r] * kHbarc, O.kz[r] * kHbarc};
  const double k4[3] = {O.kx[s] * kHbarc, O.ky[s] * kHbarc, O.kz[s] * kHbarc};
  double pr[3], pp[3], km[3], qt[3], qxk[3];
  for (int d = 0; d < 3; ++d) {
    pr[d] = 0.5 * (k1[d] - k2[d]);
    pp[d] = 0.5 * (k3[d] - k4[d]);
    km[d] = 0.5 * (pr[d] + pp[d]);
    qt[d] = pr[d] - pp[d];
  }
  const double p2 = (pr[0] * pr[0] + pr[1] * pr[1]) + pr[2] * pr[2];
  const double pp2 = (pp[0] * pp[0] + pp[1] * pp[1]) + pp[2] * pp[2];
  const double km2 = (km[0] * km[0] + km[1] * km[1]) + km[2] * km[2];
  const double q2 = (qt[0] * qt[0] + qt[1] * qt[1]) + qt[2] * qt[2];
  qxk[0] = qt[1] * km[2] - qt[2] * km[1];
  qxk[1] = qt[2] * km[0] - qt[0] * km[2];
  qxk[2] = qt[0] * km[1] - qt[1] * km[0];
  const int m1 = O.sz[p], m2 = O.sz[q], m3 = O.sz[r], m4 = O.sz[s];
  const int t1 = O.tz[p], t2 = O.tz[q], t3 = O.tz[r], t4 = O.tz[s];
  const int tsum = (t1 + t2) / 2;
  const double mn = tsum < 0 ? 9.38272046000000046e+02 : (tsum == 0 ? 9.38918267117927371e+02 : 9.39565379000000007e+02);
  const double rel = mn / sqrt(sqrt((mn * mn + p2) * (mn * mn + pp2)));
  const double dm = kd(m1, m3) * kd(m2, m4), dt = kd(t1, t3) * kd(t2, t4);
  const double tt = pauli_dot(t1, t2, t3, t4), ss = pauli_dot(m1, m2, m3, m4);
  const cplx sq = wsig(m1, m3, qt) * wsig(m2, m4, qt);
  const cplx sk = wsig(m1, m3, km) * wsig(m2, m4, km);
  const cplx mi(0.0, -0.5);
  const cplx sl = mi * wsig(m1, m3, qxk) * kd(m2, m4) + mi * wsig(m2, m4, qxk) * kd(m1, m3);
  const double c2 = (1.27 * 1.27) / (4.0 * 92.4 * 92.4);
  const double ope = -1.0 * c2 / (q2 + 138.0 * 138.0);
  const cplx vlo = (ope * tt) * sq;
  const double *c = P.lec;
  const cplx cont_lo = cplx(c[0] * dm * dt + c[1] * ss * dt, 0.0);
  const cplx cont_nlo = cplx(c[2] * q2 * dm * dt + c[3] * km2 * dm * dt + c[4] * q2 * ss * dt + c[5] * km2 * ss * dt, 0.0) +
                        (c[6] * dt) * sl + (c[7] * dt) * sq + (c[8] * dt) * sk;
  const double l2n = kLambda6;
  const double freg = exp(-((p2 * p2) * p2 / l2n + (pp2 * pp2) * pp2 / l2n));
  const cplx vdir = ((vlo + cont_lo) + cont_nlo) * (rel * freg);
  return (kHbarc * kHbarc * kHbarc) * vdir * (1.0 / O.volume);
}

// The chiral-like element factorised as m F(pq) F(rs) core(p, q, r, s): the relativity
// factor m / ((m^2 + p^2)(m^2 + p'^2))^(1/4) and the regulator exp(-(p^6 + p'^6)/L^6)
// depend on the relative momentum of one pair each, and both are unchanged when r and s
// swap, so an antisymmetrised element is m F(pq) F(rs) (core(pqrs) - core(pqsr)).
// F(pq) is evaluated once per pair; the core per element holds no transcendental.
__device__ inline double chiral_pair_factor(const DevOrbits &O, int p, int q) {
  const double x = 0.5 * (O.kx[p] * kHbarc - O.kx[q] * kHbarc), y = 0.5 * (O.ky[p] * kHbarc - O.ky[q] * kHbarc);
  const double z = 0.5 * (O.kz[p] * kHbarc - O.kz[q] * kHbarc);
  const double p2 = (x * x + y * y) + z * z;
  const double mn = pair_mass(O.tz[p], O.tz[q]);
  return exp(-(p2 * p2) * p2 / kLambda6) / sqrt(sqrt(mn * mn + p2));
}
__device__ inline cplx chiral_core(const DevOrbits &O, const DevPotential &P, int p, int q, int r, int s) {
  if (O.nx[p] + O.nx[q] != O.nx[r] + O.nx[s] || O.ny[p] + O.ny[q] != O.ny[r] + O.ny[s] ||
      O.nz[p] + O.nz[q] != O.nz[r] + O.nz[s] || O.tz[p] + O.tz[q] != O.tz[r] + O.tz[s])
    return cplx(0.0, 0.0);
  double pr[3], pp[3], km[3], qt[3], qxk[3];
  const double k1[3] = {O.kx[p], O.ky[p], O.kz[p]}, k2[3] = {O.kx[q], O.ky[q], O.kz[q]};
  const double k3[3] = {O.kx[r], O.ky[r], O.kz[r]}, k4[3] = {O.kx[s], O.ky[s], O.kz[s]};
  for (int d = 0; d < 3; ++d) {
    pr[d] = 0.5 * (k1[d] * kHbarc - k2[d] * kHbarc);
    pp[d] = 0.5 * (k3[d] * kHbarc - k4[d] * kHbarc);
    km[d] = 0.5 * (pr[d] + pp[d]);
    qt[d] = pr[d] - pp[d];
  }
  const double km2 = (km[0] * km[0] + km[1] * km[1]) + km[2] * km[2];
  const double q2 = (qt[0] * qt[0] + qt[1] * qt[1]) + qt[2] * qt[2];
  qxk[0] = qt[1] * km[2] - qt[2] * km[1];
  qxk[1] = qt[2] * km[0] - qt[0] * km[2];
  qxk[2] = qt[0] * km[1] - qt[1] * km[0];
  const int m1 = O.sz[p], m2 = O.sz[q], m3 = O.sz[r], m4 = O.sz[s];
  const int t1 = O.tz[p], t2 = O.tz[q], t3 = O.tz[r], t4 = O.tz[s];
  const double dm = kd(m1, m3) * kd(m2, m4), dt = kd(t1, t3) * kd(t2, t4);
  const double tt = pauli_dot(t1, t2, t3, t4), ss = pauli_dot(m1, m2, m3, m4);
  const cplx sq = wsig(m1, m3, qt) * wsig(m2, m4, qt);
  const cplx sk = wsig(m1, m3, km) * wsig(m2, m4, km);
  const cplx mi(0.0, -0.5);
  const cplx sl = mi * wsig(m1, m3, qxk) * kd(m2, m4) + mi * wsig(m2, m4, qxk) * kd(m1, m3);
  const double c2 = (1.27 * 1.27) / (4.0 * 92.4 * 92.4);
  const double ope = -1.0 * c2 / (q2 + 138.0 * 138.0);
  const cplx vlo = (ope * tt) * sq;
  const double *c = P.lec;
  const cplx cont_lo = cplx(c[0] * dm * dt + c[1] * ss * dt, 0.0);
  const cplx cont_nlo = cplx(c[2] * q2 * dm * dt + c[3] * km2 * dm * dt + c[4] * q2 * ss * dt + c[5] * km2 * ss * dt, 0.0) +
                        (c[6] * dt) * sl + (c[7] * dt) * sq + (c[8] * dt) * sk;
  return (kHbarc * kHbarc * kHbarc) * ((vlo + cont_lo) + cont_nlo) * (1.0 / O.volume);
}
// antisymmetrised chiral-like element from the pair factors fpq = F(pq), frs = F(rs)
__device__ inline cplx chiral_anti_factored(const DevOrbits &O, const DevPotential &P, int p, int q, int r, int s,
                                            double fpq, double frs) {
  const double w = pair_mass(O.tz[p], O.tz[q]) * fpq * frs;
  return (chiral_core(O, P, p, q, r, s) - chiral_core(O, P, p, q, s, r)) * w;
}

// ---- elements on a momentum lattice -------------------------------------------------
// Both potentials depend on the relative momenta of the two pairs only, and on a lattice
// those are integers times step: with D = n_p - n_r and E = n_p - n_s (p + q = r + s), the
// momentum transfer is q = step D and the mean relative momentum k = step E / 2, and the
// exchange term swaps D and E.  Everything transcendental and every division is then a
// table over |D|^2 or |n_p - n_q|^2 (at most 12 nmax^2 + 1 entries), and the spin structure
// is integer arithmetic: a real element takes one FP64 operation (a subtraction of two table
// entries), a complex one about twenty, against two hundred with the momenta themselves.
// That is what counts: the FP64 pipe retires two operations a clock on an SM, and generating
// a block was bound by it.  Whole interaction, MP2 start and amplitudes to the host: PNM 66
// nmax=4 Minnesota 52.8 to 2.2 ms; SNM 132 nmax=3 chiral-like 51.4 to 9.7 ms.
// A pair class: 1 and 2 same projections on both sides, aligned and opposed; 3 swapped; 0
// neither.  (delta, sigma1.sigma2) = (1, 1), (1, -1), (0, 2), (0, 0).
__host__ __device__ inline int pair_class(int m1, int m2, int m3, int m4) {
  if (m1 == m3 && m2 == m4) return m1 == m2 ? 1 : 2;
  return (m1 != m2 && m1 == m4 && m2 == m3) ? 3 : 0;
}
__device__ inline double class_delta(int c) { return c == 1 || c == 2 ? 1.0 : 0.0; }
__device__ inline double class_dot(int c) { return c == 1 ? 1.0 : c == 2 ? -1.0 : c == 3 ? 2.0 : 0.0; }

// Table rows of O.nq2 doubles.  Minnesota: row 4 cs + ct, the element of spin class cs and
// isospin class ct.  Chiral-like: rows ct the coefficient of the tensor sigma1.D sigma2.D,
// 4 + cs and 8 + cs the scalar terms in |D|^2 and |E|^2, 12 + (tz sum + 1) the pair factor.
constexpr int kLatRowsMinnesota = 16, kLatRowsChiral = 15;

template <typename S> __device__ S lat_anti(const DevPotential &P, int nq2, double step, int2 p, int2 q, int2 r, int2 s);
__device__ __forceinline__ int lat_norm2(unsigned d) { return __dp4a((int)d, (int)d, 0); }
__device__ __forceinline__ double lat_minnesota(const DevPotential &P, int nq2, int2 p, int2 q, int2 r, int2 s) {
  const int m1 = p.y & 1, m2 = q.y & 1, m3 = r.y & 1, m4 = s.y & 1;
  const int t1 = p.y >> 1, t2 = q.y >> 1, t3 = r.y >> 1, t4 = s.y >> 1;
  const int cd = 4 * pair_class(m1, m2, m3, m4) + pair_class(t1, t2, t3, t4);
  const int ce = 4 * pair_class(m1, m2, m4, m3) + pair_class(t1, t2, t4, t3);
  return P.lat[cd * nq2 + lat_norm2(__vsub4((unsigned)p.x, (unsigned)r.x))] -
         P.lat[ce * nq2 + lat_norm2(__vsub4((unsigned)p.x, (unsigned)s.x))];
}
template <> __device__ __forceinline__ double lat_anti<double>(const DevPotential &P, int nq2, double, int2 p, int2 q,
                                                               int2 r, int2 s) {
  return lat_minnesota(P, nq2, p, q, r, s);
}

struct Int3 {
  int x, y, z;
};
__device__ __forceinline__ Int3 lat_vec(unsigned d) {  // the signed low bytes
  return Int3{(int)(d << 24) >> 24, (int)(d << 16) >> 24, (int)(d << 8) >> 24};
}
// <a| sigma.v |b> for spin bits a, b, an integer complex number
__device__ __forceinline__ int2 lat_sigma(Int3 v, int a, int b) {
  return a == b ? make_int2(a ? v.z : -v.z, 0) : make_int2(v.x, a ? -v.y : v.y);
}
__device__ __forceinline__ int2 lat_mul(int2 a, int2 b) { return make_int2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
// a small integer as FP64, exactly: to FP32 and then widened by integer operations (the
// 64-bit conversions run on the FP64 pipe)
__device__ __forceinline__ double lat_f64(int i) {
  const unsigned u = __float_as_uint((float)i);
  const unsigned hi = (u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u);
  return i == 0 ? 0.0 : __hiloint2double((int)hi, (int)(u << 29));
}
// acc += sg * core / ((hbar c)^3 / volume) of the direct term (sg 1) or the exchange term
// (sg -1, with r and s, and D and E, swapped); X = D x E
__device__ __forceinline__ void lat_core(const DevPotential &P, int nq2, double u2, double sg, Int3 D, Int3 E, Int3 X,
                                         int d2, int e2, int m1, int m2, int m3, int m4, int ct, double &re, double &im) {
  const double *T = P.lat;
  const int2 zd = lat_mul(lat_sigma(D, m1, m3), lat_sigma(D, m2, m4));
  const double t = sg * T[ct * nq2 + d2];
  re = fma(t, lat_f64(zd.x), re);
  im = fma(t, lat_f64(zd.y), im);
  if (ct == 3) return;  // the contact terms are diagonal in isospin
  const int cs = pair_class(m1, m2, m3, m4);
  if (cs) re = fma(sg, T[(4 + cs) * nq2 + d2] + T[(8 + cs) * nq2 + e2], re);
  const int2 ze = lat_mul(lat_sigma(E, m1, m3), lat_sigma(E, m2, m4));
  const double ck = sg * (P.lec[8] * u2), cl = sg * (P.lec[6] * u2);
  re = fma(ck, lat_f64(ze.x), re);
  im = fma(ck, lat_f64(ze.y), im);
  int2 l = make_int2(0, 0);
  if (m2 == m4) { const int2 w = lat_sigma(X, m1, m3); l.x += w.x; l.y += w.y; }
  if (m1 == m3) { const int2 w = lat_sigma(X, m2, m4); l.x += w.x; l.y += w.y; }
  re = fma(cl, lat_f64(l.y), re);
  im = fma(-cl, lat_f64(l.x), im);
}
template <> __device__ __forceinline__ cplx lat_anti<cplx>(const DevPotential &P, int nq2, double step, int2 p, int2 q,
                                                           int2 r, int2 s) {
  if (P.kind != 1) return cplx(lat_minnesota(P, nq2, p, q, r, s), 0.0);
  const unsigned d = __vsub4((unsigned)p.x, (unsigned)r.x), e = __vsub4((unsigned)p.x, (unsigned)s.x);
  const Int3 D = lat_vec(d), E = lat_vec(e);
  const int d2 = lat_norm2(d), e2 = lat_norm2(e);
  const Int3 X{D.y * E.z - D.z * E.y, D.z * E.x - D.x * E.z, D.x * E.y - D.y * E.x};
  const int m1 = p.y & 1, m2 = q.y & 1, m3 = r.y & 1, m4 = s.y & 1;
  const int t1 = p.y >> 1, t2 = q.y >> 1, t3 = r.y >> 1, t4 = s.y >> 1;
  const double u = 0.5 * step * kHbarc, u2 = u * u;
  double re = 0.0, im = 0.0;
  lat_core(P, nq2, u2, 1.0, D, E, X, d2, e2, m1, m2, m3, m4, pair_class(t1, t2, t3, t4), re, im);
  lat_core(P, nq2, u2, -1.0, E, D, Int3{-X.x, -X.y, -X.z}, e2, d2, m1, m2, m4, m3, pair_class(t1, t2, t4, t3), re, im);
  const double *F = P.lat + (12 + t1 + t2) * nq2;
  const double w = F[lat_norm2(__vsub4((unsigned)p.x, (unsigned)q.x))] * F[lat_norm2(__vsub4((unsigned)r.x, (unsigned)s.x))];
  return cplx(re * w, im * w);
}

template <typename S> __device__ S vbare(const DevOrbits &O, const DevPotential &P, int p, int q, int r, int s);
template <> __device__ inline double vbare<double>(const DevOrbits &O, const DevPotential &P, int p, int q, int r, int s) {
  return minnesota(O, P, p, q, r, s);
}
template <> __device__ inline cplx vbare<cplx>(const DevOrbits &O, const DevPotential &P, int p, int q, int r, int s) {
  if (P.kind == 1) return chiral_like(O, P, p, q, r, s);
  return cplx(minnesota(O, P, p, q, r, s), 0.0);
}
template <typename S> __device__ inline S vanti(const DevOrbits &O, const DevPotential &P, int p, int q, int r, int s) {
  return vbare<S>(O, P, p, q, r, s) - vbare<S>(O, P, p, q, s, r);
}
// the antisymmetrised element of orbitals p, q, r, s of conserved momentum and isospin
template <typename S, bool LAT>
__device__ __forceinline__ S anti_of(const DevOrbits &O, const DevPotential &P, int p, int q, int r, int s) {
  if constexpr (LAT) return lat_anti<S>(P, O.nq2, O.step, O.lat[p], O.lat[q], O.lat[r], O.lat[s]);
  else return vanti<S>(O, P, p, q, r, s);
}
}  // namespace pot

}  // namespace ccx
