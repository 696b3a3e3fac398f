// FP64 Mie coefficients a_n, b_n of a homogeneous sphere, with forward-mode
// tangents with respect to the sphere radius a_p and index n_p.
//
// Algorithm of theory/Sphere.py:147-226 (Sphere.mie_coefficients): zero-start
// downward recurrence of the logarithmic derivative D1 inside the sphere
// (z = m x, :190-198) and in the medium (z = x, :201-204), upward recurrence of
// psi, zeta, psi*zeta and D3 (:207-214), then Eqs. (5) and (6) of Pena & Pal
// (2009) (:217-224).  n_max follows Sphere.wiscombe_yang (:91-123).
//
// The tangents propagate d/dz through the inside recurrence and d/dx through
// the medium recurrences.  a_n(x, m) is holomorphic in m, so
//   d/da_p = k d/dx,  d/dn_p = (1/n_m) d/dm,  d/dk_p = (i/n_m) d/dm = i d/dn_p.
// n_max is treated as locally constant, as the reference's JAX Jacobian does
// (theory/jaxLorenzMie.py:354-361).
//
// Homogeneous spheres run linear forms of the two upward and of the inside's
// recurrence, which have no reciprocal on their serial chains and leave the
// quotients to the lanes: mie_inside_waves steps q with
// D1_n = q_(n-1)/q_n - n/z, mie_psi and mie_zeta step psi and zeta
// from the medium's D1.  mie_d1_inside (for spheres whose q leaves FP64's
// range, |m| of a tenth at hundreds of orders) and mie_upward (for layered
// spheres, whose layers take longer than it beside them) step the
// logarithmic derivatives themselves.
#pragma once

#include "lmb_math.cuh"

namespace lmb {

typedef cplx<double> zd;

// Number of partial waves, theory/Sphere.py:110-123.  For a scalar size
// parameter np.roll(x, -1) is x itself, so n_stop = max(n_s, |x m|).
LMB_HD int wiscombe_yang(double x, zd m) {
  double xl = fabs(x);
  double ns;
  if (xl <= 8.)
    ns = floor(xl + 4. * cbrt(xl) + 1.);
  else if (xl <= 4200.)
    ns = floor(xl + 4.05 * cbrt(xl) + 2.);
  else
    ns = floor(xl + 4. * cbrt(xl) + 2.);
  double xm = hypot(x * m.re, x * m.im);
  double nstop = ns > xm ? ns : xm;
  return (int)nstop;
}

struct MieScalars {
  double k;    // wave number in the medium, rad/um (Sphere.py:174-175)
  double x;    // size parameter k a_p
  double n_m;  // medium index (real part)
  zd m;        // relative index (n_p + i k_p)/n_m
  int nmax;
};

LMB_HD MieScalars mie_setup(double a_p, double n_p, double k_p, double n_m,
                            double wavelength) {
  MieScalars s;
  double k = 2. * 3.141592653589793 / wavelength;
  k *= n_m;
  s.k = k;
  s.x = k * a_p;
  s.n_m = n_m;
  s.m = mk(n_p / n_m, k_p / n_m);
  s.nmax = wiscombe_yang(s.x, s.m);
  return s;
}


// Per-order quotients of the recurrences for order n (1 <= n <= nmax), off
// the recurrences' chains, so that a warp forms them in parallel: inside,
// nz = n/z and nz2 = n/z^2 with z = m x.
LMB_HD void mie_orders_inside(const MieScalars& s, int n, zd* nz, zd* nz2) {
  const zd z = s.x * s.m;
  const zd z2 = z * z;
  nz[n] = double(n) / z;
  nz2[n] = double(n) / z2;
}

// The medium's: nx = n/x, nx2 = n/x^2.
LMB_HD void mie_orders_medium(const MieScalars& s, int n, double* nx,
                              double* nx2) {
  nx[n] = double(n) / s.x;
  nx2[n] = nx[n] / s.x;
}

// D1(x) in the medium (real because x is real), with dD1/dx.
LMB_HD void mie_d1_medium(const MieScalars& s, const double* nx,
                          const double* nx2, double* d1, double* d1x) {
  double d = 0., dx = 0.;
  d1[s.nmax] = d;
  d1x[s.nmax] = dx;
  for (int n = s.nmax; n > 0; --n) {
    const double inv = rcp_d(d + nx[n]);
    const double dw = dx - nx2[n];
    d = nx[n] - inv;
    dx = inv * inv * dw - nx2[n];
    d1[n - 1] = d;
    d1x[n - 1] = dx;
  }
}

// D1(m x) inside the sphere, with dD1/dz at z = m x: the zero-start
// downward recurrence from n_max (Sphere.py), complex.
LMB_HD void mie_d1_inside(const MieScalars& s, const zd* nz, const zd* nz2,
                          zd* d1in, zd* d1inz) {
  zd d = mk(0., 0.), dz = mk(0., 0.);
  d1in[s.nmax] = d;
  d1inz[s.nmax] = dz;
  for (int n = s.nmax; n > 0; --n) {
    const zd inv = recip(d + nz[n]);
    const zd dw = dz - nz2[n];
    d = nz[n] - inv;
    dz = (inv * inv) * dw - nz2[n];
    d1in[n - 1] = d;
    d1inz[n - 1] = dz;
  }
}

// Upward psi (real), zeta, with d/dx; needs the medium D1.
LMB_HD void mie_upward(const MieScalars& s, const double* nxs,
                       const double* nx2s, const double* d1, const double* d1x,
                       double* psi, double* psix, zd* zeta, zd* zetax) {
  const double x = s.x;
  double sx, cx;
#if defined(__CUDA_ARCH__)
  sincos(x, &sx, &cx);
#else
  sx = sin(x);
  cx = cos(x);
#endif
  const zd e1 = mk(cx, sx);           // e^{ix}
  const zd e2 = e1 * e1;              // e^{2ix}
  double p = sx, px = cx;             // psi_0, d/dx
  zd zt = mk(sx, -cx), ztx = e1;      // zeta_0 = -i e^{ix}, d/dx = e^{ix}
  zd pz = 0.5 * (1. - e2);            // psi*zeta, Eq. (18a)
  zd pzx = mk(e2.im, -e2.re);         // d/dx = -i e^{2ix}
  zd d3 = mk(0., 1.), d3x = mk(0., 0.);
  psi[0] = p;
  psix[0] = px;
  zeta[0] = zt;
  zetax[0] = ztx;
  for (int n = 1; n <= s.nmax; ++n) {
    const double nx = nxs[n];
    const double nx2 = nx2s[n];
    const double t1 = nx - d1[n - 1];
    const double t1x = -nx2 - d1x[n - 1];
    const zd t3 = nx - d3;
    const zd t3x = (-nx2) - d3x;
    const double pn = p * t1;
    const double pnx = px * t1 + p * t1x;
    const zd zn = zt * t3;
    const zd znx = ztx * t3 + zt * t3x;
    const zd t13 = t1 * t3;
    const zd t13x = t1x * t3 + t1 * t3x;
    const zd pzn = pz * t13;
    const zd pznx = pzx * t13 + pz * t13x;
    const zd ipz = recip(pzn);
    d3 = d1[n] + mul_i(ipz);
    d3x = d1x[n] - mul_i(pznx * (ipz * ipz));
    p = pn;
    px = pnx;
    zt = zn;
    ztx = znx;
    pz = pzn;
    pzx = pznx;
    psi[n] = p;
    psix[n] = px;
    zeta[n] = zt;
    zetax[n] = ztx;
  }
}

// Start of the downward waves at n_max: they grow by up to the ratio of the
// waves at n_max and at the origin, which 2^-400 leaves room for.
#define LMB_MIE_START 3.872591914849318e-121

// Inside, q_n by q_(n-1) = ((2n+1)/z) q_n - q_(n+1) from q_(nmax+1) such
// that D1_nmax = 0; iz = 1/z.  One thread; two dependent fused multiply-adds
// an order.
LMB_HD void mie_inside_waves(int nmax, zd iz, zd* q) {
  zd q1 = mk(LMB_MIE_START, 0.);
  zd q0 = (double(nmax) * LMB_MIE_START) * iz;
  q[nmax] = q1;
  q[nmax - 1] = q0;
  double c = 2. * nmax - 1.;
  for (int n = nmax - 1; n > 0; --n, c -= 2.) {
    const double wr = c * iz.re, wi = c * iz.im;
    const zd t = mk(fma(wr, q0.re, fma(-wi, q0.im, -q1.re)),
                    fma(wr, q0.im, fma(wi, q0.re, -q1.im)));
    q1 = q0;
    q0 = t;
    q[n - 1] = t;
  }
}

// Order n's quotient r = q_n / q_(n-1) gives D1_(n-1) = n/z - r, and the
// tangent's recurrence dD1_(n-1) = r^2 dD1_n - (r^2 + 1) n/z^2 its
// coefficients rr[n] and d1inz[n-1].
LMB_HD void mie_inside_order(int n, zd iz, const zd* q, zd* d1in, zd* rr,
                             zd* d1inz) {
  const zd r = q[n] * recip(q[n - 1]);
  d1in[n - 1] = double(n) * iz - r;
  if (rr == 0) return;
  const zd r2 = r * r;
  const zd nz2 = double(n) * (iz * iz);
  rr[n] = r2;
  d1inz[n - 1] = -1. * ((r2 + 1.) * nz2);
}

// The tangent's recurrence, in place over d1inz.  One thread.
LMB_HD void mie_inside_tangent(int nmax, const zd* rr, zd* d1inz) {
  zd d = mk(0., 0.);
  d1inz[nmax] = d;
  for (int n = nmax; n > 0; --n) {
    const zd r2 = rr[n], e = d1inz[n - 1];
    d = mk(fma(r2.re, d.re, fma(-r2.im, d.im, e.re)),
           fma(r2.re, d.im, fma(r2.im, d.re, e.im)));
    d1inz[n - 1] = d;
  }
}

// psi's factors psi_n / psi_(n-1) = n/x - D1_(n-1) and their d/dx, in place
// over nx, nx2.
LMB_HD void mie_psi_order(int n, const double* d1, const double* d1x,
                          double* nx, double* nx2) {
  nx[n] = nx[n] - d1[n - 1];
  nx2[n] = -nx2[n] - d1x[n - 1];
}

// psi_n and d/dx from its factors t, tx.  One thread; one dependent multiply
// (psi) and fused multiply-add (psix) an order.
LMB_HD void mie_psi(int nmax, double sx, double cx, const double* t,
                    const double* tx, double* psi, double* psix) {
  double p = sx, px = cx;
  psi[0] = p;
  psix[0] = px;
  for (int n = 1; n <= nmax; ++n) {
    px = fma(px, t[n], p * tx[n]);
    p = p * t[n];
    psi[n] = p;
    psix[n] = px;
  }
}

// 1/psi_n and its negative d/dx.
LMB_HD void mie_psi_inverse(int n, const double* psi, const double* psix,
                            double* ip, double* ipx) {
  const double i = rcp_d(psi[n]);
  ip[n] = i;
  ipx[n] = (psix[n] * i) * i;
}

// One part (0: real, 1: imaginary) of zeta_n and its d/dx, z, zx at stride
// 2.  With D3_n = D1_n + i/(psi_n zeta_n) the reference's step
// zeta_(n+1) = zeta_n ((n+1)/x - D3_n) is zeta_n psi_(n+1)/psi_n - i/psi_n
// for n >= 1, so each part is a real recurrence with one dependent fused
// multiply-add an order; zeta_1 comes from D3_0 = i.
LMB_HD void mie_zeta(int nmax, int part, double x, double sx, double cx,
                     const double* t, const double* tx, const double* ip,
                     const double* ipx, double* z, double* zx) {
  const double ix = 1. / x, k = part ? 1. : 0.;
  // zeta_0 = (sx, -cx) and its d/dx (cx, sx), times 1/x - i
  const double a0 = part ? -cx : sx, b0 = part ? sx : cx;
  const double ao = part ? -sx : -cx, bo = part ? -cx : sx;
  double z0 = fma(a0, ix, ao), x0 = b0 * ix + bo - a0 * (ix * ix);
  z[0] = a0;
  zx[0] = b0;
  z[2] = z0;
  zx[2] = x0;
  for (int n = 1; n < nmax; ++n) {
    x0 = fma(t[n + 1], x0, fma(tx[n + 1], z0, k * ipx[n]));
    z0 = fma(t[n + 1], z0, -(k * ip[n]));
    z[2 * (n + 1)] = z0;
    zx[2 * (n + 1)] = x0;
  }
}

// a_n (which = 0) or b_n (which = 1) for 1 <= n <= nmax, and if dout != 0
// its d/da_p and d/dn_p at dout[0] and dout[2].  Eqs. (5) and (6) differ in
// the factor of D1 alone: 1/m or m.
LMB_HD zd mie_coefficient_one(const MieScalars& s, int n, int which,
                              const zd* d1in, const zd* d1inz,
                              const double* psi, const double* psix,
                              const zd* zeta, const zd* zetax, zd* dout) {
  const double x = s.x;
  const zd m = s.m;
  const double nx = double(n) / x;
  const zd im = recip(m);
  const zd mu = which ? m : im;
  const zd ha = d1in[n];
  const double ps = psi[n], ps1 = psi[n - 1];
  const zd ze = zeta[n], ze1 = zeta[n - 1];
  const zd f = ha * mu + nx;
  const zd idn = recip(f * ze - ze1);
  const zd v = (f * ps - ps1) * idn;
  if (dout == 0) return v;
  const double nx2 = nx / x;
  const zd hz = d1inz[n];
  const double psx = psix[n], ps1x = psix[n - 1];
  const zd zex = zetax[n], ze1x = zetax[n - 1];
  const zd nu = which ? mk(1., 0.) : -1. * (im * im);  // d mu / dm
  const zd f_x = (m * hz) * mu - nx2;
  const zd f_m = (x * hz) * mu + ha * nu;
  const zd v_x = ((f_x * ps + f * psx - ps1x) - v * (f_x * ze + f * zex - ze1x)) * idn;
  const zd v_m = (f_m * ps - v * (f_m * ze)) * idn;
  dout[0] = s.k * v_x;
  dout[2] = (1. / s.n_m) * v_m;
  return v;
}

}  // namespace lmb
