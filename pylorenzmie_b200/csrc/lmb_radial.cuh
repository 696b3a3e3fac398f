// Radial tables: the field of a sphere in a plane z = const.
//
// At the pixels of one plane, everything that theory/LorenzMie.py:183-342
// sums over the orders depends on the distance rho from the sphere's axis
// alone; the azimuth phi enters only through the projection:
//   E_x = U + V (x^2 - y^2),  E_y = V 2 x y,  E_z = Z x,
// with (x, y) the offset from the axis, U = (X1 + X2) / 2, V = (X1 - X2) /
// (2 rho^2), Z = Z1 / rho, X1 and X2 the x component at phi = 0 and phi = 90
// degrees and Z1 the z component at phi = 0, phase included.  So the orders are summed in FP64 at equidistant nodes of rho,
// a few per wavelength, and every pixel interpolates: a 1280x1024 frame
// needs ~2700 sums a sphere instead of 1.3 million.
//
// The field in a plane above the sphere is band-limited: its transverse
// wave numbers are at most k, plus evanescent waves that have decayed by
// e^{-kappa d} over the distance d from the sphere.  Hence the node spacing
// (RADIAL_SPACING below) and the distances of radial_clear.
// U, V and Z are even in rho, which gives the nodes at rho < 0.
//
// From the nodes each interval of one spacing around node i gets the
// polynomial of degree RADIAL_COEFS - 1 that interpolates, at the Chebyshev
// points of the interval, the Lagrange interpolant through the RADIAL_TAPS
// nodes around i.
#pragma once

#include "lmb_records.cuh"

namespace lmb {

enum {
  RADIAL_TAPS = 17,
  RADIAL_SIDE = RADIAL_TAPS / 2,
  RADIAL_COEFS = 6,
  RADIAL_FUNCS = 6,  // U, V, Z as (re, im)
  // Floats per interval: 9 float4, an odd number, so that eight neighbouring
  // intervals fall into different shared-memory banks.
  RADIAL_REC = RADIAL_FUNCS * RADIAL_COEFS
};

// Node spacing and interval width in radians (k times pixels).  At the band
// limit the 17-point interpolant is then off by at most 1e-9 (at 1 radian by
// 2e-6), and the degree-5 polynomial by 2 (0.6 / 4)^6 / 6! = 3e-8: below the
// FP32 rounding of its coefficients.  Measured against the oracle over radii
// of 0.4-24 um from 2 px above the sphere on.
#define RADIAL_SPACING 0.6
// The same for FP64 images: at half the spacing the 17-point interpolant is
// off by at most 1e-14, and a polynomial of degree 8 by 2 (0.3 / 4)^9 / 9! =
// 4e-16, of a component.
#define RADIAL_SPACING64 0.3
enum {
  RADIAL_COEFS64 = 9,
  RADIAL_REC64 = RADIAL_FUNCS * RADIAL_COEFS64  // doubles per interval: 27 double2, odd
};
// Where the tables apply: the plane's distance, times k, from the sphere's
// surface and from its centre.  The evanescent waves that reach the plane
// decay with the first; those of the lowest orders come from the centre, so
// that a small sphere's field a few px above it changes faster than the nodes
// can follow (at 1.8 from the surface a sphere of 0.02 um is off by 2e-4 of
// its largest component in FP32, 6e-7 in FP64), and so do the high orders of
// spheres of high index.  On the CPU build, radii 0.003-12 um, indices 0.1-4
// and 0.2 + 3i: from here on FP32 tables are off by at most 1.7e-7 and FP64
// ones by 4e-14 of the largest component, the rounding that they have
// anywhere; the fits' tables by 2e-7 of a column.
#define RADIAL_CLEARANCE 1.8
#define RADIAL_CLEARANCE64 5.5
#define RADIAL_CENTRE 13.

// dz: distance of the plane from the centre, a: radius (px).
LMB_HD bool radial_clear(double k, double dz, double a, bool fp64) {
  return k * dz >= RADIAL_CENTRE &&
         k * (dz - a) >= (fp64 ? RADIAL_CLEARANCE64 : RADIAL_CLEARANCE);
}

// The fits' distance (pixels) that stands for the axis itself, where D and its
// derivatives are limits: they are off by (k rho)^2 ~ 1e-8 of themselves there
// and the cancellation in D costs as much.
#define RADIAL_AXIS 1e-4
// The axis of FP32 images (radians): U, V and Z as (4 f(h) - f(2 h)) / 3, off
// by 4 h^4 = 6e-11 of a component and by 4e-11 from the cancellation in V.
// (FP64 tables take it from their neighbours, k_radial_table.)
#define RADIAL_AXIS_STEP 2e-3
// Interval width in pixels, a multiple of 1/64 so that i * width is exact
// in FP32; 0 if k is out of range.
inline double radial_spacing(double k, bool fp64) {
  const double r = fp64 ? RADIAL_SPACING64 : RADIAL_SPACING;
  const double w = fmin(floor(64. * r / k) / 64., 64.);
  return w >= 0.0625 ? w : 0.;
}

// Row c: the weights of the nodes in the coefficient of t^c, t = (rho - rho_i)
// / (half a spacing).
template <int NC = RADIAL_COEFS>
struct RadialMatrixN {
  double m[NC][RADIAL_TAPS];
};
typedef RadialMatrixN<> RadialMatrix;

// The Lagrange weights of the RADIAL_TAPS nodes around one of them at
// offset x (in spacings).
LMB_HD void radial_weights(double x, double* w) {
  // prod_{l != j} (x - l) / (j - l) by prefix and suffix products
  const double inv[RADIAL_TAPS] = {
      // 1 / ((-1)^(16-m) m! (16-m)!)
      1. / 20922789888000., -1. / 1307674368000., 1. / 174356582400.,
      -1. / 37362124800., 1. / 11496038400., -1. / 4790016000.,
      1. / 2612736000., -1. / 1828915200., 1. / 1625702400.,
      -1. / 1828915200., 1. / 2612736000., -1. / 4790016000.,
      1. / 11496038400., -1. / 37362124800., 1. / 174356582400.,
      -1. / 1307674368000., 1. / 20922789888000.};
  double p = 1.;
  for (int j = 0; j < RADIAL_TAPS; ++j) {
    w[j] = p * inv[j];
    p *= x - double(j - RADIAL_SIDE);
  }
  p = 1.;
  for (int j = RADIAL_TAPS - 1; j >= 0; --j) {
    w[j] *= p;
    p *= x - double(j - RADIAL_SIDE);
  }
}

// Coefficients in powers of t of the polynomial through values at the
// Chebyshev points t_i = cos(pi (i + 1/2) / NC): row c, column i.
template <int NC>
struct RadialPowers {
  double t[NC];
  double m[NC][NC];
  RadialPowers() {
    const double pi = 3.141592653589793;
    double tq[NC][NC] = {};  // T_q in powers
    tq[0][0] = tq[1][1] = 1.;
    for (int q = 2; q < NC; ++q)
      for (int p = 0; p < NC; ++p)
        tq[q][p] = (p ? 2. * tq[q - 1][p - 1] : 0.) - tq[q - 2][p];
    for (int i = 0; i < NC; ++i) {
      t[i] = cos(pi * (i + 0.5) / NC);
      for (int p = 0; p < NC; ++p) {
        m[p][i] = 0.;
        for (int q = 0; q < NC; ++q)
          m[p][i] += (q ? 2. : 1.) / NC * cos(pi * q * (i + 0.5) / NC) * tq[q][p];
      }
    }
  }
};

template <int NC = RADIAL_COEFS>
inline RadialMatrixN<NC> radial_matrix() {
  static const RadialPowers<NC> P;
  RadialMatrixN<NC> A = {};
  for (int i = 0; i < NC; ++i) {
    double w[RADIAL_TAPS];
    radial_weights(0.5 * P.t[i], w);
    for (int c = 0; c < NC; ++c)
      for (int j = 0; j < RADIAL_TAPS; ++j) A.m[c][j] += P.m[c][i] * w[j];
  }
  return A;
}

// U, V, Z (re, im each) at distance rho > 0 (pixels) from the axis of a
// particle at height zp, in the plane z; dzc = z - zp.  rec: order_record's
// FP64 records (2 Quads per order).  aberr: see aberration_wave.
LMB_HD void radial_field(double k, double rho, double dzc, double z, double zp,
                         bool bohren, double aberr, const Quad<double>* rec,
                         int nm, double* v) {
  const Geometry<double> g = geometry<double>(k, rho, 0., dzc, z, zp, bohren);
  const Sums<double> s = order_sum<double>(g, rec, nm);
  const double ikr = g.ikr;
  const zd e0 = (g.sint * ikr * ikr) * s.s0, e1 = ikr * s.s1, e2 = ikr * s.s2;
  zd ph = g.phase;
  if (aberr != 0.) {
    double d[3];
    ph = ph * conj(aberration_wave<double>(aberr, rho, 0., zp, d));
  }
  const zd x1 = ph * (g.sint * e0 + g.mu * e1);
  const zd x2 = -(ph * e2);
  const zd zz = ph * (g.mu * e0 - g.sint * e1);
  const double ir = 1. / rho, h = 0.5 * ir * ir;
  v[0] = 0.5 * (x1.re + x2.re);
  v[1] = 0.5 * (x1.im + x2.im);
  v[2] = h * (x1.re - x2.re);
  v[3] = h * (x1.im - x2.im);
  v[4] = ir * zz.re;
  v[5] = ir * zz.im;
}

// Distance of a pixel from the axis.  (X, Y): pixel minus particle rounded
// to 2^-10 px (exact in FP32 up to 8192 px), (a, b) the remainders; lx =
// X^2's rounding error plus 2 a X + a^2, ly alike.  rho = r0 + corr with an
// error of ~1e-7 of corr, i.e. far below the FP32 rounding of rho, which at
// 1500 px would turn the phase by 1e-4 rad; y is 1 / rho to a few ulp.
struct RadialDistance {
  f2 r0, corr, y;
};

// Quads and pairs as the kernels load them.
#if defined(__CUDACC__)
typedef float4 f4;
typedef double2 d2;
#else
struct f4 {
  float x, y, z, w;
};
struct d2 {
  double x, y;
};
#endif

LMB_HD int radial_round(float v) {
#if defined(__CUDA_ARCH__)
  return __float2int_rn(v);
#else
  return int(nearbyintf(v));
#endif
}

LMB_HD f2 pneg(f2 a) { return pk(-a.x, -a.y); }
LMB_HD f2 psub(f2 a, f2 b) { return pfma(pk(-1.f, -1.f), b, a); }

LMB_HD RadialDistance radial_distance(f2 px, f2 lx, f2 qy, f2 ly) {
  const f2 s = padd(px, qy);
  const f2 bb = psub(s, px);
  const f2 err = padd(psub(px, psub(s, bb)), psub(qy, bb));  // s + err exact
  const f2 low = padd(padd(lx, ly), err);
  const f2 sh = padd(s, low);
  const f2 sl = padd(psub(s, sh), low);
  const f2 y = pk(rsqrt_seed(fmaxf(sh.x, 1e-24f)), rsqrt_seed(fmaxf(sh.y, 1e-24f)));
  RadialDistance d;
  d.y = y;
  d.r0 = pmul(sh, y);
  const f2 e = padd(pfma(pneg(d.r0), d.r0, sh), sl);
  d.corr = pmul(pmul(pk(0.5f, 0.5f), y), e);
  return d;
}

// One complex function (re, im) at t: degree RADIAL_COEFS - 1.
LMB_HD f2 radial_eval(const f4* r, float t) {
  const f4 a = r[0], b = r[1], c = r[2];
  const f2 tt = pk(t, t);
  f2 v = pfma(pk(c.z, c.w), tt, pk(c.x, c.y));
  v = pfma(v, tt, pk(b.z, b.w));
  v = pfma(v, tt, pk(b.x, b.y));
  v = pfma(v, tt, pk(a.z, a.w));
  return pfma(v, tt, pk(a.x, a.y));
}

// The bound on an FP32 pixel's error from the tables.  A particle's field
//   E_x = U + c V,  E_y = s V,  E_z = x Z
// is off by at most RADIAL_FIELD_REL times |U| + |V| (|c| + |s|) + |x Z|, |.|
// the larger of the real and the imaginary part's: the coefficients, Horner's
// rule and c and s are rounded to FP32, and U may cancel against c V (behind
// a large sphere of high index, near its axis, both are up to a hundred times
// E).  The hologram is off by at most 2 sqrt(H) times the sum over the
// particles.  On the CPU build, over 2.4 million pixels of single spheres of
// 0.3-24 um, indices to 2.6, from 1.8 / k above the sphere on, the field is
// off by at most 2.4e-7 of that, an unmarked pixel's hologram by at most
// 7.2e-6.  1.8 |U|, what |E| comes to where U does not cancel, lowers the
// error of ordinary images further: 7.6e-8 for 8.3e-8 of the hologram over a
// batch of 128 images.  The largest error of 60 frames of 16 spheres is
// 1.45e-5 (9.3e-6 with the direct sums, whose own bound marks more; 5e-7 here
// leaves 8.9e-6, but the pixels summed again sit together and their tiles end
// late: 28 such frames 218-221 -> 228 us, one 234 -> 266).
#define RADIAL_FIELD_REL 4e-7f

LMB_HD float radial_bound(f2 u, f2 v, f2 w, float c, float s, float x) {
  const float mu = fmaxf(fabsf(u.x), fabsf(u.y));
  const float mv = fmaxf(fabsf(v.x), fabsf(v.y));
  const float mw = fmaxf(fabsf(w.x), fabsf(w.y));
  return fmaxf(1.8f * mu, fmaf(mw, fabsf(x), fmaf(mv, fabsf(c) + fabsf(s), mu)));
}

LMB_HD bool radial_needs_fp64(float h, float m1) {
  return 2.f * sqrtf(fmaxf(h, 0.f)) * RADIAL_FIELD_REL * m1 > HOLO_TOL;
}

// FP32 field (re, im) of one pixel, summed over the particles, and its bound.
struct RadialSum {
  f2 ex, ey, ez;
  float m1;
};

// Adds a particle's field at the offset (dx, dy) from its axis, the grid
// kernel's arithmetic with x and y in the two lanes.  table: the particle's
// intervals.
LMB_HD void radial_point(double dx, double dy, float inv_spacing, float spacing,
                         float inv_half, int intervals, const f4* table, RadialSum& s) {
  constexpr int RQ = RADIAL_REC / 4;
  const double ax = rint(dx * 1024.) * (1. / 1024.), ay = rint(dy * 1024.) * (1. / 1024.);
  const f2 X = pk(float(ax), float(ay)), rx = pk(float(dx - ax), float(dy - ay));
  const f2 px = pmul(X, X);
  const f2 lx = pfma(padd(rx, rx), pfma(pk(0.5f, 0.5f), rx, X), pfma(X, X, pneg(px)));
  const f2 Xr = padd(X, rx);
  const RadialDistance d =
      radial_distance(pk(px.x, px.x), pk(lx.x, lx.x), pk(px.y, px.y), pk(lx.y, lx.y));
  const int r = radial_round(d.r0.x * inv_spacing);
  const int i = r < 0 ? 0 : r < intervals ? r : intervals - 1;
  const float t = ((d.r0.x - float(i) * spacing) + d.corr.x) * inv_half;
  const f4* rec = table + size_t(i) * RQ;
  const f2 u = radial_eval(rec, t), v = radial_eval(rec + RQ / 3, t),
           w = radial_eval(rec + 2 * (RQ / 3), t);
  const float c = (Xr.x - Xr.y) * (Xr.x + Xr.y), s2 = (Xr.x + Xr.x) * Xr.y;
  s.ex = pfma(pk(c, c), v, padd(s.ex, u));
  s.ey = pfma(pk(s2, s2), v, s.ey);
  s.ez = pfma(pk(Xr.x, Xr.x), w, s.ez);
  s.m1 += radial_bound(u, v, w, c, s2, Xr.x);
}

// The same in FP64, straight from the particle's nodes (the first
// RADIAL_SIDE before the axis), e: (re, im) of E_x, E_y, E_z.
LMB_HD void radial_point64(double dx, double dy, double spacing, int intervals,
                           const d2* nodes, double* e) {
  const double rho = sqrt(dx * dx + dy * dy);
  const double u = rho / spacing;
  const int j = int(u + 0.5) < intervals ? int(u + 0.5) : intervals - 1;
  double w[RADIAL_TAPS], v[RADIAL_FUNCS];
  radial_weights(u - double(j), w);
  for (int c = 0; c < RADIAL_FUNCS; ++c) v[c] = 0.;
  const d2* s = nodes + size_t(j) * (RADIAL_FUNCS / 2);
#if defined(__CUDACC__)
#pragma unroll
#endif
  for (int l = 0; l < RADIAL_TAPS; ++l)
    for (int c = 0; c < RADIAL_FUNCS / 2; ++c) {
      const d2 n = s[l * (RADIAL_FUNCS / 2) + c];
      v[2 * c] = fma(w[l], n.x, v[2 * c]);
      v[2 * c + 1] = fma(w[l], n.y, v[2 * c + 1]);
    }
  const double c2 = dx * dx - dy * dy, s2 = 2. * dx * dy;
  for (int c = 0; c < 2; ++c) {
    e[c] += v[c] + c2 * v[2 + c];
    e[2 + c] += s2 * v[2 + c];
    e[4 + c] += dx * v[4 + c];
  }
}

}  // namespace lmb
