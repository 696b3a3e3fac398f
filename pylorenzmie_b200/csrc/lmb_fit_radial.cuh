// Evaluation of the batched fits from radial tables.
//
// A feature's pixels lie in the plane z = 0, where the hologram of one
// sphere at azimuth phi and distance rho from its axis is
//   H = 1 + M + D (x^2 - y^2),
// (x, y) the offset from the axis, M = (P + Q) / 2, D = (P - Q) / (2 rho^2),
// P = |X1|^2 + |Z1|^2 + 2 Re X1 and Q = |X2|^2 + 2 Re X2 (lmb_radial.cuh).
// M and D and their derivatives with respect to z_p, a_p, n_p (and k_p) are
// even functions of rho; those with respect to x_p and y_p follow from
// dM/drho and dD/drho, the slopes of the polynomials.  So a feature's sums
// over the orders are formed in FP64 at ~100-200 nodes, and its pixels
// (40 401 in a 201x201 crop) evaluate four pairs of degree-5 polynomials.
#pragma once

#include "lmb_kernels.cuh"
#include "lmb_radial.cuh"

namespace lmb {

enum {
  FITR_TPB = 256,
  FITR_PAIRS = 4,     // (M, D) and its z_p, a_p, n_p derivatives
  FITR_MAX_PARTS = 16,
  FITR_SUM = 64  // patches of 64 pixels in one sum of a tile
};

// float4 per interval: 3 per pair; an odd number keeps neighbouring
// intervals in different banks.
__host__ __device__ constexpr int fitr_rec(bool kp) { return kp ? 15 : 13; }
__host__ __device__ constexpr int fitr_funcs(bool kp) { return 2 * (FITR_PAIRS + (kp ? 1 : 0)); }

// Node spacing in radians of the hologram's own fastest oscillation (k q per
// pixel, fitr_rate): the degree-5 polynomials of half a spacing to either
// side are then off by 2 (0.65 / 4)^6 / 6! = 5e-8 of its amplitude.
#define FITR_SPACING 0.65
// The largest reach (k times px, times the rate where that is above 1) that
// lmb_fit_radial_reach gives: the room of ~620 intervals in shared memory,
// crops of 500 px at a magnification of 0.048 um.
#define FITR_REACH 400.

// The fastest oscillation of H along rho, in units of k: the carrier of the
// interference term turns by k sin(theta), theta the steepest ray from the
// sphere's edge to the outermost pixel, and |E|^2 by the difference of the
// directions under which a pixel sees the sphere, at most twice the angle of
// its edge from its axis.  The sphere's edge is widened by 6 / k for the
// partial waves beyond the geometric radius.
__host__ __device__ inline float fitr_rate(float k, float a_px, float z, float rho) {
  const float a = a_px + 6.f / k;
  const float far = rho + a;
  const float s1 = far * rsqrt_seed(far * far + z * z);
  const float s2 = 2.f * a * rsqrt_seed(a * a + z * z);
  return fminf(2.f, fmaxf(0.25f, fmaxf(s1, s2)));
}

// FP64 order records: alpha, beta and their a_p, n_p derivatives, and what
// the recurrences take of n alone (a division in their loop would cost as
// much as all the rest of an order).
struct FitrOrder {
  zd v[6];  // alpha, beta, d alpha/da, d beta/da, d alpha/dn, d beta/dn
  zd z[3];  // n (n+1) times alpha and its derivatives
  double fn, tn1, cn, en;  // n, 2n - 1, 1 + 1/n, (2n + 1) / (n (n + 1))
};

struct FitrPlan {      // of one part of a feature, in shared memory
  double spacing;
  float ax, rx, ay, ry;  // crop origin minus particle: 2^-10 px part, rest
  int lo, n;             // intervals
  int radial;            // 0: sum the orders at every pixel
};

// A node's geometry beyond Geometry<double>: the factors of the projected
// sums X1 = ph (A0 S0 + A1 S1), Z1 = ph (B0 S0 + B1 S1), X2 = ph C2 S2.
struct FitrProjection {
  double A0, A1, B0, B1, C2;
};
__device__ inline FitrProjection fitr_projection(const Geometry<double>& g) {
  const double w0 = g.sint * g.ikr * g.ikr;
  FitrProjection q;
  q.A0 = g.sint * w0;
  q.A1 = g.mu * g.ikr;
  q.B0 = g.mu * w0;
  q.B1 = -g.sint * g.ikr;
  q.C2 = -g.ikr;
  return q;
}

// M, D and their derivatives at a node, times 1/noise: pair j in out[2 j
// stride], out[(2 j + 1) stride].  The order sums of the value, of one
// tangent along z_p and of the a_p and n_p derivatives; the empty asm
// statements keep the compiler from mixing their terms, which would spill
// where the kernel has 128 registers a thread.  z: the pixels' plane.
template <bool kKP>
__device__ __forceinline__ void fitr_node(double k, double rho, double z, double zp,
                                          bool bohren, double aberr, double inv_noise,
                                          const FitrOrder* rec, int nm, double* out,
                                          int stride) {
  const Geometry<double> g = geometry<double>(k, rho, 0., z - zp, z, zp, bohren);
  const double ikr = g.ikr, mu = g.mu, st = g.sint;
  // d kr / dz_p = k mu, d mu / dz_p = k st^2 / kr
  const double krz = k * mu, muz = k * st * st * ikr;
  const zd zero = mk(0., 0.);
  zd sv[3] = {zero, zero, zero}, sd[3] = {zero, zero, zero};
  zd sa[3] = {zero, zero, zero}, sn[3] = {zero, zero, zero};
  {
    double pim1 = 0., pi = 1., del = 1., dpim1 = 0., dpi = 0., ddel = 0.;
    zd h2 = g.hm1, h1 = g.h0, hp2 = zero, hp1 = zero;
    const double s = g.s1mu, ik = g.ikrs, ik2 = g.ikrs * ikr * krz;
    const double sz = -g.smu * muz;  // of s = 1 - |mu|
#pragma unroll 1
    for (int n = 1; n <= nm; ++n) {
      const FitrOrder& r = rec[n];
      const double spi = s * pi;
      const double tau = pim1 + r.fn * (spi - del);
      const double dspi = sz * pi + s * dpi;
      const double dtau = dpim1 + r.fn * (dspi - ddel);
      const double a2 = r.tn1 * ik, a1 = r.fn * ik;
      const zd h = mk(a2 * h1.re - h2.re, a2 * h1.im - h2.im);
      const zd dh = mk(a1 * h.re - h1.re, a1 * h.im - h1.im);
      {
        const zd X = r.v[0] * dh, Y = r.v[1] * h, Z = r.z[0] * h;
        sv[0] = sv[0] + pi * Z;
        sv[1] = sv[1] + tau * X - pi * Y;
        sv[2] = sv[2] + pi * X - tau * Y;
        sd[0] = sd[0] + dpi * Z;
        sd[1] = sd[1] + dtau * X - dpi * Y;
        sd[2] = sd[2] + dpi * X - dtau * Y;
      }
      asm volatile("" ::: "memory");
      {
        const zd X = r.v[2] * dh, Y = r.v[3] * h, Z = r.z[1] * h;
        sa[0] = sa[0] + pi * Z;
        sa[1] = sa[1] + tau * X - pi * Y;
        sa[2] = sa[2] + pi * X - tau * Y;
      }
      asm volatile("" ::: "memory");
      {
        const zd X = r.v[4] * dh, Y = r.v[5] * h, Z = r.z[2] * h;
        sn[0] = sn[0] + pi * Z;
        sn[1] = sn[1] + tau * X - pi * Y;
        sn[2] = sn[2] + pi * X - tau * Y;
      }
      asm volatile("" ::: "memory");
      const double b2 = r.tn1 * ik2, b1 = r.fn * ik2;
      const zd hp = mk(a2 * hp1.re - b2 * h1.re - hp2.re, a2 * hp1.im - b2 * h1.im - hp2.im);
      const zd dhp = mk(a1 * hp.re - b1 * h.re - hp1.re, a1 * hp.im - b1 * h.im - hp1.im);
      {
        const zd X = r.v[0] * dhp, Y = r.v[1] * hp, Z = r.z[0] * hp;
        sd[0] = sd[0] + pi * Z;
        sd[1] = sd[1] + tau * X - pi * Y;
        sd[2] = sd[2] + pi * X - tau * Y;
      }
      // Delta_{n+1} = c_n (Delta_n - s pi_n) - s pi_n
      del = r.cn * (del - spi) - spi;
      ddel = r.cn * (ddel - dspi) - dspi;
      pim1 = pi;
      pi = pi + del;
      dpim1 = dpi;
      dpi = dpi + ddel;
      h2 = h1;
      h1 = h;
      hp2 = hp1;
      hp1 = hp;
    }
  }
  // undo the parity folding (order_sum_jac); the z tangent of pi~, tau~ and
  // h~ was carried through s and kr, so component 2 takes the same sign
  sv[2] = g.smu * sv[2];
  sd[2] = g.smu * sd[2];
  sa[2] = g.smu * sa[2];
  sn[2] = g.smu * sn[2];
  double rate = (g.sigma != 0. && g.sigma == g.smu) ? -g.s1mu : g.sigma * mu - 1.;
  rate *= k;
  zd ph = g.phase;
  if (aberr != 0.) {
    double d[3];
    ph = ph * conj(aberration_wave<double>(aberr, rho, 0., zp, d));
    rate += d[2];
  }
  const FitrProjection q = fitr_projection(g);
  const double ir2 = 0.5 / (rho * rho);
  auto put = [&](int pair, double P, double Q) {
    out[2 * pair * stride] = 0.5 * (P + Q) * inv_noise;
    out[(2 * pair + 1) * stride] = ir2 * (P - Q) * inv_noise;
  };
  const zd x1 = ph * (q.A0 * sv[0] + q.A1 * sv[1]);
  const zd z1 = ph * (q.B0 * sv[0] + q.B1 * sv[1]);
  const zd x2 = ph * (q.C2 * sv[2]);
  put(0, norm2(x1) + norm2(z1) + 2. * x1.re, norm2(x2) + 2. * x2.re);
  out[0] += inv_noise;  // the reference wave's 1
  const zd w1 = mk(x1.re + 1., x1.im), w2 = mk(x2.re + 1., x2.im);
  auto slope = [&](zd d1, zd dz, zd d2, int pair) {
    put(pair, 2. * (w1.re * d1.re + w1.im * d1.im + z1.re * dz.re + z1.im * dz.im),
        2. * (w2.re * d2.re + w2.im * d2.im));
  };
  {
    const double w0 = st * ikr * ikr;
    const double stz = -k * st * mu * ikr, ikz = -ikr * ikr * krz;
    const double w0z = stz * ikr * ikr + 2. * st * ikr * ikz;
    const double A0z = stz * w0 + st * w0z, A1z = muz * ikr + mu * ikz;
    const double B0z = muz * w0 + mu * w0z, B1z = -stz * ikr - st * ikz, C2z = -ikz;
    const zd d1 =
        ph * (A0z * sv[0] + A1z * sv[1] + q.A0 * sd[0] + q.A1 * sd[1]) + rate * mul_i(x1);
    const zd dz =
        ph * (B0z * sv[0] + B1z * sv[1] + q.B0 * sd[0] + q.B1 * sd[1]) + rate * mul_i(z1);
    const zd d2 = ph * (C2z * sv[2] + q.C2 * sd[2]) + rate * mul_i(x2);
    slope(d1, dz, d2, 1);
  }
  slope(ph * (q.A0 * sa[0] + q.A1 * sa[1]), ph * (q.B0 * sa[0] + q.B1 * sa[1]),
        ph * (q.C2 * sa[2]), 2);
  const zd n1 = ph * (q.A0 * sn[0] + q.A1 * sn[1]), nz = ph * (q.B0 * sn[0] + q.B1 * sn[1]),
           n2 = ph * (q.C2 * sn[2]);
  slope(n1, nz, n2, 3);
  // a_n, b_n are holomorphic in the index: d/dk_p = i d/dn_p
  if (kKP) slope(mul_i(n1), mul_i(nz), mul_i(n2), 4);
}

// The same as a call, for the kernel whose pixel loop sets its registers.
template <bool kKP>
__device__ __noinline__ void fitr_node_call(double k, double rho, double zp, bool bohren,
                                            double aberr, double inv_noise,
                                            const FitrOrder* rec, int nm, double* out,
                                            int stride) {
  fitr_node<kKP>(k, rho, 0., zp, bohren, aberr, inv_noise, rec, nm, out, stride);
}

// A pair of functions and their slopes at t: v = (M, D), d = dv/dt.
__device__ inline void fitr_pair_slope(const float4* r, float t, f2& v, f2& d) {
  const float4 a = r[0], b = r[1], c = r[2];
  const f2 tt = pk(t, t);
  d = pk(c.z, c.w);
  v = pfma(d, tt, pk(c.x, c.y));
  d = pfma(d, tt, v);
  v = pfma(v, tt, pk(b.z, b.w));
  d = pfma(d, tt, v);
  v = pfma(v, tt, pk(b.x, b.y));
  d = pfma(d, tt, v);
  v = pfma(v, tt, pk(a.z, a.w));
  d = pfma(d, tt, v);
  v = pfma(v, tt, pk(a.x, a.y));
}
__device__ inline f2 fitr_pair(const float4* r, float t) {
  const float4 a = r[0], b = r[1], c = r[2];
  const f2 tt = pk(t, t);
  f2 v = pfma(pk(c.z, c.w), tt, pk(c.x, c.y));
  v = pfma(v, tt, pk(b.z, b.w));
  v = pfma(v, tt, pk(b.x, b.y));
  v = pfma(v, tt, pk(a.z, a.w));
  return pfma(v, tt, pk(a.x, a.y));
}

// The sums of one pixel: f^2, J^T J (packed upper over the six slots) and
// J^T f, k_p's only with kKP.
template <bool kKP>
__device__ inline void fitr_add(float r, const float* J, float* acc) {
  constexpr int N = kKP ? 6 : 5;
  acc[0] = fmaf(r, r, acc[0]);
#pragma unroll
  for (int a = 0; a < N; ++a) {
#pragma unroll
    for (int b = a; b < N; ++b) {
      const int o = 1 + a * 6 - a * (a - 1) / 2 + (b - a);
      acc[o] = fmaf(J[a], J[b], acc[o]);
    }
    acc[22 + a] = fmaf(J[a], r, acc[22 + a]);
  }
}

// Hologram and derivatives of one pixel from the table, times 1/noise.
template <bool kKP>
__device__ inline float fitr_lookup(const float4* tab, float r0, float corr, float inv_rho,
                                    float x, float y, float inv_spacing, float spacing,
                                    float inv_half, int lo, int n, float* J) {
  const int i = min(max(__float2int_rn(r0 * inv_spacing) - lo, 0), n - 1);
  const float t = ((r0 - float(i + lo) * spacing) + corr) * inv_half;
  const float4* rec = tab + i * fitr_rec(kKP);
  f2 v, s;
  fitr_pair_slope(rec, t, v, s);
  const float u = (x - y) * (x + y);
  // dH/dx = cos(phi) B + 2 D x, B = M' + D' (x^2 - y^2)
  const float B = fmaf(s.y, u, s.x) * (inv_half * inv_rho);
  J[0] = -x * fmaf(2.f, v.y, B);
  J[1] = -y * fmaf(-2.f, v.y, B);
#pragma unroll
  for (int j = 0; j < (kKP ? 4 : 3); ++j) {
    const f2 w = fitr_pair(rec + 3 * (j + 1), t);
    J[2 + j] = fmaf(w.y, u, w.x);
  }
  return fmaf(v.y, u, v.x);
}

// The sums of one pixel; d: its measured value.
template <bool kKP>
__device__ inline void fitr_pixel(const float4* tab, float r0, float corr, float inv_rho,
                                  float x, float y, float inv_spacing, float spacing,
                                  float inv_half, int lo, int n, float d, float inv_noise,
                                  float* acc) {
  float J[6];
  const float h = fitr_lookup<kKP>(tab, r0, corr, inv_rho, x, y, inv_spacing, spacing,
                                   inv_half, lo, n, J);
  fitr_add<kKP>(fmaf(-d, inv_noise, h), J, acc);
}

// The polynomials of intervals [0, n) from the nodes val[function][stride]
// (the first node RADIAL_SIDE before interval 0's), by the whole block.
template <int REC, int NF>
__device__ inline void fitr_polynomials(const RadialMatrix& A, const double* val, int stride,
                                        int n, float4* tab) {
  for (int w = threadIdx.x; w < n * (NF / 2); w += FITR_TPB) {
    const int g = w / n, i = w - g * n;
    const double* s = val + 2 * g * stride + i;
    double cr[RADIAL_COEFS], ci[RADIAL_COEFS];
#pragma unroll
    for (int j = 0; j < RADIAL_COEFS; ++j) cr[j] = ci[j] = 0.;
#pragma unroll
    for (int l = 0; l < RADIAL_TAPS; ++l) {
      const double x = s[l], y = s[stride + l];
#pragma unroll
      for (int j = 0; j < RADIAL_COEFS; ++j) {
        cr[j] = fma(A.m[j][l], x, cr[j]);
        ci[j] = fma(A.m[j][l], y, ci[j]);
      }
    }
    float4* o = tab + size_t(i) * REC + 3 * g;
#pragma unroll
    for (int j = 0; j < RADIAL_COEFS; j += 2)
      o[j / 2] = make_float4(float(cr[j]), float(ci[j]), float(cr[j + 1]), float(ci[j + 1]));
  }
}

// f(x, y, distance, pixel) for every pixel of rows [row0, row0 + rows) of a
// grid of nx columns; (ax, rx, ay, ry): the grid's first pixel minus the
// particle, split as radial_distance wants it.  A warp takes 8x8 pixels, two
// per lane (rows y and y + 4): eight lanes on 4x2 pixels read intervals in
// different banks.  With [w0, w1) only these of the fitr_patches.
__device__ inline int fitr_patches(int nx, int rows) {
  return ((nx + 7) / 8) * ((rows + 7) / 8);
}
template <typename F>
__device__ inline void fitr_rows(int nx, int row0, int rows, float ax, float rx, float ay,
                                 float ry, int w0, int w1, F f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int pc = (nx + 7) / 8;
  const int lx = 4 * ((lane >> 3) & 1) + (lane & 3);
  const int ly = 2 * (lane >> 4) + ((lane >> 2) & 1);
  for (int w = w0 + warp; w < w1; w += FITR_TPB / 32) {
    const int pr = w / pc, col = 8 * (w - pr * pc) + lx, row = row0 + 8 * pr + ly;
    if (col >= nx || row >= row0 + rows) continue;
    const float X = ax + float(col);
    const f2 Y = pk(ay + float(row), ay + float(row + 4));
    const float px = X * X;
    const float lx2 = fmaf(2.f * rx, fmaf(0.5f, rx, X), fmaf(X, X, -px));
    const f2 qy = pmul(Y, Y), r2 = pk(ry, ry);
    const f2 ly2 = pfma(padd(r2, r2), pfma(pk(0.5f, 0.5f), r2, Y), pfma(Y, Y, pneg(qy)));
    const RadialDistance d = radial_distance(pk(px, px), pk(lx2, lx2), qy, ly2);
    f(X + rx, padd(Y, r2), d, (long long)row * nx + col, row + 4 < row0 + rows);
  }
}

// The distance of a pixel of a list; (*x, *y): its FP32 offset.
__device__ inline RadialDistance fitr_list_distance(double dx, double dy, float* x, float* y) {
  const double ax = rint(dx * 1024.) * (1. / 1024.);
  const double ay = rint(dy * 1024.) * (1. / 1024.);
  const f2 X = pk(float(ax), float(ay)), rx = pk(float(dx - ax), float(dy - ay));
  const f2 px = pmul(X, X);
  const f2 lx = pfma(padd(rx, rx), pfma(pk(0.5f, 0.5f), rx, X), pfma(X, X, pneg(px)));
  const f2 xr = padd(X, rx);
  *x = xr.x;
  *y = xr.y;
  return radial_distance(pk(px.x, px.x), pk(lx.x, lx.x), pk(px.y, px.y), pk(lx.y, lx.y));
}

// Sum of acc over the block into (add: onto) out[0..FIT_NSUM) (doubles), fixed
// order, FP32 within a warp.
// Each warp halves the values it holds at every step of the butterfly, so
// that 28 sums take 31 shuffles instead of 140.
__device__ inline void fitr_reduce(float* acc, float (*red)[32], double* out,
                                   bool add = false) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float v[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = j < FIT_NSUM ? acc[j] : 0.f;
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    const bool up = lane & w;
#pragma unroll
    for (int j = 0; j < w; ++j) {
      const float send = up ? v[j] : v[j + w];
      const float keep = up ? v[j + w] : v[j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, w);
    }
  }
  // lane l now holds the warp's sum of value l
  red[warp][lane] = v[0];
  __syncthreads();
  if (threadIdx.x < FIT_NSUM) {
    double s = add ? out[threadIdx.x] : 0.;
    for (int w = 0; w < FITR_TPB / 32; ++w) s += double(red[w][threadIdx.x]);
    out[threadIdx.x] = s;
  }
  __syncthreads();
}

// The orders summed at every pixel of tiles [t0, t1), for the parts where
// the tables do not apply (a plane that cuts or almost touches the sphere).
__device__ __noinline__ void fitr_direct(const FitCtx& c, int f, const lmb_feature& ft,
                                         const double* p, int nm, int t0, int t1, int band,
                                         Quad<float>* coef, float (*red)[32]) {
  const int nmaxp = c.nmax_cap + 1;
  stage_coef<float, true>(c.ab + size_t(f) * nmaxp * 2, c.dab + size_t(f) * nmaxp * 4, nm,
                          coef);
  __syncthreads();
  const float inv_noise = float(c.inv_noise);
  for (int t = t0; t < t1; ++t) {
    long long a = (long long)t * FITR_TILE, b = a + FITR_TILE;
    if (ft.nx > 0) {
      a = (long long)t * band * ft.nx;
      b = a + (long long)band * ft.nx;
    }
    if (b > ft.npix) b = ft.npix;
    double* out = c.partial + (size_t)(c.tile_begin[f] + t) * FIT_NSUM;
    constexpr int kSum = 64 * FITR_SUM;  // pixels in one sum, as the tables'
    for (long long a0 = a; a0 < b; a0 += kSum) {
      float acc[FIT_NSUM];
#pragma unroll
      for (int j = 0; j < FIT_NSUM; ++j) acc[j] = 0.f;
      for (long long i = a0 + threadIdx.x; i < min(b, a0 + kSum); i += FITR_TPB) {
        double x, y;
        fit_pixel_xy(ft, c.coords, i, &x, &y);
        const double dx = x - p[0], dy = y - p[1];
        const Geometry<float> g =
            geometry<float>(c.k, dx, dy, -p[2], 0., p[2], c.flags & LMB_BOHREN);
        float H, dH[6];
        if (c.aberr != 0.)
          holo_jac_pixel<true>(g, coef, nm, float(c.k), &H, dH, c.aberr, dx, dy, p[2]);
        else
          holo_jac_pixel<false>(g, coef, nm, float(c.k), &H, dH);
        const float r = (H - c.data[ft.data_offset + i]) * inv_noise;
        for (int j = 0; j < 6; ++j) dH[j] *= inv_noise;
        fitr_add<true>(r, dH, acc);
      }
      fitr_reduce(acc, red, out, a0 > a);
    }
  }
}

// Persistent CTAs pull (feature, part) items: c.parts parts a feature, each
// a run of its tiles.  A CTA builds the table of its part in shared memory
// (FP64 nodes, then the polynomials) and evaluates its pixels from it.  The
// nodes' spacing follows from the whole feature, so a tile's sums do not
// depend on how the tiles are dealt out, nor on the other features, while the
// part's intervals find room.  cap: intervals that the table has room for.
//
// 256 features of 201x201 px, 25 orders: 0.13 ms, against 1.14-1.28 ms with
// the orders summed at every pixel.  By clock64 stamps a CTA takes 9 k clocks
// for the plan, 37 k for the nodes (146 threads, FP64 latency at 128
// registers), 10 k for the polynomials and 170 k for the pixels, two CTAs an
// SM: 192 bytes of shared memory and ~230 instructions a pixel, issue and
// shared-memory bandwidth about even.  Parts: one while the features alone
// fill the 296 CTAs, since every part forms its own nodes.
template <bool kKP>
__global__ void __launch_bounds__(FITR_TPB, 2)
k_fit_eval_radial(FitCtx c, RadialMatrix A, int cap) {
  extern __shared__ __align__(16) char smem[];
  __shared__ float red[FITR_TPB / 32][32];
  __shared__ FitrPlan s_pl;
  __shared__ float s_rho[3][FITR_TPB / 32];
  __shared__ int s_item;
  constexpr int REC = fitr_rec(kKP), NF = fitr_funcs(kKP);
  const int nmaxp = c.nmax_cap + 1;
  float4* tab = reinterpret_cast<float4*>(smem);                       // [cap][REC]
  double* val = reinterpret_cast<double*>(tab + size_t(cap) * REC);    // [NF][cap + 16]
  const int vstride = cap + 2 * RADIAL_SIDE;
  FitrOrder* ord = reinterpret_cast<FitrOrder*>(val + size_t(NF) * vstride);
  // the direct sums' FP32 records, in the tables' place
  Quad<float>* direct = reinterpret_cast<Quad<float>*>(smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float inv_noise = float(c.inv_noise);
  const int ntiles = c.counters[c.tiles_slot];  // (feature, part) items
  fit_eval_begin(c);
  for (int n = threadIdx.x; n < nmaxp; n += FITR_TPB) {
    const double fn = double(n);
    ord[n].fn = fn;
    ord[n].tn1 = 2. * fn - 1.;
    ord[n].cn = n ? 1. + 1. / fn : 0.;
    ord[n].en = n ? (2. * fn + 1.) / (fn * (fn + 1.)) : 0.;
  }
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(c.counters, 1);
    __syncthreads();
    const int q = s_item;
    if (q >= ntiles) break;
    const int item = c.active_tiles[q];
    const int f = item / c.parts, part = item - f * c.parts;
    const int nt = c.tile_begin[f + 1] - c.tile_begin[f];
    const int t0 = int((long long)nt * part / c.parts);
    const int t1 = int((long long)nt * (part + 1) / c.parts);
    if (t0 == t1) {
      __syncthreads();  // s_item is rewritten
      continue;
    }
    const lmb_feature ft = c.features[f];
    const EvalPoint ep = c.ev[f];
    const int nm = min(max(c.nmax[f], 0), nmaxp - 1);
    const int band = ft.nx > 0 ? fitr_band(ft.nx) : 0;
    const long long i0 = (long long)t0 * FITR_TILE;
    const long long i1 = min((long long)t1 * FITR_TILE, ft.npix);
    // ---- the distances of a list's pixels: the part's, and the farthest
    if (ft.nx == 0) {
      float lo = 3e38f, hi = 0.f, far = 0.f;
#pragma unroll 4
      for (long long i = threadIdx.x; i < ft.npix; i += FITR_TPB) {
        const float2 xy = reinterpret_cast<const float2*>(c.coords)[ft.data_offset + i];
        const float dx = xy.x - float(ep.p[0]), dy = xy.y - float(ep.p[1]);
        const float r = sqrtf(dx * dx + dy * dy);
        far = r <= far ? far : r;  // NaN passes on
        if (i >= i0 && i < i1) {
          lo = fminf(lo, r);
          hi = r <= hi ? hi : r;
        }
      }
      for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        const float h = __shfl_xor_sync(0xffffffffu, hi, o);
        const float g = __shfl_xor_sync(0xffffffffu, far, o);
        hi = h <= hi ? hi : h;
        far = g <= far ? far : g;
      }
      if (lane == 0) {
        s_rho[0][warp] = lo;
        s_rho[1][warp] = hi;
        s_rho[2][warp] = far;
      }
      __syncthreads();
    }
    // ---- the plan (warp 0), and the order records meanwhile
    for (int n = int(threadIdx.x) - 32; n <= nm && n >= 0; n += FITR_TPB - 32) {
      const zd* ab = c.ab + (size_t(f) * nmaxp + n) * 2;
      const zd* dab = c.dab + (size_t(f) * nmaxp + n) * 4;
      const double en = ord[n].en;
      for (int j = 0; j < 3; ++j) {
        const zd* s = j == 0 ? ab : dab + 2 * (j - 1);
        ord[n].v[2 * j] = en * rot_i(s[0], n + 1);
        ord[n].z[j] = (2. * double(n) + 1.) * rot_i(s[0], n + 1);
        ord[n].v[2 * j + 1] = en * rot_i(s[1], n);
      }
    }
    if (threadIdx.x == 0) {
      FitrPlan pl;
      const float zp = float(fabs(ep.p[2])), k = float(c.k);
      const double ox = (ft.nx > 0 ? ft.x0 : 0.) - ep.p[0];
      const double oy = (ft.nx > 0 ? ft.y0 : 0.) - ep.p[1];
      // nearest and farthest distances, and the farthest of the feature's
      // pixels; FP32, as the intervals have margins
      float lo, hi, far;
      if (ft.nx > 0) {
        const float x0 = float(ox), x1 = x0 + float(ft.nx - 1);
        const float y0 = float(oy) + float(t0 * band);
        const float y1 =
            float(oy) + float(min((long long)t1 * band, (long long)ft.ny) - 1);
        const float nx = x0 > 0.f ? x0 : (x1 < 0.f ? -x1 : 0.f);
        const float ny = y0 > 0.f ? y0 : (y1 < 0.f ? -y1 : 0.f);
        const float fx = fmaxf(fabsf(x0), fabsf(x1)), fy = fmaxf(fabsf(y0), fabsf(y1));
        const float gy = fmaxf(fabsf(float(oy)), fabsf(float(oy) + float(ft.ny - 1)));
        lo = sqrtf(nx * nx + ny * ny);
        hi = sqrtf(fx * fx + fy * fy);
        far = sqrtf(fx * fx + gy * gy);
      } else {
        lo = s_rho[0][0];
        hi = s_rho[1][0];
        far = s_rho[2][0];
        for (int w = 1; w < FITR_TPB / 32; ++w) {
          lo = fminf(lo, s_rho[0][w]);
          hi = s_rho[1][w] <= hi ? hi : s_rho[1][w];
          far = s_rho[2][w] <= far ? far : s_rho[2][w];
        }
      }
      const double x = c.size_per_um * ep.p[3];  // size parameter
      float rate = fitr_rate(k, float(x) / k, zp, far);
      bool ok = radial_clear(c.k, fabs(ep.p[2]), x / c.k, false) && far < 8000.f &&
                zp < 1e6f && isfinite(ep.p[0]) && isfinite(ep.p[1]);
      if (c.aberr != 0.) {  // the aberration's phase, as lmb_radial_intervals
        const float turn = 0.5f * fabsf(float(c.aberr)) / zp;
        ok = ok && turn <= 0.2f * k;
        rate = fminf(2.f, rate + turn / k);
      }
      // a multiple of 1/64 px, so that i * spacing is exact in FP32
      const float sp = fminf(8.f, floorf(64.f * float(FITR_SPACING) / (k * rate)) * 0.015625f);
      ok = ok && sp >= 0.0625f;
      pl.spacing = double(sp);
      pl.lo = pl.n = 0;
      if (ok) {
        const float is = 1.f / sp;
        pl.lo = max(0, int(lo * is) - 1);
        pl.n = int(hi * is) + 3 - pl.lo;
        ok = pl.n <= cap;
      }
      const double ax = rint(ox * 1024.) * (1. / 1024.), ay = rint(oy * 1024.) * (1. / 1024.);
      pl.ax = float(ax);
      pl.rx = float(ox - ax);
      pl.ay = float(ay);
      pl.ry = float(oy - ay);
      pl.radial = ok;
      s_pl = pl;
    }
    __syncthreads();
    const FitrPlan pl = s_pl;
    if (threadIdx.x == 0) {
      const long long np = ft.nx > 0
          ? (min((long long)t1 * band, (long long)ft.ny) - (long long)t0 * band) * ft.nx
          : i1 - i0;
      atomicAdd(c.work, (unsigned long long)np);
      atomicAdd(c.work + 1, (unsigned long long)nm *
                                (unsigned long long)(pl.radial ? pl.n + 2 * RADIAL_SIDE : np));
    }
    if (!pl.radial) {
      fitr_direct(c, f, ft, ep.p, nm, t0, t1, band, direct, red);
      continue;  // its last barrier follows every read of s_item and s_pl
    }
    // ---- nodes, polynomials
    for (int t = threadIdx.x; t < pl.n + 2 * RADIAL_SIDE; t += FITR_TPB) {
      const int j = abs(pl.lo - RADIAL_SIDE + t);
      fitr_node_call<kKP>(c.k, j ? pl.spacing * double(j) : RADIAL_AXIS, ep.p[2],
                     c.flags & LMB_BOHREN, c.aberr, c.inv_noise, ord, nm, val + t, vstride);
    }
    __syncthreads();
    fitr_polynomials<REC, NF>(A, val, vstride, pl.n, tab);
    __syncthreads();
    // ---- pixels
    const float spacing = float(pl.spacing), inv_spacing = float(1. / pl.spacing);
    const float inv_half = float(2. / pl.spacing);
    for (int t = t0; t < t1; ++t) {
      double* out = c.partial + (size_t)(c.tile_begin[f] + t) * FIT_NSUM;
      const int rows = min(band, ft.ny - t * band);
      const int np = ft.nx > 0 ? fitr_patches(ft.nx, rows) : 1;
      // at most 16 pixels a thread in a row of FP32 additions: tiles of crops
      // wider than 512 px take several sums
      for (int w0 = 0; w0 < np; w0 += FITR_SUM) {
        float acc[FIT_NSUM];
#pragma unroll
        for (int j = 0; j < FIT_NSUM; ++j) acc[j] = 0.f;
        if (ft.nx > 0) {
          const float* data = c.data + ft.data_offset;
          fitr_rows(ft.nx, t * band, rows, pl.ax, pl.rx, pl.ay, pl.ry, w0,
                    min(np, w0 + FITR_SUM),
                    [&](float x, f2 y, const RadialDistance& d, long long i, bool two) {
                      const float d0 = data[i], d1 = two ? data[i + 4LL * ft.nx] : 0.f;
                      fitr_pixel<kKP>(tab, d.r0.x, d.corr.x, d.y.x, x, y.x, inv_spacing,
                                      spacing, inv_half, pl.lo, pl.n, d0, inv_noise, acc);
                      if (two)
                        fitr_pixel<kKP>(tab, d.r0.y, d.corr.y, d.y.y, x, y.y, inv_spacing,
                                        spacing, inv_half, pl.lo, pl.n, d1, inv_noise, acc);
                    });
        } else {
          const long long a = (long long)t * FITR_TILE, b = min(a + FITR_TILE, ft.npix);
          for (long long i = a + threadIdx.x; i < b; i += FITR_TPB) {
            const float2 xy = reinterpret_cast<const float2*>(c.coords)[ft.data_offset + i];
            float x, y;
            const RadialDistance d = fitr_list_distance(double(xy.x) - ep.p[0],
                                                        double(xy.y) - ep.p[1], &x, &y);
            fitr_pixel<kKP>(tab, d.r0.x, d.corr.x, d.y.x, x, y, inv_spacing, spacing,
                            inv_half, pl.lo, pl.n, c.data[ft.data_offset + i], inv_noise, acc);
          }
        }
        fitr_reduce(acc, red, out, w0 > 0);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Gradients of holograms (the VJP) from the same tables, in two kernels: the
// nodes of every sphere, one a thread in blocks of FITR_NODE_TPB (the chain
// of FP64 recurrences is latency-bound, so the nodes are spread over all SMs
// and each thread may hold its sums in registers); then blocks of rows,
// which take their range of nodes, form the polynomials and sum g dH/dp.
// 12 images of 401x401 px, ~109 orders: 38 and 57 us; forward and backward
// together 1.59 -> 0.57 ms against sums at every pixel.

struct GradPlan {
  double x0, y0, z, k, spacing;  // first pixel (or the box's corner), plane
  long long nx, ny, npts;
  const double* points;  // null: the grid's pixels
  int intervals;         // room per sphere
  int parts, flags;
};

enum { FITR_NODE_TPB = 32 };

// Intervals that cover the pixels of a sphere at (xp, yp).
__device__ inline int grad_count(const GradPlan& pl, double xp, double yp) {
  const double dx = fmax(fabs(pl.x0 - xp), fabs(pl.x0 + double(pl.nx - 1) - xp));
  const double dy = fmax(fabs(pl.y0 - yp), fabs(pl.y0 + double(pl.ny - 1) - yp));
  return min(pl.intervals, int(sqrt(fma(dx, dx, dy * dy)) / pl.spacing) + 2);
}

// nodes [nitems][10][intervals + 16]
__global__ void __launch_bounds__(FITR_NODE_TPB)
k_grad_nodes(GradPlan pl, const lmb_sphere* __restrict__ spheres,
             const zd* __restrict__ ab, const zd* __restrict__ dab,
             const int* __restrict__ nmax, int nmaxp, double* __restrict__ nodes) {
  extern __shared__ __align__(16) char smem[];
  FitrOrder* ord = reinterpret_cast<FitrOrder*>(smem);
  const int item = blockIdx.y;
  const lmb_sphere sp = spheres[item];
  const int first = blockIdx.x * FITR_NODE_TPB;
  const int count = grad_count(pl, sp.x_p, sp.y_p) + 2 * RADIAL_SIDE;
  if (first >= count) return;  // the whole block
  const int nm = min(max(nmax[item], 0), nmaxp - 1);
  for (int n = threadIdx.x; n <= nm; n += FITR_NODE_TPB) {
    const double fn = double(n);
    FitrOrder o;
    o.fn = fn;
    o.tn1 = 2. * fn - 1.;
    o.cn = n ? 1. + 1. / fn : 0.;
    o.en = n ? o.tn1 + 2. : 0.;
    const double en = n ? o.en / (fn * (fn + 1.)) : 0.;
    for (int j = 0; j < 3; ++j) {
      const zd* s = j == 0 ? ab + (size_t(item) * nmaxp + n) * 2
                           : dab + (size_t(item) * nmaxp + n) * 4 + 2 * (j - 1);
      o.v[2 * j] = en * rot_i(s[0], n + 1);
      o.v[2 * j + 1] = en * rot_i(s[1], n);
      o.z[j] = o.en * rot_i(s[0], n + 1);
    }
    ord[n] = o;
  }
  __syncthreads();
  const int t = first + threadIdx.x;
  if (t >= count) return;
  const int j = abs(t - RADIAL_SIDE);
  const int stride = pl.intervals + 2 * RADIAL_SIDE;
  fitr_node<true>(pl.k, j ? pl.spacing * double(j) : RADIAL_AXIS, pl.z, sp.z_p,
                  pl.flags & LMB_BOHREN, 0., 1., ord, nm,
                  nodes + size_t(item) * fitr_funcs(true) * stride + t, stride);
}

// partial [nitems][parts][6]; cap: intervals that the table has room for.
__global__ void __launch_bounds__(FITR_TPB, 2)
k_vjp_radial(GradPlan pl, RadialMatrix A, int cap, const lmb_sphere* __restrict__ spheres,
             const double* __restrict__ nodes, const float* __restrict__ gout,
             double* __restrict__ partial) {
  extern __shared__ __align__(16) char smem[];
  __shared__ double red[FITR_TPB / 32][6];
  constexpr int REC = fitr_rec(true), NF = fitr_funcs(true);
  float4* tab = reinterpret_cast<float4*>(smem);                     // [cap][REC]
  double* val = reinterpret_cast<double*>(tab + size_t(cap) * REC);  // [NF][cap + 16]
  const int vstride = cap + 2 * RADIAL_SIDE;
  const int item = blockIdx.y, part = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const lmb_sphere sp = spheres[item];
  const int count = grad_count(pl, sp.x_p, sp.y_p);
  const float* g = gout + size_t(item) * pl.npts;
  // the part: rows in whole patches of 8, or a run of the list
  const long long groups = pl.points ? pl.npts : (pl.ny + 7) / 8;
  const long long b0 = groups * part / pl.parts, b1 = groups * (part + 1) / pl.parts;
  double acc[6] = {0., 0., 0., 0., 0., 0.};
  if (b0 < b1) {
    const double ox = pl.x0 - sp.x_p, oy = pl.y0 - sp.y_p;
    float rho_lo = 0.f, rho_hi = 3e38f;  // of a list: all of the table
    const int row0 = pl.points ? 0 : int(8 * b0);
    const int rows = pl.points ? 0 : int(min(8 * b1, pl.ny) - 8 * b0);
    if (!pl.points) {
      const float x0 = float(ox), x1 = x0 + float(pl.nx - 1);
      const float y0 = float(oy) + float(row0), y1 = y0 + float(rows - 1);
      const float ex = x0 > 0.f ? x0 : (x1 < 0.f ? -x1 : 0.f);
      const float ey = y0 > 0.f ? y0 : (y1 < 0.f ? -y1 : 0.f);
      const float fx = fmaxf(fabsf(x0), fabsf(x1)), fy = fmaxf(fabsf(y0), fabsf(y1));
      rho_lo = sqrtf(ex * ex + ey * ey);
      rho_hi = sqrtf(fx * fx + fy * fy);
    }
    const float spacing = float(pl.spacing), inv_spacing = 1.f / spacing;
    const float inv_half = 2.f * inv_spacing;
    const int hi = rho_hi < 1e9f ? min(count, int(rho_hi * inv_spacing) + 3) : count;
    const int lo = max(0, min(int(rho_lo * inv_spacing) - 1, hi - 1));
    const double ax = rint(ox * 1024.) * (1. / 1024.), ay = rint(oy * 1024.) * (1. / 1024.);
    const float fax = float(ax), frx = float(ox - ax), fay = float(ay), fry = float(oy - ay);
    const int stride = pl.intervals + 2 * RADIAL_SIDE;
    const double* src = nodes + size_t(item) * NF * stride;
    // the table in pieces of cap intervals: a wide part takes several passes
    for (int at = lo; at < hi; at += cap) {
      const int n = min(cap, hi - at);
      __syncthreads();  // the previous piece is no longer read
      for (int w = threadIdx.x; w < NF * (n + 2 * RADIAL_SIDE); w += FITR_TPB) {
        const int f = w / (n + 2 * RADIAL_SIDE), i = w - f * (n + 2 * RADIAL_SIDE);
        val[f * vstride + i] = src[f * stride + at + i];
      }
      __syncthreads();
      fitr_polynomials<REC, NF>(A, val, vstride, n, tab);
      __syncthreads();
      // a pixel belongs to the piece that holds its interval (clamped to the
      // part's range)
      float sum[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      int in_sum = 0;
      auto add = [&](float r0, float corr, float iy, float x, float y, long long i) {
        const int iv = min(max(__float2int_rn(r0 * inv_spacing), lo), hi - 1);
        if (iv < at || iv >= at + n) return;
        float J[6];
        fitr_lookup<true>(tab, r0, corr, iy, x, y, inv_spacing, spacing, inv_half, at, n, J);
        const float go = g[i];
#pragma unroll
        for (int j = 0; j < 6; ++j) sum[j] = fmaf(go, J[j], sum[j]);
        if (++in_sum == 8) {  // short FP32 sums
          for (int j = 0; j < 6; ++j) {
            acc[j] += double(sum[j]);
            sum[j] = 0.f;
          }
          in_sum = 0;
        }
      };
      if (pl.points) {
        for (long long i = b0 + threadIdx.x; i < b1; i += FITR_TPB) {
          float x, y;
          const RadialDistance d = fitr_list_distance(
              pl.points[i] - sp.x_p, pl.points[pl.npts + i] - sp.y_p, &x, &y);
          add(d.r0.x, d.corr.x, d.y.x, x, y, i);
        }
      } else {
        fitr_rows(int(pl.nx), row0, rows, fax, frx, fay, fry, 0,
                  fitr_patches(int(pl.nx), rows),
                  [&](float x, f2 y, const RadialDistance& d, long long i, bool two) {
                    add(d.r0.x, d.corr.x, d.y.x, x, y.x, i);
                    if (two) add(d.r0.y, d.corr.y, d.y.y, x, y.y, i + 4 * pl.nx);
                  });
      }
      for (int j = 0; j < 6; ++j) acc[j] += double(sum[j]);
    }
  }
  for (int o = 16; o > 0; o >>= 1)
    for (int j = 0; j < 6; ++j) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
  __syncthreads();
  if (lane == 0)
    for (int j = 0; j < 6; ++j) red[warp][j] = acc[j];
  __syncthreads();
  if (threadIdx.x < 6) {
    double s = 0.;
    for (int w = 0; w < FITR_TPB / 32; ++w) s += red[w][threadIdx.x];
    partial[(size_t(item) * pl.parts + part) * 6 + threadIdx.x] = s;
  }
}

}  // namespace lmb
