// Fields and holograms on a pixel grid from radial tables (lmb_radial.cuh):
// lmb_grid_probe, lmb_radial_intervals, lmb_radial_workspace_bytes,
// lmb_field_grid, lmb_hologram_grid.  Declarations: include/lmb200.h.
#include <cuda_pipeline.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <math.h>

#include "lmb200.h"
#include "lmb_launch.cuh"
#include "lmb_radial.cuh"

using namespace lmb;

namespace {

// ---------------------------------------------------------------------------
// Is a coordinate list a unit-step pixel grid, or at least in one plane?

enum { PROBE_ROW, PROBE_OFF_GRID, PROBE_OFF_PLANE, PROBE_LO_X, PROBE_LO_Y, PROBE_HI_X,
       PROBE_HI_Y, PROBE_Z };

// Doubles as unsigned integers in the same order, and back.
__device__ inline unsigned long long ordered(double v) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(v);
  return u ^ ((u >> 63) ? ~0ull : 1ull << 63);
}
__device__ inline double unordered(unsigned long long u) {
  return __longlong_as_double((long long)(u ^ ((u >> 63) ? 1ull << 63 : ~0ull)));
}

__global__ void k_probe_init(long long npts, unsigned long long* out) {
  out[PROBE_ROW] = (unsigned long long)npts;
  out[PROBE_OFF_GRID] = out[PROBE_OFF_PLANE] = 0ull;
  out[PROBE_LO_X] = out[PROBE_LO_Y] = ~0ull;
  out[PROBE_HI_X] = out[PROBE_HI_Y] = 0ull;
}

// The first index whose y differs from the first pixel's (npts if none),
// i.e. the row length of a grid.
__global__ void k_probe_row(const double* __restrict__ coords, long long npts,
                            unsigned long long* out) {
  const double y0 = coords[npts];
  unsigned long long first = (unsigned long long)npts;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < npts;
       i += (long long)gridDim.x * blockDim.x)
    if (coords[npts + i] != y0) {
      first = (unsigned long long)i;
      break;
    }
  for (int o = 16; o > 0; o >>= 1) first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
  // most warps find a later index than is already there
  if ((threadIdx.x & 31) == 0 &&
      first < *reinterpret_cast<volatile unsigned long long*>(out + PROBE_ROW))
    atomicMin(out + PROBE_ROW, first);
}

// How many pixels are not (x0 + column, y0 + row, z0), how many are not
// finite or not in the plane z0, and the bounds of x and y.
__global__ void k_probe_check(const double* __restrict__ coords, long long npts,
                              unsigned long long* out) {
  const long long nx = (long long)out[PROBE_ROW];
  const double x0 = coords[0], y0 = coords[npts], z0 = coords[2 * npts];
  unsigned long long off = 0, plane = 0, b[4] = {~0ull, ~0ull, 0ull, 0ull};
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < npts;
       i += (long long)gridDim.x * blockDim.x) {
    const double x = coords[i], y = coords[npts + i], z = coords[2 * npts + i];
    const long long row = i / nx;
    if (!(x == x0 + double(i - row * nx)) || !(y == y0 + double(row)) || !(z == z0)) ++off;
    if (!isfinite(x) || !isfinite(y) || !isfinite(z) || z != z0) ++plane;
    b[0] = min(b[0], ordered(x));
    b[1] = min(b[1], ordered(y));
    b[2] = max(b[2], ordered(x));
    b[3] = max(b[3], ordered(y));
  }
  for (int o = 16; o > 0; o >>= 1)
    for (int j = 0; j < 4; ++j) {
      const unsigned long long v = __shfl_xor_sync(0xffffffffu, b[j], o);
      b[j] = j < 2 ? min(b[j], v) : max(b[j], v);
    }
  if (off) atomicAdd(out + PROBE_OFF_GRID, off);
  if (plane) atomicAdd(out + PROBE_OFF_PLANE, plane);
  if ((threadIdx.x & 31) == 0)
    for (int j = 0; j < 4; ++j)
      if (j < 2) atomicMin(out + PROBE_LO_X + j, b[j]);
      else atomicMax(out + PROBE_LO_X + j, b[j]);
}

__global__ void k_probe_bounds(unsigned long long* out, const double* z) {
  for (int j = PROBE_LO_X; j <= PROBE_HI_Y; ++j)
    out[j] = (unsigned long long)__double_as_longlong(unordered(out[j]));
  if (z) out[PROBE_Z] = (unsigned long long)__double_as_longlong(*z);
}

// ---------------------------------------------------------------------------
// The plan of one call, from lmb_radial_intervals' rule.

struct RadialPlan {
  double x0, y0, z;     // first pixel, plane
  long long nx, ny;
  double k, aberr;
  double spacing;       // node spacing = interval width (px), a multiple of 1/64
  float inv_half;       // 2 / spacing (1/px)
  int intervals;        // capacity per particle
  int flags;
};

// Largest distance of a particle from the grid's pixels.
__host__ __device__ inline double radial_reach(double x0, double y0, long long nx,
                                               long long ny, double xp, double yp) {
  const double dx = fmax(fabs(x0 - xp), fabs(x0 + double(nx - 1) - xp));
  const double dy = fmax(fabs(y0 - yp), fabs(y0 + double(ny - 1) - yp));
  return sqrt(fma(dx, dx, dy * dy));  // the same value wherever it is compiled
}

// Intervals a particle uses: indices 0 .. count - 1 cover its pixels.
__host__ __device__ inline int radial_count(double reach, double spacing) {
  return int(reach / spacing) + 2;
}

// ---------------------------------------------------------------------------
// Nodes and polynomials: one block per (chunk of intervals, particle).
//
// One thread sums the orders of one node in FP64 (serial recurrences, bound
// by FP64 issue: ~40 FP64 instructions an order), so a block of 128 threads
// covers 112 intervals and the 8 nodes that their polynomials reach on
// either side.  Then every thread forms the polynomials of (interval,
// function) pairs, 2 x 6 x 17 FP64 FMAs each with the matrix in the constant
// bank.  The FP64 nodes are kept for the pixels that k_field_radial sums
// again in FP64.
constexpr int kNodeThreads = 128;
constexpr int kChunk = kNodeThreads - 2 * RADIAL_SIDE;

// R = float or double: the coefficients' type (double: no nodes are kept).
template <typename R, int NC>
__global__ void __launch_bounds__(kNodeThreads)
k_radial_table(RadialPlan pl, RadialMatrixN<NC> A, const lmb_sphere* __restrict__ spheres,
               const zd* __restrict__ ab, const int* __restrict__ nmax, int nmaxp,
               R* __restrict__ table, double* __restrict__ nodes) {
  extern __shared__ __align__(16) char smem[];
  double* val = reinterpret_cast<double*>(smem);  // [RADIAL_FUNCS][kNodeThreads]
  Quad<double>* rec = reinterpret_cast<Quad<double>*>(
      smem + sizeof(double) * RADIAL_FUNCS * kNodeThreads);
  const int p = blockIdx.y, i0 = blockIdx.x * kChunk;
  const lmb_sphere sp = spheres[p];
  const int count = min(pl.intervals,
                        radial_count(radial_reach(pl.x0, pl.y0, pl.nx, pl.ny,
                                                  sp.x_p, sp.y_p), pl.spacing));
  if (i0 >= count) return;  // the whole block
  const int nm = min(max(nmax[p], 0), nmaxp - 1);
  for (int n = threadIdx.x; n <= nm; n += kNodeThreads) {
    Quad<double> q[2];
    order_record<double>(ab + (size_t(p) * nmaxp + n) * 2, (const zd*)0, n, 2, q);
    rec[2 * n] = q[0];
    rec[2 * n + 1] = q[1];
  }
  __syncthreads();
  const int j = i0 - RADIAL_SIDE + int(threadIdx.x);  // node of this thread
  const int ncap = pl.intervals + 2 * RADIAL_SIDE;
  if (j < count + RADIAL_SIDE) {
    double v[RADIAL_FUNCS];
    // V and Z at the axis are limits.  FP32: the threads of nodes 0 and -1
    // take two distances near it, node -1 being the image of node 1.  FP64:
    // from the neighbours (below).
    const double step = sizeof(R) == sizeof(float) ? RADIAL_AXIS_STEP / pl.k : 0.;
    const double rho = j == 0 ? step
                       : j == -1 && step > 0. ? 2. * step : pl.spacing * double(abs(j));
    radial_field(pl.k, rho, pl.z - sp.z_p, pl.z, sp.z_p, pl.flags & LMB_BOHREN, pl.aberr, rec,
                 nm, v);
    for (int f = 0; f < RADIAL_FUNCS; ++f) val[f * kNodeThreads + threadIdx.x] = v[f];
  }
  __syncthreads();
  if (sizeof(R) == sizeof(float) && i0 == 0) {
    if (threadIdx.x < RADIAL_FUNCS) {
      double* s = val + threadIdx.x * kNodeThreads + RADIAL_SIDE;
      s[0] = (4. * s[0] - s[-1]) * (1. / 3.);
      s[-1] = s[1];
    }
    __syncthreads();
  }
  if (sizeof(R) == sizeof(double) && i0 == 0) {
    // the even function through the nodes 1..8 and -1..-8, at 0: off by at
    // most 3e-13 at this spacing
    if (threadIdx.x >= 2 && threadIdx.x < RADIAL_FUNCS) {
      double* s = val + threadIdx.x * kNodeThreads + RADIAL_SIDE;
      double sum = 0., w = 1.;
      for (int m = 1; m <= RADIAL_SIDE; ++m) {
        w *= -double(RADIAL_SIDE + 1 - m) / double(RADIAL_SIDE + m);
        sum -= 2. * w * s[m];
      }
      s[0] = sum;
    }
    __syncthreads();
  }
  if (nodes && j < count + RADIAL_SIDE) {
    // each node is written by the chunk it lies in (the ends by the outer ones)
    const int t = threadIdx.x;
    if ((t >= RADIAL_SIDE || i0 == 0) &&
        (t < kNodeThreads - RADIAL_SIDE || i0 + kChunk >= count)) {
      double* out = nodes + (size_t(p) * ncap + (j + RADIAL_SIDE)) * RADIAL_FUNCS;
      for (int f = 0; f < RADIAL_FUNCS; ++f) out[f] = val[f * kNodeThreads + t];
    }
  }
  const int n = min(kChunk, count - i0);
  for (int w = threadIdx.x; w < n * (RADIAL_FUNCS / 2); w += kNodeThreads) {
    const int f = w / n, i = w - f * n;
    const double* s = val + 2 * f * kNodeThreads + i;
    double cr[NC], ci[NC];
#pragma unroll
    for (int q = 0; q < NC; ++q) cr[q] = ci[q] = 0.;
#pragma unroll
    for (int l = 0; l < RADIAL_TAPS; ++l) {
      const double x = s[l], y = s[kNodeThreads + l];
#pragma unroll
      for (int q = 0; q < NC; ++q) {
        cr[q] = fma(A.m[q][l], x, cr[q]);
        ci[q] = fma(A.m[q][l], y, ci[q]);
      }
    }
    // re and im of a coefficient side by side
    R* out = table + (size_t(p) * pl.intervals + i0 + i) * (RADIAL_FUNCS * NC) + f * 2 * NC;
    if constexpr (sizeof(R) == sizeof(float)) {
      static_assert(sizeof(R) == sizeof(double) || NC % 2 == 0, "whole float4");
#pragma unroll
      for (int q = 0; q < NC; q += 2)
        reinterpret_cast<float4*>(out)[q / 2] =
            make_float4(float(cr[q]), float(ci[q]), float(cr[q + 1]), float(ci[q + 1]));
    } else {
#pragma unroll
      for (int q = 0; q < NC; ++q)
        reinterpret_cast<double2*>(out)[q] = make_double2(cr[q], ci[q]);
    }
  }
}

// ---------------------------------------------------------------------------
// Pixels.

// FP64 values of the marked pixels of a tile, interpolated straight from
// the FP64 nodes (17 points, off by ~1e-9 of the field): for the pixels whose FP32 value
// may be off by more than HOLO_TOL, a few per thousand.  A tile's marked
// pixels sit together, so the particles of a pixel are spread over lanes: a
// group of lanes (the next power of two from the particle count, up to the
// warp) per pixel, combined by a fixed shuffle tree.  where(entry, x, y)
// gives a list entry's position and returns its index in out.
template <typename Where>
__device__ void radial_resum64(const RadialPlan& pl, const int* list, int F, Where where,
                               const lmb_sphere* __restrict__ spheres, int pb, int pe,
                               const double* __restrict__ nodes, float* out) {
  const int ncap = pl.intervals + 2 * RADIAL_SIDE;
  const int lane = threadIdx.x & 31;
  int group = 1;
  while (group < 32 && group < pe - pb) group <<= 1;
  const int per = 32 / group, sub = lane & (group - 1);
  const int step = int(blockDim.x >> 5) * per;
  // the same trip count for every lane of a warp
  for (int f0 = int(threadIdx.x >> 5) * per; f0 < F; f0 += step) {
    const int f = f0 + lane / group;
    const bool live = f < F;
    double x, y;
    const long long pix = where(list[live ? f : F - 1], &x, &y);
    double e[6] = {0., 0., 0., 0., 0., 0.};
    for (int p = pb + sub; live && p < pe; p += group) {
      radial_point64(x - spheres[p].x_p, y - spheres[p].y_p, pl.spacing, pl.intervals,
                     reinterpret_cast<const d2*>(nodes + size_t(p) * ncap * RADIAL_FUNCS), e);
    }
    for (int o = group >> 1; o > 0; o >>= 1)
      for (int c = 0; c < 6; ++c) e[c] += __shfl_xor_sync(0xffffffffu, e[c], o);
    const zd t[3] = {mk(e[0], e[1]), mk(e[2], e[3]), mk(e[4], e[5])};
    if (live && sub == 0) out[pix] = float(intensity<double>(t));
  }
}

struct TileParticle {
  float ax, rx, ay, ry;  // first pixel minus particle: 2^-10 px part, rest
  int lo, count;         // intervals that the tile's pixels use
};

// The intervals that a tile of w x h pixels at (tx, ty) needs of a particle,
// at most room of them.
__device__ inline TileParticle tile_particle(const RadialPlan& pl, const lmb_sphere& sp,
                                             long long tx, long long ty, int w, int h,
                                             int room) {
  const double dx = pl.x0 + double(tx) - sp.x_p, dy = pl.y0 + double(ty) - sp.y_p;
  TileParticle t;
  const double ax = rint(dx * 1024.) * (1. / 1024.), ay = rint(dy * 1024.) * (1. / 1024.);
  t.ax = float(ax);
  t.rx = float(dx - ax);
  t.ay = float(ay);
  t.ry = float(dy - ay);
  // Nearest and farthest distances of the tile's pixels.  FP32 is off by at
  // most 0.01 interval at 8000 px and one interval is spare on either side;
  // in FP64 the roots and quotients, which a block starts with, made a batch
  // of 512 spheres on 201x201 pixels 155 instead of 149 us.  Past the last
  // interval of its own a particle's table is unwritten, and unused.
  const float ex = float(w - 1), ey = float(h - 1), x = float(dx), y = float(dy);
  const float nx = x > 0.f ? x : fmaxf(-(x + ex), 0.f);
  const float ny = y > 0.f ? y : fmaxf(-(y + ey), 0.f);
  const float fx = fmaxf(fabsf(x), fabsf(x + ex)), fy = fmaxf(fabsf(y), fabsf(y + ey));
  const float per = 0.5f * pl.inv_half;
  const int last = pl.intervals - 1;
  t.lo = max(0, min(last, int(sqrtf(nx * nx + ny * ny) * per) - 1));
  const int hi = min(last + 1, int(sqrtf(fx * fx + fy * fy) * per) + 3);
  t.count = max(1, min(hi - t.lo, room));
  return t;
}

constexpr int kTile = 32;          // tiles of 32 x 32 pixels
constexpr int kPixThreads = 256;   // a 2x2 group each
constexpr int kTileGroup = 32;     // particles whose TileParticle is staged at once

// One block per 32x32-pixel tile and item, 4 pixels per thread.  For each
// particle the intervals that the tile needs (its distances span at most
// 43.9 px, ~70 intervals of 144 bytes) are copied to shared memory, kStages
// - 1 copies ahead, and every pixel reads its interval's coefficients (9
// LDS.128) and evaluates the three complex polynomials with (re, im) in the
// two lanes of packed FP32, so that the coefficients come paired from memory
// and only t is duplicated.  A pixel's value depends on its position alone,
// not on its neighbours (groups of pixels that share an interval would read
// less, but differ from the same pixel in a list by their rounding).
// A 1280x1024 frame of 16 spheres: 121 us, 72% of the shared-memory pipe's
// peak (144 bytes a pixel and particle); with the orders summed at every
// pixel (k_field_pair) 1.44 ms.
constexpr int kStages = 3;
constexpr int kStepX = 8, kStepY = 4;
template <bool kHolo>
__global__ void __launch_bounds__(kPixThreads, 2)
k_field_radial(RadialPlan pl, const lmb_sphere* __restrict__ spheres,
               const int* __restrict__ item_start, const float* __restrict__ table,
               const double* __restrict__ nodes, int buffer, void* out) {
  extern __shared__ __align__(16) float4 buf[];  // [kStages][buffer]
  __shared__ TileParticle s_tp[kTileGroup];
  __shared__ int s_marked;
  const int item = blockIdx.z;
  const int pb = item_start[item], pe = item_start[item + 1];
  const long long tx = (long long)blockIdx.x * kTile, ty = (long long)blockIdx.y * kTile;
  // A warp takes 16x8 pixels as four patches of 8x4, a pixel of each per
  // lane: columns cx and cx + kStepX, rows cy and cy + kStepY.  The eight
  // lanes of a quarter warp, whose LDS.128 go together, sit on 4x2 pixels,
  // whose distances span less than eight intervals: no bank conflicts.
  const int lane_id = threadIdx.x & 31, warp_id = threadIdx.x >> 5;
  const int cx = 16 * (warp_id & 1) + 4 * ((lane_id >> 3) & 1) + (lane_id & 3);
  const int cy = 8 * (warp_id >> 1) + 2 * (lane_id >> 4) + ((lane_id >> 2) & 1);
  // Tiles at the image's far edges: only the warps with pixels in the image
  // work (a 201x201 image spans 49 tiles, a fifth of whose pixels lie outside:
  // 164 -> 155 us for 128 such images of 4 spheres).
  const int tw = int(min((long long)kTile, pl.nx - tx));
  const int th = int(min((long long)kTile, pl.ny - ty));
  const bool inside = 16 * (warp_id & 1) < tw && 8 * (warp_id >> 1) < th;
  const float inv_spacing = float(1. / pl.spacing), spacing = float(pl.spacing);
  constexpr int RQ = RADIAL_REC / 4;  // float4 per interval
  // field sums (re, im) and error bounds of the pixels (2 row + column)
  f2 ex[4], ey[4], ez[4];
  float m1[4];
  for (int q = 0; q < 4; ++q) {
    ex[q] = ey[q] = ez[q] = pk(0.f, 0.f);
    m1[q] = 0.f;
  }
  for (int g0 = pb; g0 < pe; g0 += kTileGroup) {
    const int G = min(kTileGroup, pe - g0);
    __syncthreads();  // the previous group's data is no longer read
    if (threadIdx.x < G) {
      const TileParticle t = tile_particle(pl, spheres[g0 + threadIdx.x], tx, ty, tw, th,
                                           buffer / RQ);
      s_tp[threadIdx.x] = t;
    }
    __syncthreads();
    // a commit per particle, empty past the last, so that the wait below
    // always leaves the kStages - 2 newest copies in flight
    auto fetch = [&](int g) {
      if (g < G) {
        const TileParticle t = s_tp[g];
        const float4* src = reinterpret_cast<const float4*>(table) +
                            (size_t(g0 + g) * pl.intervals + t.lo) * RQ;
        float4* dst = buf + (g % kStages) * buffer;
        for (int i = threadIdx.x; i < t.count * RQ; i += kPixThreads)
          __pipeline_memcpy_async(dst + i, src + i, 16);
      }
      __pipeline_commit();
    };
    for (int g = 0; g < kStages - 1; ++g) fetch(g);
    for (int g = 0; g < G; ++g) {
      __pipeline_wait_prior(kStages - 2);
      // copy g has landed, and everyone is done with the buffer that the
      // next fetch refills (that of particle g - 1)
      __syncthreads();
      fetch(g + kStages - 1);
      if (!inside) continue;
      const TileParticle t = s_tp[g];
      const float4* rec = buf + (g % kStages) * buffer;
      // column and row terms
      const f2 X = padd(pk(t.ax, t.ax), pk(float(cx), float(cx + kStepX)));
      const f2 px = pmul(X, X);
      const f2 lx = pfma(pk(2.f * t.rx, 2.f * t.rx), padd(X, pk(0.5f * t.rx, 0.5f * t.rx)),
                         pfma(X, X, pneg(px)));
      const f2 Xr = padd(X, pk(t.rx, t.rx)), X2 = padd(Xr, Xr);
      const f2 Y = padd(pk(t.ay, t.ay), pk(float(cy), float(cy + kStepY)));
      const f2 qy = pmul(Y, Y);
      const f2 ly = pfma(pk(2.f * t.ry, 2.f * t.ry), padd(Y, pk(0.5f * t.ry, 0.5f * t.ry)),
                         pfma(Y, Y, pneg(qy)));
      const f2 Yr = padd(Y, pk(t.ry, t.ry));
      RadialDistance d[2];
      d[0] = radial_distance(px, lx, pk(qy.x, qy.x), pk(ly.x, ly.x));
      d[1] = radial_distance(px, lx, pk(qy.y, qy.y), pk(ly.y, ly.y));
      auto lane = [](f2 v, int q) { return (q & 1) ? v.y : v.x; };
      f2 c2[2], s2[2];
      float tq[4];
      const float4* r4[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float r0 = lane(d[q >> 1].r0, q);
        const int i = min(max(__float2int_rn(r0 * inv_spacing) - t.lo, 0), t.count - 1);
        tq[q] = ((r0 - float(i + t.lo) * spacing) + lane(d[q >> 1].corr, q)) * pl.inv_half;
        r4[q] = rec + i * RQ;
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const f2 yr = r ? pk(Yr.y, Yr.y) : pk(Yr.x, Yr.x);
        c2[r] = pmul(psub(Xr, yr), padd(Xr, yr));
        s2[r] = pmul(X2, yr);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const f2 u = radial_eval(r4[q], tq[q]);
        const f2 v = radial_eval(r4[q] + RQ / 3, tq[q]);
        const f2 w = radial_eval(r4[q] + 2 * (RQ / 3), tq[q]);
        const float c = lane(c2[q >> 1], q), s = lane(s2[q >> 1], q), x = lane(Xr, q);
        ex[q] = pfma(pk(c, c), v, padd(ex[q], u));
        ey[q] = pfma(pk(s, s), v, ey[q]);
        ez[q] = pfma(pk(x, x), w, ez[q]);
        if (kHolo) m1[q] += radial_bound(u, v, w, c, s, x);
      }
    }
  }
  int mark = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const long long col = tx + cx + (q & 1) * kStepX;
    const long long row = ty + cy + (q >> 1) * kStepY;
    if (col >= pl.nx || row >= pl.ny) continue;
    const long long pix = row * pl.nx + col;
    cplx<float> e[3] = {mk(ex[q].x, ex[q].y), mk(ey[q].x, ey[q].y), mk(ez[q].x, ez[q].y)};
    const long long npts = pl.nx * pl.ny;
    if (kHolo) {
      const float h = intensity<float>(e);
      float* o = reinterpret_cast<float*>(out) + size_t(item) * npts;
      if (radial_needs_fp64(h, m1[q]))
        mark |= 1 << q;
      else
        o[pix] = h;
    } else {
      float2* o = reinterpret_cast<float2*>(out) + size_t(item) * 3 * npts;
      for (int c = 0; c < 3; ++c) o[c * npts + pix] = make_float2(e[c].re, e[c].im);
    }
  }
  if (kHolo) {
    if (threadIdx.x == 0) s_marked = 0;
    // also the barrier after which the table buffers may be overwritten
    if (!__syncthreads_or(mark)) return;
    int* list = reinterpret_cast<int*>(buf);  // up to kTile * kTile entries
    for (int q = 0; q < 4; ++q)
      if (mark >> q & 1)
        list[atomicAdd(&s_marked, 1)] =
            (cy + (q >> 1) * kStepY) * kTile + cx + (q & 1) * kStepX;
    __syncthreads();
    auto where = [&](int l, double* x, double* y) {
      const long long col = tx + l % kTile, row = ty + l / kTile;
      *x = pl.x0 + double(col);
      *y = pl.y0 + double(row);
      return row * pl.nx + col;
    };
    radial_resum64(pl, list, s_marked, where, spheres, pb, pe, nodes,
                   reinterpret_cast<float*>(out) + size_t(item) * pl.nx * pl.ny);
  }
}

// FP64 images: the same in double, tiles of 32 x 16 pixels, two pixels (rows
// y and y + 4) per thread, 8x8 pixels per warp.  27 LDS.128 a pixel and
// particle: bound by shared memory (60% of its peak; the rest is barriers,
// two tables of 48 KB in flight).  1279x1023 px of 5 spheres: 164 us, the
// call 955 -> 197 us against sums at every pixel.
constexpr int kTileH64 = 16;
template <bool kHolo>
__global__ void __launch_bounds__(kPixThreads, 2)
k_field_radial64(RadialPlan pl, const lmb_sphere* __restrict__ spheres,
                 const int* __restrict__ item_start, const double* __restrict__ table,
                 int buffer, int stages, void* out) {
  extern __shared__ __align__(16) double2 buf64[];  // [stages][buffer]
  __shared__ TileParticle s_tp[kTileGroup];
  constexpr int RQ = RADIAL_REC64 / 2;  // double2 per interval
  const int item = blockIdx.z;
  const int pb = item_start[item], pe = item_start[item + 1];
  const long long tx = (long long)blockIdx.x * kTile, ty = (long long)blockIdx.y * kTileH64;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cx = 8 * (warp & 3) + 4 * ((lane >> 3) & 1) + (lane & 3);
  const int cy = 8 * (warp >> 2) + 2 * (lane >> 4) + ((lane >> 2) & 1);
  const double inv_spacing = 1. / pl.spacing, inv_half = 2. / pl.spacing;
  const double x0 = pl.x0 + double(tx + cx), y0 = pl.y0 + double(ty + cy);
  const int tw = int(min((long long)kTile, pl.nx - tx));
  const int th = int(min((long long)kTileH64, pl.ny - ty));
  const bool inside = 8 * (warp & 3) < tw && 8 * (warp >> 2) < th;
  double2 e[2][3];
  for (int q = 0; q < 2; ++q)
    for (int c = 0; c < 3; ++c) e[q][c] = make_double2(0., 0.);
  for (int g0 = pb; g0 < pe; g0 += kTileGroup) {
    const int G = min(kTileGroup, pe - g0);
    __syncthreads();  // the previous group's data is no longer read
    if (threadIdx.x < G)
      s_tp[threadIdx.x] = tile_particle(pl, spheres[g0 + threadIdx.x], tx, ty, tw, th,
                                        buffer / RQ);
    __syncthreads();
    auto fetch = [&](int g) {
      if (g < G) {
        const TileParticle t = s_tp[g];
        const double2* src = reinterpret_cast<const double2*>(table) +
                             (size_t(g0 + g) * pl.intervals + t.lo) * RQ;
        double2* dst = buf64 + (g % stages) * buffer;
        for (int i = threadIdx.x; i < t.count * RQ; i += kPixThreads)
          __pipeline_memcpy_async(dst + i, src + i, 16);
      }
      __pipeline_commit();
    };
    if (stages > 1) fetch(0);
    for (int g = 0; g < G; ++g) {
      if (stages > 1) {
        fetch(g + 1);
        __pipeline_wait_prior(1);
      } else {
        fetch(g);
        __pipeline_wait_prior(0);
      }
      __syncthreads();  // copy g has landed
      const TileParticle t = s_tp[g];
      const double2* rec = buf64 + (g % stages) * buffer;
      const double dx = x0 - spheres[g0 + g].x_p, dy0 = y0 - spheres[g0 + g].y_p;
#pragma unroll
      for (int q = 0; q < 2 && inside; ++q) {
        const double dy = dy0 + 4. * q;
        const double rho = sqrt(fma(dx, dx, dy * dy));
        const int i = min(max(__double2int_rn(rho * inv_spacing) - t.lo, 0), t.count - 1);
        const double u = (rho - double(i + t.lo) * pl.spacing) * inv_half;
        const double2* r = rec + i * RQ;
        const double c2 = (dx - dy) * (dx + dy), s2 = 2. * dx * dy;
        double2 v[3];
#pragma unroll
        for (int f = 0; f < 3; ++f) {
          v[f] = r[f * RADIAL_COEFS64 + RADIAL_COEFS64 - 1];
#pragma unroll
          for (int j = RADIAL_COEFS64 - 2; j >= 0; --j) {
            const double2 c = r[f * RADIAL_COEFS64 + j];
            v[f].x = fma(v[f].x, u, c.x);
            v[f].y = fma(v[f].y, u, c.y);
          }
        }
        e[q][0].x = fma(c2, v[1].x, e[q][0].x + v[0].x);
        e[q][0].y = fma(c2, v[1].y, e[q][0].y + v[0].y);
        e[q][1].x = fma(s2, v[1].x, e[q][1].x);
        e[q][1].y = fma(s2, v[1].y, e[q][1].y);
        e[q][2].x = fma(dx, v[2].x, e[q][2].x);
        e[q][2].y = fma(dx, v[2].y, e[q][2].y);
      }
      __syncthreads();  // this buffer is refilled from here on
    }
  }
  const long long npts = pl.nx * pl.ny;
  for (int q = 0; q < 2; ++q) {
    const long long col = tx + cx, row = ty + cy + 4 * q;
    if (col >= pl.nx || row >= pl.ny) continue;
    const long long pix = row * pl.nx + col;
    if (kHolo) {
      const zd t[3] = {mk(e[q][0].x, e[q][0].y), mk(e[q][1].x, e[q][1].y),
                       mk(e[q][2].x, e[q][2].y)};
      reinterpret_cast<double*>(out)[size_t(item) * npts + pix] = intensity<double>(t);
    } else {
      double2* o = reinterpret_cast<double2*>(out) + size_t(item) * 3 * npts;
      for (int c = 0; c < 3; ++c) o[c * npts + pix] = e[q][c];
    }
  }
}

// The same from an explicit pixel list in the plane (points [3][npts]; the
// plan's grid is its bounding box): one thread per pixel, the coefficients
// of its own intervals read through the caches.  The values are the grid
// kernel's to the rounding of the polynomials.
constexpr int kListThreads = 128;
template <bool kHolo>
__global__ void __launch_bounds__(kListThreads)
k_points_radial(RadialPlan pl, const double* __restrict__ points, long long npts,
                const lmb_sphere* __restrict__ spheres, const int* __restrict__ item_start,
                const float* __restrict__ table, const double* __restrict__ nodes, void* out) {
  __shared__ int s_list[kListThreads], s_marked;
  const int item = blockIdx.y;
  const int pb = item_start[item], pe = item_start[item + 1];
  const long long base = (long long)blockIdx.x * kListThreads, pix = base + threadIdx.x;
  bool mark = false;
  if (pix < npts) {
    const double x = points[pix], y = points[npts + pix];
    const float inv_spacing = float(1. / pl.spacing), spacing = float(pl.spacing);
    RadialSum r = {pk(0.f, 0.f), pk(0.f, 0.f), pk(0.f, 0.f), 0.f};
    for (int p = pb; p < pe; ++p)
      radial_point(x - spheres[p].x_p, y - spheres[p].y_p, inv_spacing, spacing, pl.inv_half,
                   pl.intervals,
                   reinterpret_cast<const f4*>(table + size_t(p) * pl.intervals * RADIAL_REC),
                   r);
    const cplx<float> e[3] = {mk(r.ex.x, r.ex.y), mk(r.ey.x, r.ey.y), mk(r.ez.x, r.ez.y)};
    if (kHolo) {
      const float h = intensity<float>(e);
      mark = radial_needs_fp64(h, r.m1);
      if (!mark) reinterpret_cast<float*>(out)[size_t(item) * npts + pix] = h;
    } else {
      float2* o = reinterpret_cast<float2*>(out) + size_t(item) * 3 * npts;
      for (int c = 0; c < 3; ++c) o[c * npts + pix] = make_float2(e[c].re, e[c].im);
    }
  }
  if (kHolo) {
    if (threadIdx.x == 0) s_marked = 0;
    if (!__syncthreads_or(mark)) return;
    if (mark) s_list[atomicAdd(&s_marked, 1)] = threadIdx.x;
    __syncthreads();
    auto where = [&](int l, double* x, double* y) {
      *x = points[base + l];
      *y = points[npts + base + l];
      return base + l;
    };
    radial_resum64(pl, s_list, s_marked, where, spheres, pb, pe, nodes,
                   reinterpret_cast<float*>(out) + size_t(item) * npts);
  }
}

constexpr size_t kSmemLimit = size_t(200) * 1024;

// float4 of the intervals that a tile's pixels can span, with the margins of
// TileParticle.
size_t radial_buffer(double spacing) {
  return (size_t((kTile - 1) * 1.4142135623730951 / spacing) + 7) * (RADIAL_REC / 4);
}

size_t up256(size_t v) { return (v + 255) / 256 * 256; }

size_t radial_buffer64(double spacing) {  // double2
  const double w = kTile - 1, h = kTileH64 - 1;
  return (size_t(sqrt(w * w + h * h) / spacing) + 7) * (RADIAL_REC64 / 2);
}

size_t table_bytes(int nparticles, int intervals, bool fp64) {
  const size_t rec = fp64 ? sizeof(double) * RADIAL_REC64 : sizeof(float) * RADIAL_REC;
  return up256(rec * size_t(nparticles) * size_t(intervals));
}

size_t node_bytes(int nparticles, int intervals) {
  return up256(sizeof(double) * RADIAL_FUNCS * size_t(nparticles) *
               (size_t(intervals) + 2 * RADIAL_SIDE));
}

int grid_common(bool holo, const lmb_grid* grid, const lmb_sphere* spheres,
                const double* points, long long npts, const int* item_start, int nitems,
                int nparticles, int intervals, const double* ab, const int* nmax,
                int nmax_cap, double k, int flags, double aberr, void* out, void* workspace, size_t workspace_bytes,
                void* stream) {
  if (nitems < 0 || nparticles < 0 || nmax_cap < 1 || nmax_cap > LMB_NMAX_LIMIT)
    return LMB_ERR_ARG;
  if (!grid || grid->nx < 0 || grid->ny < 0 || npts < 0) return LMB_ERR_ARG;
  // the pixel kernels write nx * ny values an item, the output holds npts
  if (!points && !grid_holds(grid, npts)) return LMB_ERR_ARG;
  if (nitems == 0 || grid->nx == 0 || grid->ny == 0 || (points && npts == 0))
    return LMB_OK;
  if (!spheres || !item_start || !ab || !nmax || !out || intervals < 1) return LMB_ERR_ARG;
  const bool fp64 = flags & LMB_FP64;
  if (!(flags & LMB_CARTESIAN) || (fp64 && points)) return LMB_ERR_UNSUPPORTED;
  if (!isfinite(aberr) || !(k > 0.) || nparticles > 65535 || nitems > 65535)
    return LMB_ERR_ARG;
  const long long tx = (grid->nx + kTile - 1) / kTile, ty = (grid->ny + kTile - 1) / kTile;
  if (tx > 0x7fffffffLL || ty > 65535 || (npts + kListThreads - 1) / kListThreads > 0x7fffffffLL)
    return LMB_ERR_ARG;
  if (!workspace || workspace_bytes < lmb_radial_workspace_bytes(nparticles, intervals, flags))
    return LMB_ERR_WORKSPACE;
  RadialPlan pl;
  pl.spacing = radial_spacing(k, fp64);
  if (!(pl.spacing > 0.)) return LMB_ERR_UNSUPPORTED;
  pl.x0 = grid->x0;
  pl.y0 = grid->y0;
  pl.z = grid->z;
  pl.nx = grid->nx;
  pl.ny = grid->ny;
  pl.k = k;
  pl.aberr = aberr;
  pl.inv_half = float(2. / pl.spacing);
  pl.intervals = intervals;
  pl.flags = flags;
  float* table = reinterpret_cast<float*>(workspace);
  double* table64 = reinterpret_cast<double*>(workspace);
  double* nodes = reinterpret_cast<double*>(reinterpret_cast<char*>(workspace) +
                                            table_bytes(nparticles, intervals, false));
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (nparticles > 0) {
    const size_t smem = sizeof(double) * RADIAL_FUNCS * kNodeThreads +
                        sizeof(Quad<double>) * 2 * (size_t(nmax_cap) + 1);
    const dim3 g(unsigned((intervals + kChunk - 1) / kChunk), unsigned(nparticles));
    const zd* abz = reinterpret_cast<const zd*>(ab);
    if (fp64) {
      auto fn = k_radial_table<double, RADIAL_COEFS64>;
      LMB_CK(smem_attr((const void*)fn, smem));
      fn<<<g, kNodeThreads, smem, st>>>(pl, radial_matrix<RADIAL_COEFS64>(), spheres, abz, nmax,
                                        nmax_cap + 1, table64, nullptr);
    } else {
      auto fn = k_radial_table<float, RADIAL_COEFS>;
      LMB_CK(smem_attr((const void*)fn, smem));
      fn<<<g, kNodeThreads, smem, st>>>(pl, radial_matrix(), spheres, abz, nmax, nmax_cap + 1,
                                        table, nodes);
    }
    LMB_CK(cudaGetLastError());
  }
  if (fp64) {
    const long long rows = (grid->ny + kTileH64 - 1) / kTileH64;
    const size_t buffer = radial_buffer64(pl.spacing);
    // two buffers, or one where k is so large that they do not fit
    const int stages = 2 * sizeof(double2) * buffer <= kSmemLimit ? 2 : 1;
    const size_t smem = stages * sizeof(double2) * buffer;
    auto fn = holo ? k_field_radial64<true> : k_field_radial64<false>;
    if (smem > kSmemLimit || rows > 65535) return LMB_ERR_UNSUPPORTED;
    LMB_CK(smem_attr((const void*)fn, smem));
    const dim3 g{unsigned(tx), unsigned(rows), unsigned(nitems)};
    fn<<<g, kPixThreads, smem, st>>>(pl, spheres, item_start, table64, int(buffer),
                                   stages, out);
    LMB_CK(cudaGetLastError());
    return LMB_OK;
  }
  if (points) {
    auto list = holo ? k_points_radial<true> : k_points_radial<false>;
    const dim3 g{unsigned((npts + kListThreads - 1) / kListThreads), unsigned(nitems)};
    list<<<g, kListThreads, 0, st>>>(pl, points, npts, spheres, item_start, table, nodes, out);
    LMB_CK(cudaGetLastError());
    return LMB_OK;
  }
  const size_t buffer = radial_buffer(pl.spacing);
  const size_t smem = std::max(kStages * sizeof(float4) * buffer,
                               sizeof(int) * size_t(kTile * kTile));
  auto fn = holo ? k_field_radial<true> : k_field_radial<false>;
  if (smem > kSmemLimit) return LMB_ERR_UNSUPPORTED;
  LMB_CK(smem_attr((const void*)fn, smem));
  const dim3 g{unsigned(tx), unsigned(ty), unsigned(nitems)};
  fn<<<g, kPixThreads, smem, st>>>(pl, spheres, item_start, table, nodes, int(buffer), out);
  LMB_CK(cudaGetLastError());
  return LMB_OK;
}

int probe(const double* coords, long long npts, unsigned long long* out, bool z,
          void* stream) {
  if (npts < 1 || !coords || !out) return LMB_ERR_ARG;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const unsigned blocks = unsigned(std::min<long long>((npts + 255) / 256, 1184));
  k_probe_init<<<1, 1, 0, st>>>(npts, out);
  k_probe_row<<<blocks, 256, 0, st>>>(coords, npts, out);
  k_probe_check<<<blocks, 256, 0, st>>>(coords, npts, out);
  k_probe_bounds<<<1, 1, 0, st>>>(out, z ? coords + 2 * npts : nullptr);
  LMB_CK(cudaGetLastError());
  return LMB_OK;
}

}  // namespace

extern "C" {

int lmb_grid_probe(const double* coords, long long npts, unsigned long long* out,
                   void* stream) {
  return probe(coords, npts, out, false, stream);
}

int lmb_plane_probe(const double* coords, long long npts, unsigned long long* out,
                    void* stream) {
  return probe(coords, npts, out, true, stream);
}

int lmb_radial_intervals(const lmb_grid* grid, long long npts, const lmb_sphere* spheres,
                         int n, double k, double magnification, int flags, double aberration) {
  if (!grid || !spheres || n < 1 || grid->nx < 1 || grid->ny < 1) return 0;
  if (!(flags & LMB_CARTESIAN)) return 0;
  const bool fp64 = flags & LMB_FP64;
  if (!(k > 0.) || !isfinite(k) || !(magnification > 0.) || !isfinite(aberration)) return 0;
  if (!isfinite(grid->x0) || !isfinite(grid->y0) || !isfinite(grid->z)) return 0;
  const double spacing = radial_spacing(k, fp64);
  if (!(spacing > 0.)) return 0;
  // a tile's intervals fit in shared memory
  if ((fp64 ? sizeof(double2) * radial_buffer64(spacing)
            : kStages * sizeof(float4) * radial_buffer(spacing)) > kSmemLimit)
    return 0;
  if (fp64 && grid->ny > 65535LL * kTileH64) return 0;
  double far = 0.;
  for (int i = 0; i < n; ++i) {
    const lmb_sphere& s = spheres[i];
    const double reach = radial_reach(grid->x0, grid->y0, grid->nx, grid->ny, s.x_p, s.y_p);
    const double dz = fabs(grid->z - s.z_p);
    // offsets up to 8192 px split exactly in FP32 (radial_distance)
    if (!(reach < 8000.) || !(s.a_p > 0.) || !isfinite(s.z_p)) return 0;
    if (!radial_clear(k, dz, s.a_p / magnification, fp64)) return 0;
    // the aberration's phase turns by at most |c| / (2 |z_p|) per pixel, at
    // rho = |z_p|, where the field's own band ends at 0.7 k
    if (aberration != 0. && !(0.5 * fabs(aberration) <= 0.2 * k * fabs(s.z_p))) return 0;
    if (reach > far) far = reach;
  }
  const int count = radial_count(far, spacing);
  // A node costs about as much as two pixels' direct sums.
  if (double(npts) < 2. * (count + 2 * RADIAL_SIDE))
    return 0;
  return count;
}

size_t lmb_radial_workspace_bytes(int nparticles, int intervals, int flags) {
  if (nparticles < 0 || intervals < 1) return 0;
  if (flags & LMB_FP64) return table_bytes(nparticles, intervals, true);
  return table_bytes(nparticles, intervals, false) + node_bytes(nparticles, intervals);
}

int lmb_field_grid(const lmb_grid* grid, const double* points, long long npts,
                   const lmb_sphere* spheres, const int* item_start,
                   int nitems, int nparticles, int intervals, const double* ab,
                   const int* nmax, int nmax_cap, double k, int flags, double aberration,
                   void* out, void* workspace, size_t workspace_bytes, void* stream) {
  return grid_common(false, grid, spheres, points, npts, item_start, nitems, nparticles, intervals, ab,
                     nmax, nmax_cap, k, flags, aberration, out, workspace, workspace_bytes,
                     stream);
}

int lmb_hologram_grid(const lmb_grid* grid, const double* points, long long npts,
                      const lmb_sphere* spheres, const int* item_start,
                      int nitems, int nparticles, int intervals, const double* ab,
                      const int* nmax, int nmax_cap, double k, int flags, double aberration,
                      void* out, void* workspace, size_t workspace_bytes, void* stream) {
  return grid_common(true, grid, spheres, points, npts, item_start, nitems, nparticles, intervals, ab,
                     nmax, nmax_cap, k, flags, aberration, out, workspace, workspace_bytes,
                     stream);
}

}  // extern "C"
