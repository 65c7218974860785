// adjoint.cu - gradients of a per-pixel loss L(depth, shade) with respect to
// the formula parameters (Mandelbulb power; Mandelbox scale and min radius
// squared) and the camera (position at fixed view angles, yaw).
//
// Only the forward hit depth t per pixel is stored.  The backward pass
// recomputes, per hit pixel, the distance estimate at the hit point and at
// the six central-difference normal samples of CalculateNormals
// (src/shader_calculate_normals.cpp:44-79) in forward-mode dual numbers
// carrying six tangents (power, scale, mR2, x, y, z); the formula iteration
// follows Compute<calcModeNormal> (src/compute_fractal.cpp:175-321) and the
// formulas (fractal_mandelbulb.cpp:29-43, fractal_mandelbox.cpp:66-107) in the
// reference's order of operations.
//
// Depth: the hit t solves F(t) = dist(o + t d) - thr(t) = 0 with
// thr(t) = c0 * |o - p| = c0 * t |d| (CalcDistThresh, render_worker.cpp:653-679),
// so by the implicit function theorem
//   dt/dθ = -(∂dist/∂θ + ∇dist·∂p/∂θ|_t) / (∇dist·d - c0 |d|).
// Pixels whose stored depth is not a root of F (the refinement ended on a
// jump of the distance estimate) contribute nothing.
// Shade: the Lambert term s = N·L of the normal N = g/|g|, g_a = dist(p + δe_a)
// - dist(p - δe_a), δ = thr * smoothness, differentiated through p(θ) and δ(θ).
// A distance estimate whose orbit does not escape (a sample inside the set)
// is taken as constant: its value is ~0 and its exact derivative through
// dozens of chaotic iterations is noise.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "mbr_internal.h"
#include "pixel_ops.cuh"

namespace mbr {

// The tangents a formula's estimate carries: the point, and the Mandelbulb's
// power or the Mandelbox's scale and squared minimum radius.
enum { TN_X = 0, TN_Y, TN_Z, TN_P0, TN_P1 };
template <bool BULB>
struct Tangents {
  static constexpr int n = BULB ? 4 : 5;
};

template <class T, int TN>
struct Dn {
  T v;
  T d[TN];
};

template <int TN, class T>
__device__ __forceinline__ Dn<T, TN> dconst(T v) {
  Dn<T, TN> r;
  r.v = v;
#pragma unroll
  for (int i = 0; i < TN; i++) r.d[i] = T(0);
  return r;
}
template <int TN, class T>
__device__ __forceinline__ Dn<T, TN> dseed(T v, int k) {
  Dn<T, TN> r = dconst<TN>(v);
  if (k >= 0) r.d[k] = T(1);
  return r;
}
template <class T, int TN>
__device__ __forceinline__ Dn<T, TN> operator+(const Dn<T, TN> &a, const Dn<T, TN> &b) {
  Dn<T, TN> r;
  r.v = a.v + b.v;
#pragma unroll
  for (int i = 0; i < TN; i++) r.d[i] = a.d[i] + b.d[i];
  return r;
}
template <class T, int TN>
__device__ __forceinline__ Dn<T, TN> operator-(const Dn<T, TN> &a, const Dn<T, TN> &b) {
  Dn<T, TN> r;
  r.v = a.v - b.v;
#pragma unroll
  for (int i = 0; i < TN; i++) r.d[i] = a.d[i] - b.d[i];
  return r;
}
template <class T, int TN>
__device__ __forceinline__ Dn<T, TN> operator*(const Dn<T, TN> &a, const Dn<T, TN> &b) {
  Dn<T, TN> r;
  r.v = a.v * b.v;
#pragma unroll
  for (int i = 0; i < TN; i++) r.d[i] = a.d[i] * b.v + a.v * b.d[i];
  return r;
}
template <class T, int TN>
__device__ __forceinline__ Dn<T, TN> operator/(const Dn<T, TN> &a, const Dn<T, TN> &b) {
  Dn<T, TN> r;
  r.v = a.v / b.v;
  const T ib2 = T(1) / (b.v * b.v);
#pragma unroll
  for (int i = 0; i < TN; i++) r.d[i] = (a.d[i] * b.v - a.v * b.d[i]) * ib2;
  return r;
}
template <class T, int TN>
__device__ __forceinline__ Dn<T, TN> operator+(const Dn<T, TN> &a, T b) {
  Dn<T, TN> r = a;
  r.v = a.v + b;
  return r;
}
template <class T, int TN>
__device__ __forceinline__ Dn<T, TN> operator-(const Dn<T, TN> &a, T b) {
  Dn<T, TN> r = a;
  r.v = a.v - b;
  return r;
}
template <class T, int TN>
__device__ __forceinline__ Dn<T, TN> operator*(const Dn<T, TN> &a, T b) {
  Dn<T, TN> r;
  r.v = a.v * b;
#pragma unroll
  for (int i = 0; i < TN; i++) r.d[i] = a.d[i] * b;
  return r;
}
template <class T, int TN>
__device__ __forceinline__ Dn<T, TN> neg(const Dn<T, TN> &a) {
  return a * T(-1);
}
template <class T, int TN>
__device__ __forceinline__ Dn<T, TN> chain(const Dn<T, TN> &a, T fv, T dfa) {
  Dn<T, TN> r;
  r.v = fv;
#pragma unroll
  for (int i = 0; i < TN; i++) r.d[i] = dfa * a.d[i];
  return r;
}
template <class T, int TN>
__device__ __forceinline__ Dn<T, TN> dsqrt(const Dn<T, TN> &a) {
  const T s = m_sqrt(a.v);
  return chain(a, s, s > T(0) ? T(0.5) / s : T(0));
}
template <class T, int TN>
__device__ __forceinline__ Dn<T, TN> dabs(const Dn<T, TN> &a) {
  return a.v < T(0) ? neg(a) : a;
}
template <class T, int TN>
__device__ __forceinline__ Dn<T, TN> dlog(const Dn<T, TN> &a) {
  return chain(a, m_log(a.v), T(1) / a.v);
}

template <class T, int TN>
__device__ __forceinline__ Dn<T, TN> dlen3(const Dn<T, TN> &x, const Dn<T, TN> &y, const Dn<T, TN> &z) {
  return dsqrt(x * x + y * y + z * z);
}

// The distance estimate of a non-hybrid Mandelbulb or Mandelbox scene in
// dual numbers: Compute<calcModeNormal> + CalculateDistanceSimple.
template <class T, bool BULB>
__device__ Dn<T, Tangents<BULB>::n> de_dual(const DevScene &sc, T x, T y, T z, T detail) {
  constexpr int TN = Tangents<BULB>::n;
  typedef Dn<T, TN> Dual;
  const Dual px = dseed<TN>(x, TN_X), py = dseed<TN>(y, TN_Y), pz = dseed<TN>(z, TN_Z);
  const DevSlot &s = sc.slot[0];
  const int maxN = sc.formula_maxiter;
  Dual zx = px, zy = py, zz = pz;
  const Dual cx = zx * T(sc.cmul[0]), cy = zy * T(sc.cmul[1]), cz = zz * T(sc.cmul[2]);
  Dual r = dlen3(zx, zy, zz);
  Dual DE = dconst<TN>(T(1));
  const T bailout = T(s.d[P_BAILOUT]);
  // parameters with tangents
  const Dual power = dseed<TN>(T(s.d[P_POWER]), BULB ? TN_P0 : -1);
  const Dual scale = dseed<TN>(T(s.d[P_MB_SCALE]), BULB ? -1 : TN_P0);
  const Dual mR2 = dseed<TN>(T(s.d[P_MB_MR2]), BULB ? -1 : TN_P1);
  const Dual fR2 = dconst<TN>(T(s.d[P_MB_FR2]));
  const Dual factor1 = fR2 / mR2;
  const T limit = T(s.d[P_MB_LIMIT]), value = T(s.d[P_MB_VALUE]);
  int i;
  bool escaped = false;
  for (i = 0; i < maxN; i++) {
    if (BULB) {
      // th0 = asin(z/r) + beta; ph0 = atan2(y, x) + alpha
      const Dual q = zz / r;
      Dual th0 = chain(q, m_asin(q.v), T(1) / m_sqrt(T(1) - q.v * q.v)) + T(s.d[P_BETA]);
      Dual ph0;
      {
        const T den = zx.v * zx.v + zy.v * zy.v;
        ph0.v = m_atan2(zy.v, zx.v);
#pragma unroll
        for (int k = 0; k < TN; k++) ph0.d[k] = (zx.v * zy.d[k] - zy.v * zx.d[k]) / den;
        ph0 = ph0 + T(s.d[P_ALPHA]);
      }
      // rp = r^(power-1): d = (p-1) r^(p-2) dr + r^(p-1) ln r dp
      const Dual pm1 = power - T(1);
      Dual rp;
      {
        const T v = m_pow(r.v, pm1.v);
        const T dr = pm1.v * m_pow(r.v, pm1.v - T(1));
        const T dp = r.v > T(0) ? v * m_log(r.v) : T(0);
        rp.v = v;
#pragma unroll
        for (int k = 0; k < TN; k++) rp.d[k] = dr * r.d[k] + dp * pm1.d[k];
      }
      const Dual th = th0 * power, ph = ph0 * power;
      T sth, cth, sph, cph;
      m_sincos(th.v, &sth, &cth);
      m_sincos(ph.v, &sph, &cph);
      const Dual Cth = chain(th, cth, -sth), Sth = chain(th, sth, cth);
      const Dual Cph = chain(ph, cph, -sph), Sph = chain(ph, sph, cph);
      DE = (rp * DE) * power + T(1);
      rp = rp * r;
      zx = Cth * Cph * rp;
      zy = Cth * Sph * rp;
      zz = Sth * rp;
    } else {
      if (m_abs(zx.v) > limit) zx = dconst<TN>(m_copysign(value, zx.v)) - zx;
      if (m_abs(zy.v) > limit) zy = dconst<TN>(m_copysign(value, zy.v)) - zy;
      if (m_abs(zz.v) > limit) zz = dconst<TN>(m_copysign(value, zz.v)) - zz;
      const Dual r2 = zx * zx + zy * zy + zz * zz;
      const T offx = T(s.d[P_MB_OFF_X]), offy = T(s.d[P_MB_OFF_Y]), offz = T(s.d[P_MB_OFF_Z]);
      zx = zx + offx;
      zy = zy + offy;
      zz = zz + offz;
      if (r2.v < mR2.v) {
        zx = zx * factor1;
        zy = zy * factor1;
        zz = zz * factor1;
        DE = DE * factor1;
      } else if (r2.v < fR2.v) {
        const Dual t = fR2 / r2;
        zx = zx * t;
        zy = zy * t;
        zz = zz * t;
        DE = DE * t;
      }
      zx = zx - offx;
      zy = zy - offy;
      zz = zz - offz;
      zx = zx * scale;
      zy = zy * scale;
      zz = zz * scale;
      DE = DE * dabs(scale) + T(1);
    }
    if (s.add_c) {
      zx = zx + cx;
      zy = zy + cy;
      zz = zz + cz;
    }
    r = dlen3(zx, zy, zz);
    if (!(isfinite(r.v))) break;
    if (s.check_bailout && r.v > bailout) {
      escaped = true;
      break;
    }
  }
  Dual dist;
  if (DE.v > T(0)) {
    if (sc.de_analytic == 2) dist = (r.v > T(1)) ? (r * T(0.5)) * dlog(r) / DE : dconst<TN>(T(0));
    else if (sc.de_analytic == 3) dist = (r - T(2)) / DE;
    else dist = r / DE;
  } else {
    dist = r;
  }
  const int iters = i + 1;
  if (iters < sc.min_n && dist.v < detail) dist = dconst<TN>(detail);
  if (dist.v < T(0)) dist = dconst<TN>(T(0));
  if (dist.v > T(10)) dist = dconst<TN>(T(10));
  // a non-escaping orbit (a point inside the set): the estimate is ~0 and
  // constant to first order; its exact derivative is chaotic noise
  if (!escaped) dist = dconst<TN>(dist.v);
  return dist;
}

struct AdjointFrame {
  double dM[9];  // d(mRot)/d(yaw)
};

// One thread per pixel, with the formula's tangents only (with both formulas'
// six, at 255 registers, a 256x256 Mandelbox image took 302 us instead of 218).
template <class T, bool BULB>
__global__ void __launch_bounds__(128) adjoint_pixel_kernel(const __grid_constant__ DevScene sc,
                                                      const __grid_constant__ DevFrame fr,
                                                      const __grid_constant__ AdjointFrame af, const double *depth,
                                                      const uint8_t *hit, const float *dl_ddepth,
                                                      const float *dl_dshade, double *partials) {
  typedef Dn<T, Tangents<BULB>::n> Dual;
  const long long n = (long long)fr.width * fr.height;
  double acc[MBR_GRAD_COUNT];
#pragma unroll
  for (int k = 0; k < MBR_GRAD_COUNT; k++) acc[k] = 0.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    if (!hit[i]) continue;
    const double wt = dl_ddepth ? double(dl_ddepth[i]) : 0.0;
    const double ws = dl_dshade ? double(dl_dshade[i]) : 0.0;
    if (wt == 0.0 && ws == 0.0) continue;
    const int x = int(i % fr.width), y = int(i / fr.width);
    double ix, iy;
    image_point(fr, double(x), double(y), &ix, &iy);
    const D3 v0 = d3norm(D3{ix * fr.fov, 1.0, iy * fr.fov});
    const D3 w = rotate(fr, v0);
    const double wn = 1.0 / d3len(w);
    const D3 dir{w.x * wn, w.y * wn, w.z * wn};
    const double t = depth[i];
    const D3 cam = camera_of(fr);
    const D3 p = d3ray(cam, dir, t);
    const double thr = dist_thresh(sc, fr, p);
    const double c0 = fr.resolution * fr.fov / fr.detail_level * d3len(dir);
    // dist and its tangents at the hit point
    const Dual dh = de_dual<T, BULB>(sc, T(p.x), T(p.y), T(p.z), T(thr));
    // implicit differentiation needs F(t) = dist - thr = 0 at the stored
    // depth; a refinement that ended on a jump of the distance estimate (an
    // orbit's bailout iteration changing along the ray) has no derivative
    if (fabs(double(dh.v) - thr) > (sizeof(T) == 8 ? 1e-6 : 1e-4) * thr) continue;
    const D3 g{double(dh.d[TN_X]), double(dh.d[TN_Y]), double(dh.d[TN_Z])};
    // ∂p/∂θ at fixed t
    D3 dp[MBR_GRAD_COUNT];
#pragma unroll
    for (int k = 0; k < MBR_GRAD_COUNT; k++) dp[k] = D3{0.0, 0.0, 0.0};
    dp[MBR_GRAD_CAMERA_X] = D3{1.0, 0.0, 0.0};
    dp[MBR_GRAD_CAMERA_Y] = D3{0.0, 1.0, 0.0};
    dp[MBR_GRAD_CAMERA_Z] = D3{0.0, 0.0, 1.0};
    {
      const double *m = af.dM;
      const D3 dw{m[0] * v0.x + m[1] * v0.y + m[2] * v0.z, m[3] * v0.x + m[4] * v0.y + m[5] * v0.z,
                  m[6] * v0.x + m[7] * v0.y + m[8] * v0.z};
      dp[MBR_GRAD_YAW] = d3mul(dw, t * wn);
    }
    double dd[MBR_GRAD_COUNT];
#pragma unroll
    for (int k = 0; k < MBR_GRAD_COUNT; k++) dd[k] = 0.0;
    if (BULB) {
      dd[MBR_GRAD_BULB_POWER] = double(dh.d[TN_P0]);
    } else {
      dd[MBR_GRAD_MANDELBOX_SCALE] = double(dh.d[TN_P0]);
      dd[MBR_GRAD_MANDELBOX_MIN_R2] = double(dh.d[Tangents<BULB>::n - 1]);
    }
    const double denom = d3dot(g, dir) - c0;
    double dt[MBR_GRAD_COUNT];
#pragma unroll
    for (int k = 0; k < MBR_GRAD_COUNT; k++) dt[k] = -(dd[k] + d3dot(g, dp[k])) / denom;
    // the Lambert term through the six normal samples
    double ds[MBR_GRAD_COUNT];
#pragma unroll
    for (int k = 0; k < MBR_GRAD_COUNT; k++) ds[k] = 0.0;
    if (ws != 0.0) {
      const double delta = thr * fr.smoothness;
      double gv[3];
      double gd[3][MBR_GRAD_COUNT];
      for (int a = 0; a < 3; a++) {
        const D3 e{a == 0 ? 1.0 : 0.0, a == 1 ? 1.0 : 0.0, a == 2 ? 1.0 : 0.0};
        const D3 pp = d3add(p, d3mul(e, delta)), pm = d3sub(p, d3mul(e, delta));
        const Dual sp = de_dual<T, BULB>(sc, T(pp.x), T(pp.y), T(pp.z), T(thr));
        const Dual sm = de_dual<T, BULB>(sc, T(pm.x), T(pm.y), T(pm.z), T(thr));
        gv[a] = double(sp.v) - double(sm.v);
        const D3 gp{double(sp.d[TN_X]), double(sp.d[TN_Y]), double(sp.d[TN_Z])};
        const D3 gm{double(sm.d[TN_X]), double(sm.d[TN_Y]), double(sm.d[TN_Z])};
#pragma unroll
        for (int k = 0; k < MBR_GRAD_COUNT; k++) {
          const D3 dpt = d3add(dp[k], d3mul(dir, dt[k]));
          const double ddelta = c0 * fr.smoothness * dt[k];
          double dplus = d3dot(gp, d3add(dpt, d3mul(e, ddelta)));
          double dminus = d3dot(gm, d3sub(dpt, d3mul(e, ddelta)));
          if (k == (BULB ? MBR_GRAD_BULB_POWER : MBR_GRAD_MANDELBOX_SCALE)) {
            dplus += double(sp.d[TN_P0]);
            dminus += double(sm.d[TN_P0]);
          } else if (!BULB && k == MBR_GRAD_MANDELBOX_MIN_R2) {
            dplus += double(sp.d[Tangents<BULB>::n - 1]);
            dminus += double(sm.d[Tangents<BULB>::n - 1]);
          }
          gd[a][k] = dplus - dminus;
        }
      }
      const double gl = sqrt(gv[0] * gv[0] + gv[1] * gv[1] + gv[2] * gv[2]);
      const D3 N{gv[0] / gl, gv[1] / gl, gv[2] / gl};
      const D3 L{fr.light[0], fr.light[1], fr.light[2]};
      const double s = d3dot(N, L);
      if (s > 0.0) {
        const double scale = double(fr.material_shading) * double(fr.light_intensity);
#pragma unroll
        for (int k = 0; k < MBR_GRAD_COUNT; k++) {
          const D3 dg{gd[0][k], gd[1][k], gd[2][k]};
          const double ndg = d3dot(N, dg);
          const D3 dn = d3mul(d3sub(dg, d3mul(N, ndg)), 1.0 / gl);
          ds[k] = scale * d3dot(dn, L);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < MBR_GRAD_COUNT; k++) acc[k] += wt * dt[k] + ws * ds[k];
  }
  // warp reduction, then the block's warps in order: one partial sum per
  // block and parameter, summed by adjoint_sum_kernel in block order, so the
  // gradient does not depend on the order in which blocks ran
  __shared__ double warp_sum[4][MBR_GRAD_COUNT];
#pragma unroll
  for (int k = 0; k < MBR_GRAD_COUNT; k++) {
    double v = acc[k];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5][k] = v;
  }
  __syncthreads();
  if (threadIdx.x < MBR_GRAD_COUNT) {
    const int k = threadIdx.x;
    partials[(long long)blockIdx.x * MBR_GRAD_COUNT + k] =
        ((warp_sum[0][k] + warp_sum[1][k]) + warp_sum[2][k]) + warp_sum[3][k];
  }
}

// The value of lane `from` of this lane's group of eight.
__device__ __forceinline__ double of_lane(double v, int from) { return __shfl_sync(0xffffffffu, v, from, 8); }

// Eight lanes per hit pixel: lanes 2a and 2a + 1 take the normal samples on
// either side of axis a, lane 6 the hit point (lane 7 idles); then each lane
// takes one of the eight parameters.  The seven dual estimates of a hit lie
// within a threshold of each other, so their orbits run alike, and a hit takes
// one estimate's time instead of seven; each group looks for its next hit by
// itself, so misses cost no lane an estimate.  With
// one thread per pixel, seven estimates in turn and six tangents (255
// registers) the 256x256 Mandelbulb took 234 us, now 81 us.
template <class T, bool BULB>
__global__ void __launch_bounds__(128) adjoint_kernel(const __grid_constant__ DevScene sc,
                                                      const __grid_constant__ DevFrame fr,
                                                      const __grid_constant__ AdjointFrame af, const double *depth,
                                                      const uint8_t *hit, const float *dl_ddepth,
                                                      const float *dl_dshade, double *partials) {
  static_assert(MBR_GRAD_COUNT == 8, "a lane of a group of eight per parameter");
  const long long n = (long long)fr.width * fr.height;
  const int lane8 = threadIdx.x & 7;
  const long long groups = ((long long)gridDim.x * blockDim.x) >> 3;
  const D3 cam = camera_of(fr);
  double acc = 0.0;
  long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  for (;; i += groups) {
    double wt = 0.0, ws = 0.0;
    for (; i < n; i += groups) {  // the group's next hit with a weight
      if (!hit[i]) continue;
      wt = dl_ddepth ? double(dl_ddepth[i]) : 0.0;
      ws = dl_dshade ? double(dl_dshade[i]) : 0.0;
      if (wt != 0.0 || ws != 0.0) break;
    }
    const bool live = i < n;
    if (!__any_sync(0xffffffffu, live)) break;
    const long long pix = live ? i : 0;
    const int x = int(pix % fr.width), y = int(pix / fr.width);
    double ix, iy;
    image_point(fr, double(x), double(y), &ix, &iy);
    const D3 v0 = d3norm(D3{ix * fr.fov, 1.0, iy * fr.fov});
    const D3 w = rotate(fr, v0);
    const double wn = 1.0 / d3len(w);
    const D3 dir{w.x * wn, w.y * wn, w.z * wn};
    const double t = live ? depth[pix] : 0.0;
    const D3 p = d3ray(cam, dir, t);
    const double thr = dist_thresh(sc, fr, p);
    const double c0 = fr.resolution * fr.fov / fr.detail_level * d3len(dir);
    const double *m = af.dM;
    const D3 dw{m[0] * v0.x + m[1] * v0.y + m[2] * v0.z, m[3] * v0.x + m[4] * v0.y + m[5] * v0.z,
                m[6] * v0.x + m[7] * v0.y + m[8] * v0.z};
    const D3 dyaw = d3mul(dw, t * wn);  // d(hit point)/d(yaw) at fixed t
    const double delta = thr * fr.smoothness;
    // this lane's estimate and its tangents
    const int axis = lane8 >> 1;
    const D3 e{axis == 0 ? 1.0 : 0.0, axis == 1 ? 1.0 : 0.0, axis == 2 ? 1.0 : 0.0};
    const D3 off = d3mul(e, delta);
    const D3 q = lane8 >= 6 ? p : ((lane8 & 1) ? d3sub(p, off) : d3add(p, off));
    Dn<T, Tangents<BULB>::n> s = dconst<Tangents<BULB>::n>(T(0));
    if (live && lane8 < 7 && (lane8 == 6 || ws != 0.0)) s = de_dual<T, BULB>(sc, T(q.x), T(q.y), T(q.z), T(thr));
    __syncwarp();
    const D3 gs{double(s.d[TN_X]), double(s.d[TN_Y]), double(s.d[TN_Z])};
    const double tan0 = double(s.d[TN_P0]), tan1 = double(s.d[Tangents<BULB>::n - 1]);  // its parameter tangents
    // the hit point's, from lane 6.  Implicit differentiation needs
    // F(t) = dist - thr = 0 at the stored depth; a refinement that ended on a
    // jump of the distance estimate (an orbit's bailout iteration changing
    // along the ray) has no derivative
    const double dist = of_lane(double(s.v), 6);
    const bool root = live && !(fabs(dist - thr) > (sizeof(T) == 8 ? 1e-6 : 1e-4) * thr);
    const D3 g{of_lane(gs.x, 6), of_lane(gs.y, 6), of_lane(gs.z, 6)};
    const double denom = d3dot(g, dir) - c0;
    // this lane's parameter: the tangent of an estimate at a fixed point, and
    // dp/dtheta at fixed t
    const int k = lane8;
    const auto own = [&](int from) {
      const double a = of_lane(tan0, from), b = of_lane(tan1, from);
      if (BULB) return k == MBR_GRAD_BULB_POWER ? a : 0.0;
      return k == MBR_GRAD_MANDELBOX_SCALE ? a : (k == MBR_GRAD_MANDELBOX_MIN_R2 ? b : 0.0);
    };
    D3 dp{k == MBR_GRAD_CAMERA_X ? 1.0 : 0.0, k == MBR_GRAD_CAMERA_Y ? 1.0 : 0.0, k == MBR_GRAD_CAMERA_Z ? 1.0 : 0.0};
    if (k == MBR_GRAD_YAW) dp = dyaw;
    const double dt = -(own(6) + d3dot(g, dp)) / denom;
    // the Lambert term: the normal from the six samples and its tangent
    const D3 dpt = d3add(dp, d3mul(dir, dt));
    const double ddelta = c0 * fr.smoothness * dt;
    D3 gv, dg;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const D3 ea{a == 0 ? ddelta : 0.0, a == 1 ? ddelta : 0.0, a == 2 ? ddelta : 0.0};
      const D3 gp{of_lane(gs.x, 2 * a), of_lane(gs.y, 2 * a), of_lane(gs.z, 2 * a)};
      const D3 gm{of_lane(gs.x, 2 * a + 1), of_lane(gs.y, 2 * a + 1), of_lane(gs.z, 2 * a + 1)};
      const double dplus = d3dot(gp, d3add(dpt, ea)) + own(2 * a);
      const double dminus = d3dot(gm, d3sub(dpt, ea)) + own(2 * a + 1);
      const double v = of_lane(double(s.v), 2 * a) - of_lane(double(s.v), 2 * a + 1);
      if (a == 0) gv.x = v, dg.x = dplus - dminus;
      else if (a == 1) gv.y = v, dg.y = dplus - dminus;
      else gv.z = v, dg.z = dplus - dminus;
    }
    if (root) {
      double ds = 0.0;
      if (ws != 0.0) {
        const double gl = sqrt(gv.x * gv.x + gv.y * gv.y + gv.z * gv.z);
        const D3 N{gv.x / gl, gv.y / gl, gv.z / gl};
        const D3 Lt{fr.light[0], fr.light[1], fr.light[2]};
        if (d3dot(N, Lt) > 0.0) {
          const D3 dn = d3mul(d3sub(dg, d3mul(N, d3dot(N, dg))), 1.0 / gl);
          ds = double(fr.material_shading) * double(fr.light_intensity) * d3dot(dn, Lt);
        }
      }
      acc += wt * dt + ws * ds;
    }
    __syncwarp();
  }
  // warp reduction, then the block's warps in order: one partial sum per
  // block and parameter, summed by adjoint_sum_kernel in a fixed order, so the
  // gradient does not depend on the order in which blocks ran
  __shared__ double warp_sum[4][MBR_GRAD_COUNT];
  acc += __shfl_down_sync(0xffffffffu, acc, 16);
  acc += __shfl_down_sync(0xffffffffu, acc, 8);
  if ((threadIdx.x & 31) < MBR_GRAD_COUNT) warp_sum[threadIdx.x >> 5][threadIdx.x & 31] = acc;
  __syncthreads();
  if (threadIdx.x < MBR_GRAD_COUNT) {
    const int k = threadIdx.x;
    partials[(long long)blockIdx.x * MBR_GRAD_COUNT + k] =
        ((warp_sum[0][k] + warp_sum[1][k]) + warp_sum[2][k]) + warp_sum[3][k];
  }
}

// grad[k] += the blocks' partial sums of parameter k: a warp per parameter,
// each lane every 32nd block, then the lanes (one thread per parameter read
// 512 blocks in turn in 17 us).
__global__ void __launch_bounds__(32 * MBR_GRAD_COUNT) adjoint_sum_kernel(const double *partials, int blocks, double *grad) {
  const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double v = 0.0;
  for (int b = lane; b < blocks; b += 32) v += partials[(long long)b * MBR_GRAD_COUNT + k];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (lane == 0) grad[k] += v;
}

}  // namespace mbr

using namespace mbr;

extern "C" mbr_status mbr_adjoint(mbr_ctx *ctx, const mbr_camera *camera, const mbr_render_params *params,
                                  const double *depth, const uint8_t *hit, const float *dl_ddepth,
                                  const float *dl_dshade, double *grad, int engine, void *stream) {
  if (!ctx || !camera || !params || !depth || !hit || !grad) return set_err(ctx, MBR_EINVAL, "null argument");
  const DevScene *sc = ctx_scene(ctx);
  if (!sc) return set_err(ctx, MBR_EINVAL, "no scene set");
  if (!camera->use_angles)
    return set_err(ctx, MBR_EINVAL, "the adjoint differentiates a camera given by position and angles (use_angles = 1)");
  if (camera->perspective_type != MBR_PROJECTION_THREE_POINT)
    return set_err(ctx, MBR_EUNSUPPORTED, "the adjoint covers the three-point projection");
  if (params->slow_shading)
    return set_err(ctx, MBR_EUNSUPPORTED, "the adjoint differentiates the six-sample normals (no slow shading)");
  if (params->advanced_quality || params->constant_de_threshold)
    return set_err(ctx, MBR_EUNSUPPORTED, "the adjoint covers thresholds proportional to the distance (no advanced "
                                          "quality clamps, no constant threshold)");
  if (sc->mbrot.folds || sc->mbrot.main)
    return set_err(ctx, MBR_EUNSUPPORTED, "the adjoint covers the Mandelbox without rotations");
  if (sc->n_prims > 0 || sc->n_nodes > 0 || sc->limits || sc->gbox || sc->gsph)
    return set_err(ctx, MBR_EUNSUPPORTED,
                   "the adjoint covers scenes without primitives, objects tree, limit box or global folds");
  if (sc->delta_de || sc->de_final > DEF_IFS)
    return set_err(ctx, MBR_EUNSUPPORTED, "the adjoint covers the analytic linear and logarithmic DE functions");
  if (sc->is_hybrid || sc->has_w || sc->iter_thresh || sc->interior ||
      (sc->slot[0].formula != MBR_FORMULA_MANDELBULB && sc->slot[0].formula != MBR_FORMULA_MANDELBOX))
    return set_err(ctx, MBR_EUNSUPPORTED,
                   "the adjoint covers non-hybrid Mandelbulb and Mandelbox scenes without interior, iteration "
                   "threshold or 4-D modes");
  if (engine != MBR_ENGINE_PLAIN_FP64 && engine != MBR_ENGINE_PLAIN_MIXED)
    return set_err(ctx, MBR_EINVAL, "adjoint engine must be MBR_ENGINE_PLAIN_FP64 or MBR_ENGINE_PLAIN_MIXED");
  DevFrame fr;
  mbr_status st = build_frame(ctx, *camera, *params, &fr, stream);
  if (st != MBR_OK) return st;
  // d(mRot)/d(yaw) with mRot = Rz(yaw) Rx(pitch) Ry(roll) (PrepareMainVectors)
  AdjointFrame af;
  {
    const double yaw = camera->angles[0], pitch = camera->angles[1], roll = camera->angles[2];
    const double dz[9] = {-std::sin(yaw), -std::cos(yaw), 0, std::cos(yaw), -std::sin(yaw), 0, 0, 0, 0};
    const double cx = std::cos(pitch), sx = std::sin(pitch), cy = std::cos(roll), sy = std::sin(roll);
    const double rx[9] = {1, 0, 0, 0, cx, -sx, 0, sx, cx};
    const double ry[9] = {cy, 0, sy, 0, 1, 0, -sy, 0, cy};
    double t[9];
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++) t[i * 3 + j] = dz[i * 3] * rx[j] + dz[i * 3 + 1] * rx[3 + j] + dz[i * 3 + 2] * rx[6 + j];
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++)
        af.dM[i * 3 + j] = t[i * 3] * ry[j] + t[i * 3 + 1] * ry[3 + j] + t[i * 3 + 2] * ry[6 + j];
  }
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const long long n = (long long)fr.width * fr.height;
  // Eight lanes per hit, or one thread per pixel: for a Mandelbox image of 128^2
  // pixels and more, whose estimate, 12 passes without library functions, is
  // short enough that many pixels in flight hide it, and the groups' exchange
  // costs more than their parallel samples save (per pixel / eight lanes: 100x95
  // 85 / 61 us, 160x160 108 / 139 us, 256x256 218 / 319 us, 512x505 765 / 1202
  // us; the Mandelbulb 64x60 60 / 14 us, 256x256 182 / 81 us, 512x505 1664 / 802
  // us); and without a shade gradient, where a hit has one estimate and seven
  // lanes of the group would idle (the whole call, per pixel / eight lanes:
  // Mandelbulb 64x64 51 / 53 us, 160x160 53 / 75 us, 256x256 65 / 109 us, 400x400
  // 89 / 202 us; Mandelbox 100x100 53 / 67 us).
  const bool bulb = sc->slot[0].formula == MBR_FORMULA_MANDELBULB;
  const bool per_pixel = !dl_dshade || (!bulb && n >= 16384);
  const long long blocks = per_pixel ? (n + 127) / 128 : (n + 15) / 16;
  const int grid = int(std::max<long long>(1, std::min<long long>(blocks, (long long)sms * 16)));
  double *partials = nullptr;
  st = ctx_adjoint_partials(ctx, size_t(grid) * MBR_GRAD_COUNT * sizeof(double), &partials);
  if (st != MBR_OK) return st;
#define ADJOINT(KERNEL) KERNEL<<<grid, 128, 0, s>>>(*sc, fr, af, depth, hit, dl_ddepth, dl_dshade, partials)
  if (engine == MBR_ENGINE_PLAIN_FP64) {
    if (bulb && per_pixel) ADJOINT((adjoint_pixel_kernel<double, true>));
    else if (bulb) ADJOINT((adjoint_kernel<double, true>));
    else if (per_pixel) ADJOINT((adjoint_pixel_kernel<double, false>));
    else ADJOINT((adjoint_kernel<double, false>));
  } else {
    if (bulb && per_pixel) ADJOINT((adjoint_pixel_kernel<float, true>));
    else if (bulb) ADJOINT((adjoint_kernel<float, true>));
    else if (per_pixel) ADJOINT((adjoint_pixel_kernel<float, false>));
    else ADJOINT((adjoint_kernel<float, false>));
  }
#undef ADJOINT
  adjoint_sum_kernel<<<1, 32 * MBR_GRAD_COUNT, 0, s>>>(partials, grid, grad);
  count_launches(2);
  return cuda_err(ctx, int(cudaGetLastError()), "adjoint kernel launch");
}
