// staged_plain.cuh - the plain FP64 engines' frames as a pipeline of stages.
//
// The same per-pixel work as plain_kernel (plain_kernel.cuh), operation for
// operation, split so that no lane waits for another kind of work.  One thread
// per pixel left 13 to 18 of 32 lanes active (a warp ran its longest orbit in
// every estimate, its longest march in every ray, and its AO rays one after
// the other), and the slowest warp's chain of march, normals, shadow and AO
// rays set the frame's time.  What bounds the stages now is FP64 latency and
// issue, and in stages P and S the longest single ray.  One thread per pixel
// -> stages: Mandelbox 801x451, 4 AO rays, 2.33 -> 1.56 ms of kernels; a
// pseudo-Kleinian view 320x240, 4 AO rays, 33.7 -> 6.8 ms.
//   stage P  per pixel: camera ray, march, binary search; hits are appended
//   stage N  per hit: the six normal samples and the Lambert term
//   stage S  per hit: the shadow march and each AO march as a task of its own
//   stage F  per hit: the AO results summed in ray order, colour, outputs
// The stages run on the wavefront's persistent skeleton (run_stage).
#pragma once
#include "wavefront.cuh"

namespace mbr {

struct RefHit {
  double px, py, pz, depth, thr;
  double nx, ny, nz;
  long long ray;  // pixel of the frame
  int iters;
  float lambert;  // before the shadow
};

struct RefLaunch {
  Counters4 *ctr;
  RefHit *hits;
  double *ao;     // per hit and AO task: the march's result (fast AO: the AO factor)
  float *shadow;  // per hit: AuxShadow's result
  long long pixels;
  FastDiv div_tx, div_per;
  int tiles_x, per, shadow_tasks, ao_tasks, refill_k, need_normal;
};

struct RefParams {
  const DevScene &sc;
};

// One distance estimate of a scene without the extended features, a pass at a time.
template <class T, int F, bool NORMAL>
struct RefPass {
  typedef double D;
  typedef RefParams Params;
  enum { kWide = 1, kHyb = 1, kTotal = 0 };
  typedef OrbitLane<T> State;
  template <int FK>
  __device__ static void start(State &e, const Params &fp, double qx, double qy, double qz) {
    orbit_begin<T>(e, T(qx), T(qy), T(qz), fp.sc.formula_maxiter * ((NORMAL && fp.sc.iter_thresh) ? 5 : 1));
  }
  template <int FK>
  __device__ static bool step(int, State &e, const Params &fp) {
    orbit_pass<T, F>(fp.sc, e, fp.sc.formula_maxiter * ((NORMAL && fp.sc.iter_thresh) ? 5 : 1));
    return e.end == ORBIT_RUNS;
  }
  template <int FK>
  __device__ static double distance(State &e, const Params &fp, double detail, int &iters) {
    const V4<T> z{e.zx, e.zy, e.zz, T(0.0)};
    iters = e.end == ORBIT_MAXITER ? e.it + 1 : e.it;
    const T d = final_distance<T, F, false>(fp.sc, z, len4<T, false>(z), e.de);
    return double(distance_tail<T>(fp.sc, d, iters, e.end != ORBIT_BAILOUT, T(detail), NORMAL));
  }
};

// The whole estimate in one step: extended scenes (every formula, objects
// trees, delta DE) and blended sequences.
template <class T, int F, bool NORMAL>
struct RefWhole {
  typedef double D;
  typedef RefParams Params;
  enum { kWide = 1, kHyb = 1, kTotal = 1 };
  struct State {
    double x, y, z;
    int total;
  };
  template <int FK>
  __device__ static void start(State &e, const Params &, double qx, double qy, double qz) {
    e.x = qx;
    e.y = qy;
    e.z = qz;
  }
  template <int FK>
  __device__ static bool step(int, State &, const Params &) {
    return false;
  }
  template <int FK>
  __device__ static double distance(State &e, const Params &fp, double detail, int &iters) {
    return double(calc_distance<T, F, false>(fp.sc, T(e.x), T(e.y), T(e.z), T(detail), NORMAL, &iters, &e.total));
  }
};

struct RefPrimaryStage {
  typedef double Real;
  typedef double D;
  static constexpr bool kMulti = false;
  const RefParams &prm;
  const DevScene &sc;
  const DevFrame &fr;
  const RefLaunch &L;
  const DevOutputs &out;
  D3 dir, last;
  double scan, stp, dir_len, thr, dist;
  int phase, count, last_iters;  // phase 0 march, > 0 binary search round, < 0 step back
  ParkMiller pm;
  long long ray;
  unsigned int n_binary;

  __device__ const RefParams &params() const { return prm; }
  __device__ int kind() const { return 0; }
  __device__ double detail() const { return thr; }
  __device__ D3 at() const { return d3ray(camera_of(fr), dir, scan); }

  __device__ bool start(long long idx, double &qx, double &qy, double &qz) {
    const unsigned long long tile = (unsigned long long)idx >> 5;
    const int w = int(idx & 31);
    const unsigned long long ty = fdiv(tile, L.div_tx);
    const int x = int(tile - ty * (unsigned long long)L.tiles_x) * 8 + (w & 7);
    const int y = fr.row0 + int(ty) * 4 + (w >> 3);
    if (x >= fr.width || y >= fr.row1) return false;
    ray = (long long)y * fr.width + x;
    last_iters = 0;
    double ix, iy;
    image_point(fr, double(x), double(y), &ix, &iy);
    if (hemisphere_cut(fr.persp, fr.fov, ix, iy)) return miss(true);
    dir = d3norm(view_vector(fr, ix, iy));
    pm = pm_for_ray((unsigned long long)ray, fr.seed);
    dir_len = d3len(dir);
    scan = stp = thr = dist = 0.0;
    phase = count = 0;
    last = D3{1e30, 1e30, 1e30};
    return advance(qx, qy, qz);
  }

  // the next march point; a point that did not move or is not finite is a hit where it stands
  __device__ bool advance(double &qx, double &qy, double &qz) {
    const D3 p = at();
    if ((p.x == last.x && p.y == last.y && p.z == last.z) || !(isfinite(p.x) && isfinite(p.y) && isfinite(p.z)))
      return sc.iter_thresh ? step_back(qx, qy, qz) : hit();
    last = p;
    thr = dist_thresh(sc, fr, p);
    qx = p.x;
    qy = p.y;
    qz = p.z;
    return true;
  }

  __device__ bool miss(bool cut) {
    float rgb[3] = {fr.background[0], fr.background[1], fr.background[2]};
    if (cut) rgb[0] = rgb[1] = rgb[2] = 0.0f;
    const long long o = out.pixel_offset + ray;
    if (out.depth) out.depth[o] = 1e20;
    if (out.iters) out.iters[o] = last_iters;
    if (out.hit) out.hit[o] = 0;
    if (out.normal) out.normal[3 * o] = out.normal[3 * o + 1] = out.normal[3 * o + 2] = 0.0f;
    if (out.shade) out.shade[o] = 0.0f;
    if (out.ao) out.ao[o] = 1.0f;
    if (out.rgb) {
      out.rgb[3 * o + 0] = rgb[0];
      out.rgb[3 * o + 1] = rgb[1];
      out.rgb[3 * o + 2] = rgb[2];
    }
    if (out.rgb8) to_rgb8(fr, rgb, &out.rgb8[3 * o]);
    return false;
  }

  __device__ bool hit() {
    RefHit &r = L.hits[atomicAdd(&L.ctr->hits, 1ull)];
    const D3 p = at();
    r.px = p.x;
    r.py = p.y;
    r.pz = p.z;
    r.depth = scan;
    r.thr = thr;
    r.ray = ray;
    r.iters = last_iters;
    return false;
  }

  // iteration_threshold_mode: every hit ends with an estimate one threshold back
  __device__ bool step_back(double &qx, double &qy, double &qz) {
    scan -= thr;
    phase = -1;
    const D3 p = at();
    qx = p.x;
    qy = p.y;
    qz = p.z;
    return true;
  }

  // one round of the binary search (ray_marching, pixel_ops.cuh)
  __device__ bool refine(double &qx, double &qy, double &qz) {
    const double search_limit = 1.0 - 0.001 * fr.detail_level;
    if (phase <= fr.binary_steps && !(dist < thr && dist > thr * search_limit)) {
      if (dist > thr) scan += stp;
      else if (dist < thr * search_limit) scan -= stp;
    } else {
      return sc.iter_thresh ? step_back(qx, qy, qz) : hit();
    }
    const D3 p = at();
    thr = dist_thresh(sc, fr, p);
    qx = p.x;
    qy = p.y;
    qz = p.z;
    return true;
  }

  __device__ bool step(double d, int iters, double &qx, double &qy, double &qz) {
    last_iters = iters;
    dist = d;
    if (phase != 0) {
      n_binary++;
      if (phase < 0) return hit();
      phase++;
      stp *= 0.5;
      return refine(qx, qy, qz);
    }
    count++;
    if (dist < thr) {
      phase = 1;
      stp *= 0.5;
      return refine(qx, qy, qz);
    }
    const double jit = fr.jitter ? (1.0 - tenthousandths(pm.random(1000))) : 1.0;
    if (sc.interior)
      stp = (dist - 0.8 * thr) * fr.de_factor * jit;
    else
      stp = (dist - 0.5 * thr) * fr.de_factor * jit;
    stp = step_limit(fr, stp, thr);
    scan += stp / dir_len;
    if (scan > fr.view_distance_max || count >= fr.max_steps) return miss(false);
    return advance(qx, qy, qz);
  }
};

struct RefNormalStage {
  typedef double Real;
  typedef double D;
  static constexpr bool kMulti = false;
  const RefParams &prm;
  const DevScene &sc;
  const DevFrame &fr;
  const RefLaunch &L;
  RefHit *r;
  D3 q, n;
  double thr, delta, first;
  int sub;

  __device__ const RefParams &params() const { return prm; }
  __device__ int kind() const { return 0; }
  __device__ double detail() const { return thr; }
  __device__ void point(double &qx, double &qy, double &qz) const {
    const int axis = sub >> 1;
    const D3 e{axis == 0 ? delta : 0.0, axis == 1 ? delta : 0.0, axis == 2 ? delta : 0.0};
    const D3 p = (sub & 1) ? d3sub(q, e) : d3add(q, e);
    qx = p.x;
    qy = p.y;
    qz = p.z;
  }
  __device__ bool start(long long idx, double &qx, double &qy, double &qz) {
    r = &L.hits[idx];
    q = D3{r->px, r->py, r->pz};
    thr = r->thr;
    delta = thr * fr.smoothness;
    if (sc.interior) delta = thr * 0.2 * fr.smoothness;
    sub = 0;
    point(qx, qy, qz);
    return true;
  }
  __device__ bool step(double d, int, double &qx, double &qy, double &qz) {
    if (!(sub & 1)) {
      first = d;
    } else {
      const double g = first - d;
      if (sub == 1) n.x = g;
      else if (sub == 3) n.y = g;
      else n.z = g;
    }
    if (++sub < 6) {
      point(qx, qy, qz);
      return true;
    }
    if (fabs(n.x) < 1e-50 && fabs(n.y) < 1e-50 && fabs(n.z) < 1e-50)
      n = D3{1.0, 0.0, 0.0};
    else
      n = d3norm(n);
    if (!(isfinite(n.x) && isfinite(n.y) && isfinite(n.z))) n = D3{1.0, 0.0, 0.0};
    r->nx = n.x;
    r->ny = n.y;
    r->nz = n.z;
    float s = 0.0f;
    if (fr.shading_enable) {
      s = float(d3dot(n, D3{fr.light[0], fr.light[1], fr.light[2]}));
      if (s < 0) s = 0;
      s = 1.0f - fr.material_shading + s * fr.material_shading;
      s = s * fr.light_intensity;
      if (s > 500.0f) s = 500.0f;
    }
    r->lambert = s;
    return false;
  }
};

// Task k of a hit: 0 the shadow march (when shadows are on), then the AO
// marches along the ray's own draws of the hit's stream, or the one fast AO.
// EXT: the limit box, which a soft shadow's samples may lie outside of.
template <bool EXT>
struct RefShadeStage {
  typedef double Real;
  typedef double D;
  static constexpr bool kMulti = false;
  const RefParams &prm;
  const DevScene &sc;
  const DevFrame &fr;
  const RefLaunch &L;
  D3 q, v;
  double t, end, thr, keep, sum;  // keep: soft shadow's largest term; fast AO's previous sample
  float thr_f;
  long long slot;   // where the result goes
  int mode, count;  // mode 0 shadow, 1 AO march, 2 fast AO
  unsigned int n_shadow, trips;

  __device__ const RefParams &params() const { return prm; }
  __device__ int kind() const { return 0; }
  __device__ double detail() const { return thr; }
  __device__ bool request(double &qx, double &qy, double &qz) const {
    const D3 p = d3ray(q, v, t);
    qx = p.x;
    qy = p.y;
    qz = p.z;
    return true;
  }
  __device__ bool shadow(double s) {
    L.shadow[slot] = float(s);
    return false;
  }
  __device__ bool ao(double s) {
    L.ao[slot] = s;
    return false;
  }
  __device__ bool soft() const { return fr.soft_range > 0.0 && !sc.interior && !sc.iter_thresh; }

  __device__ bool start(long long idx, double &qx, double &qy, double &qz) {
    const long long h = (long long)fdiv((unsigned long long)idx, L.div_per);
    const int k = int(idx - h * L.per);
    const RefHit &r = L.hits[h];
    q = D3{r.px, r.py, r.pz};
    thr = r.thr;
    thr_f = float(thr);
    t = thr;
    count = 0;
    if (k < L.shadow_tasks) {
      mode = 0;
      slot = h;
      if (!(r.lambert > 0.001f)) return shadow(0.0);
      v = D3{fr.light[0], fr.light[1], fr.light[2]};
      end = fr.penetrating ? calc_delta(fr, q) / fr.resolution : fr.view_distance_max;
      if (sc.interior) t = thr * fr.de_factor;
      keep = 0.0;
      if (!(t < end)) return shadow(1.0);
      return request(qx, qy, qz);
    }
    const int a = k - L.shadow_tasks;
    slot = h * L.ao_tasks + a;
    const D3 n{r.nx, r.ny, r.nz};
    if (fr.ao_fast) {
      mode = 2;
      v = n;
      keep = 1e20;
      sum = 0.0;
      if (!(1 < fr.ao_quality * fr.ao_quality)) return ao(fast_factor());
      return request(qx, qy, qz);
    }
    mode = 1;
    end = calc_delta(fr, q) / fr.resolution;
    if (!(t < end)) return ao(1.0);
    Pcg32 rng = pcg_init(fr.ao_seed, (unsigned long long)r.ray);
    rng.state = pcg_advance(rng.state, rng.inc, 2ull * (unsigned long long)a);
    const double u1 = rng.uniform(), u2 = rng.uniform();
    v = cosine_dir(n, u1, u2);
    return request(qx, qy, qz);
  }
  __device__ double fast_factor() const {
    float f = 1.0f - 0.2f * float(sum);
    if (f < 0) f = 0;
    return f;
  }

  __device__ bool step(double dist, int, double &qx, double &qy, double &qz) {
    count++;
    if (mode == 0) {
      n_shadow++;
      if (soft()) {
        bool outside = false;
        if (EXT && sc.limits) {
          const D3 p = d3ray(q, v, t);
          outside = p.x < sc.lim_min[0] || p.x > sc.lim_max[0] || p.y < sc.lim_min[1] || p.y > sc.lim_max[1] ||
                    p.z < sc.lim_min[2] || p.z > sc.lim_max[2];
        }
        if (!outside) {
          double angle = (dist - double(thr_f)) / t;
          if (angle < 0) angle = 0;
          if (dist < double(thr_f)) angle = 0;
          double s = 1.0 - angle / fr.soft_range;
          if (fr.penetrating) s *= (end - t) / end;
          if (s < 0) s = 0;
          if (s > keep) keep = s;
        }
      }
      if (dist < double(thr_f)) {
        double s = 0.0;
        if (fr.penetrating) {
          s = 1.0 - (end - t) / end;
          if (s < 0.0) s = 0.0;
        }
        return shadow(soft() ? 1.0 - keep : s);
      }
      double stp = fmin(dist, 1000000.0) * fr.de_factor;
      stp = fmax(stp, 1e-15);
      if (count > fr.max_steps) return shadow(soft() ? 1.0 - keep : 1.0);
      t += stp;
      if (!(t < end)) return shadow(soft() ? 1.0 - keep : 1.0);
      return request(qx, qy, qz);
    }
    if (mode == 2) {
      if (dist > keep * 2) dist = keep * 2.0;
      keep = dist;
      sum = double(float(sum + ldexp(1.0, -count) * (t - fr.ao_fast_tune * dist) / thr));
      t = double((count + 1) * (count + 1)) * thr;
      if (!(count + 1 < fr.ao_quality * fr.ao_quality)) return ao(fast_factor());
      return request(qx, qy, qz);
    }
    if (dist < double(thr_f)) {
      double s = 1.0 - (end - t) / end;
      if (s < 0.0) s = 0.0;
      return ao(s);
    }
    t += dist * 2.0;
    if (!(t < end)) return ao(1.0);
    if (count >= fr.max_steps) {  // the cap ended it: a watchdog trip
      trips++;
      return ao(1.0);
    }
    return request(qx, qy, qz);
  }
};

// Blocks of 128 per SM that the registers leave room for: a pass-by-pass
// Mandelbox frame (801x451, 4 AO rays) takes 1.76 ms unbounded, 1.60 at 5/6/6
// (stages P/S/N), 1.56 at 6/7/8 and 1.58 at 8/8/10; a whole extended estimate
// is faster with all its registers (14.6 ms against 15.0, 15.9 and 16.2).
enum RefBlocks { REF_P = 6, REF_S = 7, REF_N = 8 };

template <class P, int FK, int V>
__global__ void __launch_bounds__(128, P::kTotal ? 0 : REF_P) ref_primary_kernel(const __grid_constant__ DevScene sc,
                                                                                 const __grid_constant__ DevFrame fr,
                                                                                 const __grid_constant__ RefLaunch L,
                                                                                 DevOutputs out) {
  const RefParams fp{sc};
  RefPrimaryStage S{fp, sc, fr, L, out};
  S.n_binary = 0;
  unsigned int my_de = 0;
  unsigned long long my_iters = 0;
  const long long total = (long long)L.tiles_x * ((fr.row1 - fr.row0 + 3) / 4) * 32;
  run_stage<FK, P>(S, fp, &L.ctr->pixels_next, total, L.refill_k, &my_de, &my_iters);
  flush_counts(out, my_de, my_iters, K_MARCH, my_de - S.n_binary, K_BINARY, S.n_binary);
}

template <class P, int FK, int V>
__global__ void __launch_bounds__(128, P::kTotal ? 0 : REF_N) ref_normal_kernel(const __grid_constant__ DevScene sc,
                                                                                const __grid_constant__ DevFrame fr,
                                                                                const __grid_constant__ RefLaunch L,
                                                                                DevOutputs out) {
  const RefParams fp{sc};
  RefNormalStage S{fp, sc, fr, L};
  unsigned int my_de = 0;
  unsigned long long my_iters = 0;
  run_stage<FK, P>(S, fp, &L.ctr->normals_next, (long long)L.ctr->hits, L.refill_k, &my_de, &my_iters);
  flush_counts(out, my_de, my_iters, K_NORMAL, my_de, K_NORMAL, 0);
}

template <class P, int FK, bool EXT, int V>
__global__ void __launch_bounds__(128, P::kTotal ? 0 : REF_S) ref_shade_kernel(const __grid_constant__ DevScene sc,
                                                                               const __grid_constant__ DevFrame fr,
                                                                               const __grid_constant__ RefLaunch L,
                                                                               DevOutputs out) {
  const RefParams fp{sc};
  RefShadeStage<EXT> S{fp, sc, fr, L};
  S.n_shadow = S.trips = 0;
  unsigned int my_de = 0;
  unsigned long long my_iters = 0;
  run_stage<FK, P>(S, fp, &L.ctr->shade_next, (long long)L.ctr->hits * L.per, L.refill_k, &my_de, &my_iters);
  flush_counts(out, my_de, my_iters, K_AO, my_de - S.n_shadow, K_SHADOW, S.n_shadow);
  const unsigned int trips = __reduce_add_sync(0xffffffffu, S.trips);
  if ((threadIdx.x & 31) == 0 && trips) {
    if (out.stats) atomicAdd(reinterpret_cast<unsigned long long *>(out.stats) + K_WATCHDOG, (unsigned long long)trips);
    if (out.status) atomicOr(out.status, int(STATUS_AO_MARCH_CAP));
  }
}

template <int V>
__global__ void __launch_bounds__(256) ref_finish_kernel(const __grid_constant__ DevFrame fr,
                                                         const __grid_constant__ RefLaunch L, DevOutputs out) {
  const long long nh = (long long)L.ctr->hits;
  const long long first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (first == 0 && out.stats)
    atomicAdd(reinterpret_cast<unsigned long long *>(out.stats) + K_PIXELS, (unsigned long long)L.pixels);
  for (long long h = first; h < nh; h += (long long)gridDim.x * blockDim.x) {
    const RefHit &r = L.hits[h];
    const long long o = out.pixel_offset + r.ray;
    float shade = 0.0f, ao = 1.0f;
    if (fr.shading_enable) shade = r.lambert * (fr.shadow_enable ? L.shadow[h] : 1.0f);
    if (L.ao_tasks > 0) {
      double sum = 0.0;
      for (int k = 0; k < L.ao_tasks; k++) sum += L.ao[h * L.ao_tasks + k];
      ao = fr.ao_fast ? float(L.ao[h]) : float(sum / fr.ao_rays);
    }
    const float col = fr.albedo * (shade + fr.ambient * ao);
    float rgb[3] = {col, col, col};
    if (out.depth) out.depth[o] = r.depth;
    if (out.iters) out.iters[o] = r.iters;
    if (out.hit) out.hit[o] = 1;
    if (out.normal) {
      out.normal[3 * o + 0] = L.need_normal ? float(r.nx) : 0.0f;
      out.normal[3 * o + 1] = L.need_normal ? float(r.ny) : 0.0f;
      out.normal[3 * o + 2] = L.need_normal ? float(r.nz) : 0.0f;
    }
    if (out.shade) out.shade[o] = shade;
    if (out.ao) out.ao[o] = ao;
    if (out.rgb) {
      out.rgb[3 * o + 0] = col;
      out.rgb[3 * o + 1] = col;
      out.rgb[3 * o + 2] = col;
    }
    if (out.rgb8) to_rgb8(fr, rgb, &out.rgb8[3 * o]);
  }
}

// Frames the stages take: a 3-D state, the reference's refinement, no GI and
// no iteration-count normals.  Of these plain_kernel keeps what it renders
// faster (per-pixel / stages, us):
//  - The delta DE, four orbits an estimate that run alike in neighbouring pixels
//    (strict engine: Mandelbox 160x120 7660 / 8811, 320x240 with 4 AO rays 19202 /
//    22364; box fold bulb pow 2 320x240 6453 / 8718, with 4 rays 12628 / 10970).
//    With contraction it would magnify the difference between the two forms'
//    rounding (depths within 1e-15) 1e7-fold.
//  - Explicit objects trees with fewer than 4 AO rays: a tree's walk branches by
//    where a point lies, and neighbouring pixels, which a warp of plain_kernel
//    marches together, branch alike.  Six trees, 64x48 to 1024x768: without AO
//    1029 / 1188 to 12132 / 16940 (0.68 to 1.04 of its speed), 2 rays 0.83 to
//    1.27, 4 rays 0.96 to 1.64, 8 rays 1.07 to 2.74.
//  - Of the other extended scenes (primitives, limits, folds, rotations, other
//    formulas and nine by settings key, 16x12 to 640x480, 0 and 4 rays: 1.04 to
//    6.3), frames below 160x120 with fewer than 4 AO rays where the estimates are
//    short: the Menger sponge (with a sphere 16x12 194 / 208, 128x96 519 / 548,
//    160x120 636 / 593), the Mandelbulb (with folds 16x12 254 / 269, 64x48 649 /
//    664, 160x120 1205 / 1077) and sequences (in a limit box 16x12 157 / 165,
//    64x48 208 / 252, 160x120 917 / 816; with a sphere 16x12 268 / 278).
//  - The Menger sponge without extensions (64x48 to 1024x768 frames run at 0.70 to
//    0.95 of its speed by stages).
//  - Small frames without many marches, where the stages' separate tails cost
//    more than they even out: Mandelbulb without AO 256x192 694 / 752, 400x300
//    1274 / 1513, 640x480 3077 / 2671, 1024x768 7490 / 5316; with 4 AO rays 64x48
//    322 / 296, 400x300 2041 / 1871, 1024x768 14449 / 7001; Mandelbox without AO
//    256x192 233 / 257, 640x480 1076 / 776.
// The gain depends on the view.  Two Mandelboxes, the Mandelbulb and two
// sequences from four sides, 4 rays: 128x96 0.81 to 1.75 (mean 1.28), 320x240 0.83
// to 1.97 (1.29), 640x480 0.91 to 2.82 (1.76), 800x600 1.13 to 2.99; 8 rays 0.89 at
// the least, 16 rays 1.04.  It is below 1 where one ray's chain of estimates sets
// the time, which takes longer in stages than in a warp of its own: the Mandelbox
// seen from above an edge up to 640x480, the Mandelbulb's limb at 128x96.
// The size is the frame's, whatever rows of it are asked for: a band of a frame
// has to equal the frame's rows bit for bit, so it takes the frame's kernels.
inline bool staged_plain_takes(const DevScene &sc, const DevFrame &fr) {
  bool delta = sc.delta_de != 0;
  for (int k = 0; k < sc.n_nodes; k++) delta = delta || sc.node[k].delta_de != 0;
  if (sc.has_w || fr.gi_samples > 0 || fr.refine != MBR_REFINE_REFERENCE || fr.slow_shading || delta) return false;
  if (fr.ao_rays >= 4) return scene_extended(sc) || sc.is_hybrid || sc.uniform_formula != MBR_FORMULA_MENGER_SPONGE;
  const long long pixels = (long long)fr.width * fr.height;
  if (sc.n_nodes > 0) return false;
  if (scene_extended(sc))
    return pixels >= 19200 || !(sc.is_hybrid || sc.uniform_formula == MBR_FORMULA_MENGER_SPONGE ||
                                sc.uniform_formula == MBR_FORMULA_MANDELBULB);
  return pixels >= 262144 && (sc.is_hybrid || sc.uniform_formula != MBR_FORMULA_MENGER_SPONGE);
}

// Scratch bytes of a frame.
inline size_t staged_plain_bytes(const DevFrame &fr) {
  const size_t n = size_t(fr.width) * size_t(fr.row1 - fr.row0);
  return 256 + n * (sizeof(RefHit) + sizeof(double) * size_t(ao_tasks(fr)) + sizeof(float));
}

// The launch of a frame over its scratch.
inline RefLaunch ref_launch(const DevFrame &fr, void *scratch) {
  RefLaunch L;
  L.pixels = (long long)fr.width * (fr.row1 - fr.row0);
  char *p = static_cast<char *>(scratch);
  L.ctr = reinterpret_cast<Counters4 *>(p);
  L.hits = reinterpret_cast<RefHit *>(p + 256);
  L.ao_tasks = ao_tasks(fr);
  L.ao = reinterpret_cast<double *>(L.hits + L.pixels);
  L.shadow = reinterpret_cast<float *>(L.ao + L.pixels * L.ao_tasks);
  L.tiles_x = (fr.width + 7) / 8;
  L.shadow_tasks = (fr.shading_enable && fr.shadow_enable) ? 1 : 0;
  L.per = L.shadow_tasks + L.ao_tasks;
  L.div_tx = make_fastdiv(L.tiles_x);
  L.div_per = make_fastdiv(std::max(1, L.per));
  L.need_normal = fr.shading_enable || L.ao_tasks > 0 || fr.want_normal;
  L.refill_k = 2;
  return L;
}

// Stages P, N and S with the estimate PM of the marches and PN of the normals.
template <class PM, class PN, int FK, bool EXT, int V>
int ref_stages(const DevScene &sc, const DevFrame &fr, const RefLaunch &L, const DevOutputs &out, cudaStream_t s) {
  const long long most = (long long)sm_count() * 12;
  const int grid = int(std::min<long long>(most, (L.pixels + 127) / 128 + 1));
  const int grid_s = int(std::min<long long>(most, (L.pixels * std::max(1, L.per) + 127) / 128 + 1));
  ref_primary_kernel<PM, FK, V><<<grid, 128, 0, s>>>(sc, fr, L, out);
  if (L.need_normal) ref_normal_kernel<PN, FK, V><<<grid, 128, 0, s>>>(sc, fr, L, out);
  if (L.per > 0) ref_shade_kernel<PM, FK, EXT, V><<<grid_s, 128, 0, s>>>(sc, fr, L, out);
  count_launches(1 + (L.need_normal ? 1 : 0) + (L.per > 0 ? 1 : 0));
  return int(cudaGetLastError());
}

// A scene of one formula by settings key and none of the extensions: the
// formula is inlined in kernels of its own (a 320x240 pseudo-Kleinian view
// with 4 AO rays 13.6 -> 6.8 ms; in the kernels that carry every formula it is
// a call with the orbit in local memory).
inline int keyed_alone(const DevScene &sc) {
  const bool plain = !sc.is_hybrid && sc.n_nodes == 0 && sc.n_prims == 0 && !sc.limits && !sc.gbox && !sc.gsph &&
                     !sc.delta_de && sc.slot[0].d[P_WEIGHT] == 1.0;
  return plain ? sc.uniform_formula : 0;
}
template <class T, int V>
int ref_keyed_stages(int formula, const DevScene &sc, const DevFrame &fr, const RefLaunch &L, const DevOutputs &out,
                     cudaStream_t s, bool *taken) {
#define KEYED(FORMULA) \
  case FORMULA: return ref_stages<RefWhole<T, -FORMULA, false>, RefWhole<T, -FORMULA, true>, FK_ANY, false, V>(sc, fr, L, out, s)
  *taken = true;
  switch (formula) {
    KEYED(MBR_FORMULA_BOX_FOLD_BULB_POW2);
    KEYED(MBR_FORMULA_GENERALIZED_FOLD_BOX);
    KEYED(MBR_FORMULA_MENGER_MOD1);
    KEYED(MBR_FORMULA_PSEUDO_KLEINIAN_STD_DE);
    KEYED(MBR_FORMULA_PSEUDO_KLEINIAN);
    KEYED(MBR_FORMULA_ABOX_MOD11);
    KEYED(MBR_FORMULA_BOX_FOLD_BULB_POW2_V2);
    KEYED(MBR_FORMULA_PSEUDO_KLEINIAN_MOD4);
    KEYED(MBR_FORMULA_MANDELBULB_PUPUKU);
    KEYED(MBR_FORMULA_DIFS_HEXTGRID2);
    default: *taken = false; return 0;
  }
#undef KEYED
}
int ref_keyed_fp64(int formula, const DevScene &sc, const DevFrame &fr, const RefLaunch &L, const DevOutputs &out,
                   cudaStream_t s, bool *taken);
int ref_keyed_fp64_strict(int formula, const DevScene &sc, const DevFrame &fr, const RefLaunch &L, const DevOutputs &out,
                          cudaStream_t s, bool *taken);

template <class T, int V>
int launch_staged_plain_t(const DevScene &sc, const DevFrame &fr, const DevOutputs &out, void *scratch, void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const RefLaunch L = ref_launch(fr, scratch);
  int e = int(cudaMemsetAsync(L.ctr, 0, sizeof(Counters4), s));
  if (e) return e;
  const int F = sc.is_hybrid ? 0 : sc.uniform_formula;
#define WHOLE(FF, EXT) ref_stages<RefWhole<T, FF, false>, RefWhole<T, FF, true>, FK_ANY, EXT, V>(sc, fr, L, out, s)
#define PASS(FF, FK) ref_stages<RefPass<T, FF, false>, RefPass<T, FF, true>, FK, false, V>(sc, fr, L, out, s)
  if (scene_extended(sc)) {
    bool taken = false;
    const int formula = keyed_alone(sc);
    if (formula) e = V ? ref_keyed_fp64_strict(formula, sc, fr, L, out, s, &taken) : ref_keyed_fp64(formula, sc, fr, L, out, s, &taken);
    if (!taken) e = WHOLE(F_EXT, true);
  } else if (F == MBR_FORMULA_MANDELBULB) {
    e = PASS(MBR_FORMULA_MANDELBULB, FK_BULB);
  } else if (F == MBR_FORMULA_MANDELBOX) {
    e = PASS(MBR_FORMULA_MANDELBOX, FK_BOX);
  } else {
    e = orbit_blends(sc) ? WHOLE(0, false) : PASS(0, FK_ANY);
  }
#undef WHOLE
#undef PASS
  if (e) return e;
  ref_finish_kernel<V><<<sm_count() * 4, 256, 0, s>>>(fr, L, out);
  count_launches(1);
  return int(cudaGetLastError());
}

}  // namespace mbr
