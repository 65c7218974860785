// wavefront.cuh - the batched wavefront form, with FP32 or FP64 iteration: the
// kernels and the launch of one pipeline (launch_pipeline).  The pipelines are
// instantiated in wavefront32.cu, wavefront64.cu, wavefront_batch.cu and
// wavefront_hybrid.cu; the entry points are in wavefront.cu.
//
// A frame (or a batch of frames of uneven size) is rendered as a short
// pipeline of persistent kernels, each over a homogeneous task space:
//
//   stage P  one task per pixel:  the primary march + binary refinement
//            (cRenderWorker::RayMarching, src/render_worker.cpp:708-951);
//            misses are written out, hits are appended to a compact hit list
//   stage N  one task per hit:    the six central-difference DE samples of
//            CalculateNormals (src/shader_calculate_normals.cpp:40-125) and
//            the Lambert term of LightShading (src/shader_light_shading.cpp:61-72)
//   stage D  one thread per stage-S task: AO directions and start records
//   stage S  (1 + ao_rays) tasks per hit: the hard AuxShadow march
//            (src/shader_aux_shadow.cpp:94-321) and one AmbientOcclusion
//            march per AO direction (src/shader_ambient_occlusion.cpp:60-110)
//   stage F  one thread per hit: colour, 8-bit conversion, outputs
//
// Every march is a stream of distance requests p = origin + dir * t.  In
// stages P, N and S each lane holds one task; it runs 2 to 12 formula
// iterations (by formula) between warp votes and, once at most k lanes of the warp are still
// iterating, the lanes whose estimate is done take their march step and
// start their next request, or take the next task from the warp's share of
// the stage's queue (a chunk of tasks per atomicAdd on the stage's counter).  Because a warp only ever runs one
// kind of march, those steps stay converged and cheap, and divergent orbit
// lengths and march lengths cost only the k-lane wait.  A batch walks a job
// table (per-job camera, image size and formula parameters) with the same
// stages, captured once into a CUDA graph.
//
// Two precision policies share the stages:
//   Prec32  the formula iteration in FP32 (fast_formula.cuh) with the ray
//           origin, t and the refinement in FP64;
//   Prec64  the formula iteration in FP64 in the reference's operation order
//           (de_core.cuh) with the march arithmetic of the plain FP64 kernel.
// FP32 points resolve distances down to about 2^-24 of their coordinates;
// where the hit threshold of a view is not well above that (deep zooms, a
// camera inside the solid) the FP32 estimate is noise at the scale the march
// needs.  MBR_ENGINE_WAVEFRONT_AUTO chooses the policy per frame (per job in a
// batch) from the distance estimate at the camera: no ray meets the surface
// closer than that distance, so DE(camera) * threshold-per-unit-distance
// bounds the smallest hit threshold of the view from below.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "de_core.cuh"
#include "fast_formula.cuh"
#include "fastdiv.h"
#include "mbr_internal.h"
#include "pixel_ops.cuh"

namespace mbr {

// formula kinds of the iteration switch
enum { FK_ANY = 0, FK_BULB = 2, FK_MENGER = 7, FK_BOX = 8, FK_BOX_SIMPLE = 108 };

// One render job of a launch: its camera, image size and place in the queue.
struct WJob {
  double cam[3];
  double mrot[9];
  int32_t mrot_zero;
  int32_t width, height, tiles_x;
  int32_t row0, rows;      // the job renders rows [row0, row0 + rows) of its frame
  int32_t persp;           // mbr_projection
  int32_t legacy_y;        // legacy coordinate system (image y flipped)
  long long first;         // first work item of this job in the pixel queue
  long long pixel_offset;  // first pixel of this job in the outputs
  double fov, aspect;
  double resolution, detail;  // CalcDistThresh factors (1/height, detail level)
  float c0;                // threshold per unit distance: resolution * fov / detail (halved: equirectangular)
  float fovf;              // AO end distance per unit distance: fov (halved: equirectangular)
  float cthr;              // constant threshold (halved: equirectangular)
  FastDiv div_w, div_tx;   // divisions by width and tiles_x
};

// A surface hit, produced by stage P and completed by stages N and S.
struct HitRec {
  double px, py, pz;  // hit point
  double depth;       // scan distance t of the hit
  double thr;         // distThresh at the hit
  long long pix;      // output index
  int iters;          // iters of the last primary DE evaluation
  float nx, ny, nz;   // normal
  float shade;        // Lambert term before the shadow
  float shadow;       // AuxShadow result
  int job;
  unsigned int ray;   // pixel index within its job (RNG streams)
  // sum of the AO march results in 32.32 fixed point: integer atomics make
  // the sum independent of the order in which the AO marches finish
  unsigned long long ao_q;
};

__device__ __forceinline__ void ao_add(HitRec *r, double s) {
  atomicAdd(&r->ao_q, (unsigned long long)(s * 4294967296.0));
}

// Device-side counters of one launch (in the context's scratch).
struct Counters4 {
  unsigned long long pixels_next;  // stage P queue
  unsigned long long hits;         // hits appended by stage P
  unsigned long long normals_next; // stage N queue
  unsigned long long shade_next;   // stage S queue
};

// FP64 parameters of a non-hybrid formula: the slot's double parameters, read
// by the reference-order formulas of de_core.cuh, and the Compute settings.
struct WideParams {
  DevSlot slot;
  int formula, maxN, de_fn, min_n;
  int julia, add_c, check_bailout, box_simple;  // box_simple: as FastParams::box_simple
  double bailout;
  double jc[3];  // julia_c * fractal_constant_factor
  double cm[3];  // fractal_constant_factor
  // simple Mandelbox: folding limit, fR2, fR2/mR2, scale, bailout^2, and the
  // squared radii outside which the sphere fold's factor is fmx or 1 whatever
  // the rounding of the reciprocal (2^-40 away from mR2 and fR2)
  double lim, fr2, fmx, scale, bailout2, r2_inner, r2_outer;
  MbRot rot;  // Mandelbox rotations (the simple form is off when any is on)
};

__host__ __device__ inline WideParams load_wide_params(const DevScene &sc) {
  WideParams w;
  w.slot = sc.slot[0];
  w.formula = sc.slot[0].formula;
  w.maxN = sc.formula_maxiter;
  w.de_fn = sc.de_analytic;
  w.min_n = sc.min_n;
  w.julia = sc.julia;
  w.add_c = sc.slot[0].add_c;
  w.check_bailout = sc.slot[0].check_bailout;
  w.bailout = sc.slot[0].d[P_BAILOUT];
  for (int k = 0; k < 3; k++) {
    w.jc[k] = sc.julia_c[k] * sc.cmul[k];
    w.cm[k] = sc.cmul[k];
  }
  const DevSlot &s = sc.slot[0];
  const double L = s.d[P_MB_LIMIT], F = s.d[P_MB_FACTOR1];
  w.rot = sc.mbrot;
  w.box_simple = (s.formula == MBR_FORMULA_MANDELBOX && s.d[P_MB_VALUE] == 2.0 * L && L > 0.0 && F > 1.0 &&
                  !s.has_offset && !sc.mbrot.folds && !sc.mbrot.main) ? 1 : 0;
  w.lim = L;
  w.fr2 = s.d[P_MB_FR2];
  w.fmx = F;
  w.scale = s.d[P_MB_SCALE];
  w.bailout2 = w.bailout * w.bailout;
  w.r2_inner = w.fr2 / w.fmx * (1.0 - 0x1p-40);
  w.r2_outer = w.fr2 * (1.0 + 0x1p-40);
  return w;
}

struct Launch {
  const WJob *jobs;        // njobs entries (device)
  const FastParams *fps;   // per job (device), FP32 policy
  const WideParams *wps;   // per job (device), FP64 policy
  int njobs;
  long long total;         // pixel work items
  HitRec *hits;            // capacity: total
  float4 *sorg;            // per hit: FP32 hit point and threshold (stage S origins)
  float4 *sdir;            // per stage-S task: direction and end (w < 0: shadow, w == 0: no march)
  Counters4 *ctr;
  const int *gate;         // MBR_ENGINE_WAVEFRONT_AUTO: the policy flag; null: always run
  int gate_value;          // the flag value this pipeline runs under (0 FP32, 1 FP64)
  int refill_k;
  int layout;
  int ao_rays;             // AO tasks per hit (1 for fast AO)
  int ao_fast;             // fast AO: the AO task samples along the normal
  int shadow_tasks;        // 1 when the shadow march runs (shading && shadow)
  int want_normal;
  FastDiv div_per;         // division by shadow_tasks + ao_rays (set by launch_pipeline)
  // GI frames
  double *path_rad;              // radiance of every path of the launch
  HitRec *hits_next;             // the next level's vertex list
  unsigned long long *next_hits; // its counter
  FastDiv div_spp;               // division by samples per pixel
  int level;                     // bounce level of the vertex list in `hits`
  int row0;                      // first row of the launch
  int normal_slot;               // stats counter of stage N (K_NORMAL; K_GI in GI frames)
};

// Stage-S AO tasks per hit: the AO marches, or the one fast-AO task.
static inline int ao_tasks(const DevFrame &fr) { return fr.ao_fast ? 1 : fr.ao_rays; }

// True when this pipeline's kernels have nothing to do (the other precision
// renders the frame).
__device__ __forceinline__ bool gated_off(const Launch &L) { return L.gate && *L.gate != L.gate_value; }

__device__ __forceinline__ int job_of(const WJob *jobs, int n, long long idx) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].first <= idx) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__host__ __device__ inline int fast_kind(const FastParams &f) {
  if (f.formula == MBR_FORMULA_MANDELBOX) return f.box_simple ? FK_BOX_SIMPLE : FK_BOX;
  if (f.formula == MBR_FORMULA_MANDELBULB) return FK_BULB;
  return FK_MENGER;
}

__host__ __device__ inline int wide_kind(const WideParams &w) {
  if (w.formula == MBR_FORMULA_MANDELBOX) return w.box_simple ? FK_BOX_SIMPLE : FK_BOX;
  if (w.formula == MBR_FORMULA_MANDELBULB) return FK_BULB;
  return FK_MENGER;
}

__device__ __forceinline__ float fmadd(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fmadd(double a, double b, double c) { return fma(a, b, c); }

// Formula iterations between warp votes.  A vote (active mask, ballot, count)
// costs a few instructions per lane; orbits of the folding formulas run 7-19
// iterations per estimate, so a vote every 12 is cheap against the wait it
// causes (measured on the 1080p Mandelbox: 2 -> 7.5 ms, 6 -> 6.4 ms,
// 12 -> 6.3 ms per frame), while the Mandelbulb's 1-3 iterations per
// estimate at the usual views want a vote every 2.  The iterations between
// two votes are unrolled where one is a few dozen instructions; the
// reference-order policy's iteration (kHyb: a dispatch over formulas, library
// functions inlined) is not: four copies of it overran the instruction
// caches, half of all stall samples (1080p x 16 spp hybrid GI 338.8 ->
// 188.2 ms, an 800x600 frame with primitives 14.77 -> 8.59 ms); the FP64
// Mandelbox is by four (12: 33.8 ms on the 1080p deep zoom, 2 to 6: 31.4 ms).
template <int FK>
struct kVoteEvery {
  static constexpr int n = (FK == FK_BULB) ? 2 : ((FK == FK_ANY) ? 4 : 12);
};

// True when more than k bits of m are set.  k <= 2 takes the lowest set bit
// off on the ALU pipe instead of a POPC on the (eighth-rate) XU pipe.
__device__ __forceinline__ bool more_than(unsigned m, int k) {
  if (k == 0) return m != 0u;
  if (k == 1) return (m & (m - 1u)) != 0u;
  if (k == 2) {
    const unsigned a = m & (m - 1u);
    return (a & (a - 1u)) != 0u;
  }
  return __popc(m) > k;
}

// ============================================================================
// Precision policies: the per-lane state of one distance estimate, its
// start, one formula iteration and the final distance.
// ============================================================================
struct Prec32 {
  typedef Prec32 Normal;  // the policy of the normal stage
  typedef float D;  // distance and threshold arithmetic of the march
  typedef FastParams Params;
  enum { kWide = 0, kHyb = 0, kGI = 1, kFastAO = 1, kTotal = 0 };
  struct State {
    Z3 z, c;
    float dr, r2;
    int it;
  };
  __host__ __device__ static int kind(const Params &f) { return fast_kind(f); }
  __device__ static const Params &job_params(const Launch &L, int job) { return L.fps[job]; }

  template <int FK>
  __device__ static void start(State &e, const Params &fp, float qx, float qy, float qz) {
    e.z.x = qx;
    e.z.y = qy;
    e.z.z = qz;
    if (!fp.add_c) e.c = Z3{0.f, 0.f, 0.f};
    else if (fp.julia) e.c = Z3{fp.jc_x, fp.jc_y, fp.jc_z};
    else e.c = Z3{qx * fp.cm_x, qy * fp.cm_y, qz * fp.cm_z};
    e.dr = 1.f;
    e.it = 0;
    e.r2 = fmaf(qx, qx, fmaf(qy, qy, qz * qz));
  }
  template <int FK>
  __device__ static void start(State &e, const Params &fp, double qx, double qy, double qz) {
    start<FK>(e, fp, float(qx), float(qy), float(qz));
  }

  // One iteration; false once the orbit is done (bailout or maxN).
  template <int FK>
  __device__ static bool step(int kind, State &e, const Params &fp) {
    const int k = (FK == FK_ANY) ? kind : FK;
    if (k == FK_BOX_SIMPLE) it_mandelbox<true>(e.z, e.dr, e.c, fp);
    else if (k == FK_BOX) it_mandelbox<false>(e.z, e.dr, e.c, fp);
    else if (k == FK_BULB) it_mandelbulb(e.z, e.dr, e.c, fp, sqrtf(e.r2));
    else it_menger(e.z, e.dr, e.c, fp);
    e.it++;
    e.r2 = fmaf(e.z.x, e.z.x, fmaf(e.z.y, e.z.y, e.z.z * e.z.z));
    return e.r2 <= fp.bailout2 && e.it < fp.maxN;
  }

  template <int FK>
  __device__ static float distance(const State &e, const Params &fp, float detail, int &iters) {
    iters = (e.r2 > fp.bailout2) ? e.it : e.it + 1;
    return final_de(fp, e.r2, e.dr, iters, detail);
  }
};

// 2 clamp(z, -L, L) - z, for |z| > L the rounded 2L - z or -2L - z, else z itself
__device__ __forceinline__ double box_fold(double z, double L) {
  const double w = copysign(2.0 * L, z) - z;
  return fabs(z) > L ? w : z;
}

struct Prec64 {
  typedef Prec64 Normal;
  typedef double D;
  typedef WideParams Params;
  enum { kWide = 1, kHyb = 0, kGI = 1, kFastAO = 1, kTotal = 0 };
  struct State {
    double zx, zy, zz, cx, cy, cz, dr, r;
    int it, brk;  // iterations done; 1 when the loop ended by a break (bailout or NaN)
  };
  __host__ __device__ static int kind(const Params &w) { return wide_kind(w); }
  __device__ static const Params &job_params(const Launch &L, int job) { return L.wps[job]; }

  // Compute's start (compute_fractal.cpp:74-130): z = c = the point, DE = 1.
  // The simple Mandelbox keeps what is added to every pass in place of c.
  template <int FK>
  __device__ static void start(State &e, const Params &fp, double qx, double qy, double qz) {
    e.zx = qx;
    e.zy = qy;
    e.zz = qz;
    if (FK == FK_BOX_SIMPLE) {
      e.cx = !fp.add_c ? 0.0 : (fp.julia ? fp.jc[0] : qx * fp.cm[0]);
      e.cy = !fp.add_c ? 0.0 : (fp.julia ? fp.jc[1] : qy * fp.cm[1]);
      e.cz = !fp.add_c ? 0.0 : (fp.julia ? fp.jc[2] : qz * fp.cm[2]);
      e.dr = 1.0;
      e.r = fma(qx, qx, fma(qy, qy, qz * qz));
      e.it = 0;
      e.brk = 0;
      return;
    }
    e.cx = qx;
    e.cy = qy;
    e.cz = qz;
    e.dr = 1.0;
    e.r = len4<double, false>(V4<double>{qx, qy, qz, 0.0});
    e.it = 0;
    e.brk = 0;
  }

  // One pass of the Compute loop body for a non-hybrid scene, as
  // calc_distance<double, F, false> runs it (compute_fractal.cpp:170-321).
  // The simple Mandelbox (folding value 2 * limit, no offset) runs the fold
  // rewrites of fast_formula.cuh in FP64: box fold 2 clamp(z, -L, L) - z,
  // sphere-fold factor clamp(fR2 / r2, 1, fR2 / mR2) with a correctly rounded
  // reciprocal, scale and c-addition fused, bailout tested on |z|^2 and |z|
  // taken once when the orbit ends; the result differs from the reference's
  // operation order in the last bits only.  The FP64 minimum and maximum are
  // several instructions each, so the folds are a compare and a select, and
  // the reciprocal is taken only between the radii (with the fold as minimum
  // and maximum and the reciprocal in every pass: 86 instead of about 50
  // instructions a pass; the 1080p deep zoom 57.9 -> 28.4 ms, a stage-S tail of
  // orbits that never leave 96 -> 66 ms.  With the reciprocal in every pass
  // 32.2 ms; two passes per bailout test, the second speculative, 30.5 ms).
  template <int FK>
  __device__ static bool step(int kind, State &e, const Params &fp) {
    const int k = (FK == FK_ANY) ? kind : FK;
    if (k == FK_BOX_SIMPLE) {
      const double L = fp.lim;
      const double x = box_fold(e.zx, L), y = box_fold(e.zy, L), z = box_fold(e.zz, L);
      const double r2 = fma(x, x, fma(y, y, z * z));
      double fs = r2 <= fp.r2_inner ? fp.fmx : 1.0;
      if (r2 > fp.r2_inner && r2 < fp.r2_outer) {
        fs = fp.fr2 * __drcp_rn(r2);
        fs = fs < 1.0 ? 1.0 : fs;
        fs = fs > fp.fmx ? fp.fmx : fs;
      }
      const double s = fs * fp.scale;
      e.dr = fma(e.dr, fabs(s), 1.0);  // fs > 0: |fs scale| is fs |scale|
      e.zx = fma(x, s, e.cx);
      e.zy = fma(y, s, e.cy);
      e.zz = fma(z, s, e.cz);
      e.it++;
      e.r = fma(e.zx, e.zx, fma(e.zy, e.zy, e.zz * e.zz));  // |z|^2: distance() takes the root
      if (!(e.r <= fp.bailout2)) {  // a single formula always checks its bailout
        e.brk = 1;
        return false;
      }
      return e.it < fp.maxN;
    }
    V4<double> z{e.zx, e.zy, e.zz, 0.0};
    const V4<double> last = z;
    double de = e.dr;
    if (k == FK_BULB) f_mandelbulb<double>(z, e.r, de, fp.slot);
    else if (k == FK_MENGER) f_menger<double, false>(z, de, fp.slot);
    else f_mandelbox<double, false, true>(z, de, fp.slot, &fp.rot);
    if (fp.add_c) {
      if (fp.julia) {
        z.x = z.x + fp.jc[0];
        z.y = z.y + fp.jc[1];
        z.z = z.z + fp.jc[2];
      } else {
        z.x = z.x + e.cx * fp.cm[0];
        z.y = z.y + e.cy * fp.cm[1];
        z.z = z.z + e.cz * fp.cm[2];
      }
    }
    e.it++;
    e.dr = de;
    if (nan4<double, false>(z)) {  // revert to the last finite orbit point
      e.zx = last.x;
      e.zy = last.y;
      e.zz = last.z;
      e.r = len4<double, false>(last);
      e.brk = 1;
      return false;
    }
    e.zx = z.x;
    e.zy = z.y;
    e.zz = z.z;
    e.r = len4<double, false>(z);
    if (fp.check_bailout && e.r > fp.bailout) {
      e.brk = 1;
      return false;
    }
    return e.it < fp.maxN;
  }

  // Final DE and CalculateDistanceSimple's clamps (compute_fractal.cpp:561-621,
  // calculate_distance.cpp:569, 604-605).
  template <int FK>
  __device__ static double distance(const State &e, const Params &fp, double detail, int &iters) {
    iters = e.brk ? e.it : e.it + 1;
    const double r = FK == FK_BOX_SIMPLE ? sqrt(e.r) : e.r, DE = e.dr;
    double d;
    if (DE > 0.0) {
      if (fp.de_fn == 2) d = (r > 1.0) ? 0.5 * r * log(r) / DE : 0.0;
      else if (fp.de_fn == 1) d = r / DE;
      else if (fp.de_fn == 3) d = (r - 2.0) / DE;
      else d = r;
    } else {
      d = r;
    }
    if (iters < fp.min_n && d < detail) d = detail;
    if (d < 0.0) d = 0.0;
    if (d > 10.0) d = 10.0;
    return d;
  }
};

// Hybrid sequences and extended scenes (single-frame launches): the FP32
// iteration of calc_distance<float, 0 or F_EXT, false> one pass at a time -
// the slot of iteration i from the sequence table (CreateSequence), per-slot
// formula, c-addition, weight blend, NaN revert and per-slot bailout
// (compute_fractal.cpp:170-321), and the DE function of the final distance
// (:503-557).  The scene is a launch parameter, so a slot known at compile
// time is read as constant operands.
struct HybParams {
  DevScene sc;
};

// What a kernel's iteration carries.  Every formula of a kernel is in the
// instruction stream of its loop, the Mandelbulb's with six library
// functions; a kernel for all of them spends its time fetching instructions.
enum HybFeature {
  HB_BULB = 1,
  HB_BOX = 2,
  HB_MENGER = 4,
  HB_SEQ = 8,     // a sequence: the slot changes with the iteration
  HB_BLEND = 16,  // a slot's weight is not 1
  HB_EXT = 32,    // limit box, global folds, primitives, Mandelbox rotations, every DE function
  HB_ALL = 64,    // the formulas beyond the three (with HB_EXT)
  HB_NORMAL = 128 // the normal stage (see square_of)
};

template <int FEAT>
struct PrecHybT {
  typedef float D;
  typedef HybParams Params;
  typedef PrecHybT<FEAT | HB_NORMAL> Normal;  // the policy of the normal stage
  static constexpr bool EXT = (FEAT & HB_EXT) != 0, ALL = (FEAT & HB_ALL) != 0;
  static constexpr bool KEEP_R = (FEAT & (HB_ALL | HB_BLEND)) != 0;  // the general kernels
  // the general kernels take GI frames of every scene and fast AO
  enum { kWide = 0, kHyb = 1, kGI = (FEAT & HB_SEQ) != 0, kFastAO = (FEAT & HB_BLEND) != 0, kTotal = 0 };
  struct State {
    float zx, zy, zz, cx, cy, cz, dr, r;  // r: |z|, with KEEP_R only
    int it, brk;
  };
  __host__ __device__ static int kind(const Params &) { return FK_ANY; }

  // |z|^2 with its fused operations spelled out, so that every kernel and
  // every feature set rounds alike: x before y, at the starting point of a
  // normal sample y before x, the order of the general kernels, whose len4 the
  // compiler fuses (tests/test_gpu_hybrid_rounding.py compares their bits).
  __device__ static float square_of(const V4<float> &z) { return fmaf(z.z, z.z, fmaf(z.x, z.x, __fmul_rn(z.y, z.y))); }
  __device__ static float start_square_of(const V4<float> &z) {
    if (!(FEAT & HB_NORMAL)) return square_of(z);
    return fmaf(z.z, z.z, fmaf(z.y, z.y, __fmul_rn(z.x, z.x)));
  }

  // smooth4 (SmoothCVector) in the sequences' kernel, its first length given:
  // |z| as the pass before rounded it, except in every fourth pass, which
  // computes it anew with the other fused operation first.  Which of the two it
  // is shows in the last bits only, but also in iteration counts and 8-bit
  // colours of single pixels; the orbits keep the rounding of a loop whose
  // passes come in groups of four (tests/test_gpu_blended_bits.py).
  __device__ static float last_length(int i, float r, const V4<float> &z) {
    if (i & 3) return r;
    if (FEAT & HB_NORMAL) return sqrtf(square_of(z));
    return sqrtf(fmaf(z.z, z.z, fmaf(z.y, z.y, __fmul_rn(z.x, z.x))));
  }
  __device__ static V4<float> blend(const V4<float> &v1, const V4<float> &v2, double k, float l1) {
    if (k <= 0.0) return v1;
    const float kk = float(k), nk = float(1.0 - k);
    const float l2 = len4<float, false>(v2);
    const float length = l1 * nk + l2 * kk;
    const V4<float> t{v1.x * nk + v2.x * kk, v1.y * nk + v2.y * kk, v1.z * nk + v2.z * kk, 0.0f};
    const float lt = len4<float, false>(t);
    if (lt > 0.0f) return V4<float>{t.x / lt * length, t.y / lt * length, t.z / lt * length, 0.0f};
    return v1;
  }

  template <int FK>
  __device__ static void start(State &e, const Params &, float qx, float qy, float qz) {
    e.zx = qx;
    e.zy = qy;
    e.zz = qz;
    e.cx = qx;
    e.cy = qy;
    e.cz = qz;
    e.dr = 1.0f;
    if (KEEP_R) e.r = len4<float, false>(V4<float>{qx, qy, qz, 0.0f});
    e.it = 0;
    e.brk = 0;
  }
  template <int FK>
  __device__ static void start(State &e, const Params &fp, double qx, double qy, double qz) {
    start<FK>(e, fp, float(qx), float(qy), float(qz));
  }

  template <int FK>
  __device__ static bool step(int, State &e, const Params &fp) {
    const DevScene &sc = fp.sc;
    const int i = e.it;
    const int k = (FEAT & HB_SEQ) ? ((i < sc.length) ? int(sc.seq[i]) : int(sc.seq[0])) : 0;
    const DevSlot &s = sc.slot[k];
    V4<float> z{e.zx, e.zy, e.zz, 0.0f};
    const V4<float> last = z;
    float de = e.dr;
    float r = e.r;
    if (!KEEP_R && ((FEAT & HB_BULB) || EXT)) r = sqrtf(i == 0 ? start_square_of(z) : square_of(z));
    if (EXT) global_folds<float, false>(sc, z, r, de);
    const V4<float> tempZ = z;
    const float tempDE = de;
    if (!(FEAT & HB_BLEND) || s.d[P_WEIGHT] > 0.0) {
      if constexpr (ALL) {
        // the Aexion, the one formula that replaces c, is 4-D and never runs here
        V4<float> c{e.cx, e.cy, e.cz, 0.0f};
        AuxX<float> ax{1.0f, 0.0f, 0.0f, 1.0f, 1000.0f, c};  // formulas with orbit state do not run here (check_supported)
        formula_dispatch<float, false, true, true>(s.formula, z, r, de, s, &sc.mbrot, &sc.ifs, i, c, ax);
      } else {
        constexpr int F = FEAT & (HB_BULB | HB_BOX | HB_MENGER);
        if ((FEAT & HB_BULB) && (F == HB_BULB || s.formula == MBR_FORMULA_MANDELBULB))
          f_mandelbulb<float>(z, r, de, s);
        else if ((FEAT & HB_BOX) && (!(FEAT & HB_MENGER) || s.formula == MBR_FORMULA_MANDELBOX))
          f_mandelbox<float, false, EXT>(z, de, s, &sc.mbrot);
        else
          f_menger<float, false, true>(z, de, s);
      }
    }
    if (s.add_c) {
      if (sc.julia) {
        z.x = add_julia<float>(sc, z.x, 0);
        z.y = add_julia<float>(sc, z.y, 1);
        z.z = add_julia<float>(sc, z.z, 2);
      } else {
        z.x = fused<float>(e.cx, sc.fcmul[0], z.x);
        z.y = fused<float>(e.cy, sc.fcmul[1], z.y);
        z.z = fused<float>(e.cz, sc.fcmul[2], z.z);
      }
    }
    if ((FEAT & HB_BLEND) && sc.is_hybrid) {
      const double kw = s.d[P_WEIGHT];
      if (kw < 1.0) {
        z = EXT ? smooth4<float, false>(tempZ, z, kw) : blend(tempZ, z, kw, last_length(i, e.r, tempZ));
        de = de * float(kw) + tempDE * float(1.0 - kw);
      }
    }
    e.it = i + 1;
    e.dr = de;
    if (nan4<float, false>(z)) {
      e.zx = last.x;
      e.zy = last.y;
      e.zz = last.z;
      if (KEEP_R) e.r = len4<float, false>(last);
      e.brk = 1;
      return false;
    }
    e.zx = z.x;
    e.zy = z.y;
    e.zz = z.z;
    bool out;
    if (KEEP_R) {
      e.r = len4<float, false>(z);
      out = e.r > P<float>(s, P_BAILOUT);
    } else {  // the same outcome without the root (bailout.h)
      out = square_of(z) > P<float>(s, P_BAILOUT_R2);
    }
    if (s.check_bailout && out) {
      e.brk = 1;
      return false;
    }
    return e.it < sc.formula_maxiter;
  }

  template <int FK>
  __device__ static float distance(const State &e, const Params &fp, float detail, int &iters) {
    const DevScene &sc = fp.sc;
    if (EXT && sc.limits) {  // outside the limit box: its distance (the iteration is not used)
      const float lbd = limit_box_distance<float>(sc, e.cx, e.cy, e.cz);
      if (lbd > detail) {
        iters = 0;
        return lbd;
      }
    }
    iters = e.brk ? e.it : e.it + 1;
    const V4<float> z{e.zx, e.zy, e.zz, 0.0f};
    float d = final_distance<float, EXT ? F_EXT : 0, false>(sc, z, KEEP_R ? e.r : sqrtf(square_of(z)), e.dr);
    if (iters < sc.min_n && d < detail) d = detail;
    if (d < 0.0f) d = 0.0f;
    if (d > 10.0f) d = 10.0f;
    if (EXT) {  // the union with the primitives, at the request point c
      for (int k = 0; k < sc.n_prims; k++) {
        const float pd = prim_distance<float>(sc.prim[k], e.cx, e.cy, e.cz);
        if (pd < d) d = pd;
      }
    }
    return d;
  }
};

// The formula parameters a stage reads: a batch's lanes hold their job's copy,
// a single frame refers to the launch parameter.
template <bool MULTI, class P>
struct StageParams {
  typedef typename P::Params type;
};
template <class P>
struct StageParams<false, P> {
  typedef const typename P::Params &type;
};

// ============================================================================
// The persistent skeleton: refill lanes from a task counter, iterate, step.
// Stage provides (Real: the precision of its request points, D: of its distances):
//   bool start(long long task, Real &qx, &qy, &qz)   - first request (false: nothing to march)
//   bool step(D d, int iters, Real &qx, &qy, &qz)    - consume a result; true: next request
//   const Params &params()  - formula of the current task
//   int kind()              - formula kind (FK_ANY launches)
//   D detail()              - detail size of the current request
// ============================================================================
// fpk: the formula parameters of a single-job launch, the kernel parameter
// itself, so that the iteration reads its constants as constant-bank operands
// (a copy held in the stage is read through indexed constant loads); batch
// launches (Stage::kMulti) read the per-job copy the stage loads.
template <int FK, class P, class Stage>
__device__ __forceinline__ void run_stage(Stage &S, const typename P::Params &fpk, unsigned long long *counter,
                                          long long total, int refill_k, unsigned int *my_de,
                                          unsigned long long *my_iters) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned lanemask_lt = (1u << lane) - 1u;
  typename P::State e = {};
  bool has = false, iterating = false, drained = false;
  long long q_next = 0, q_end = 0;  // the warp's unstarted tasks [q_next, q_end)
  const long long warps = (long long)gridDim.x * (long long)(blockDim.x >> 5);
  const int chunk = (int)min(64ll, max(1ll, total / (32ll * max(warps, 1ll))));
  unsigned int de_n = 0;
  unsigned long long it_n = 0;
  for (;;) {
    // ---- refill lanes without a task from the warp's share of the queue.
    // A warp takes max(chunk, waiting lanes) tasks per atomic on the stage's
    // counter; chunk grows with the tasks per resident warp (up to 64), so a
    // large queue costs fewer atomics and dependent waits, while a small one
    // keeps its tail balanced.
    unsigned need = __ballot_sync(FULL, !has && !drained);
    while (need) {
      const int waiting = __popc(need);
      if (q_next >= q_end) {
        const int take_n = max(chunk, waiting);
        unsigned long long base = 0ull;
        if (lane == 0) base = atomicAdd(counter, (unsigned long long)take_n);
        base = __shfl_sync(FULL, base, 0);
        if ((long long)base >= total) {
          drained = true;
          break;
        }
        q_next = (long long)base;
        q_end = min((long long)base + take_n, total);
      }
      const int take = (int)min((long long)waiting, q_end - q_next);
      const int rank = __popc(need & lanemask_lt);
      if (((need >> lane) & 1u) && rank < take) {
        typename Stage::Real qx, qy, qz;
        if (S.start(q_next + rank, qx, qy, qz)) {
          P::template start<FK>(e, Stage::kMulti ? S.params() : fpk, qx, qy, qz);
          has = true;
          iterating = true;
        }
      }
      q_next += take;
      need = __ballot_sync(FULL, !has && !drained);
    }
    if (!__any_sync(FULL, iterating)) break;
    const int k = drained ? 0 : refill_k;
    // ---- formula iterations, kVoteEvery<FK> between votes, until <= k lanes
    // still iterate.  A lane whose orbit ends leaves the loop by a branch, so
    // the remaining lanes run the iteration without select instructions for
    // finished ones; the vote counts the lanes still in the loop.
    const typename P::Params &fp = Stage::kMulti ? S.params() : fpk;
    const int kind = S.kind();
    if (iterating) {
      for (;;) {
        bool ended = false;
#pragma unroll (P::kHyb ? 1 : (P::kWide && FK == FK_BOX_SIMPLE ? 4 : kVoteEvery<FK>::n))
        for (int u = 0; u < kVoteEvery<FK>::n; u++) {
          if (!P::template step<FK>(kind, e, fp)) {
            ended = true;
            break;
          }
        }
        if (ended) {
          iterating = false;
          break;
        }
        if (!more_than(__ballot_sync(__activemask(), 1), k)) break;
      }
    }
    __syncwarp();
    // ---- lanes whose estimate is done: distance, then the march step
    if (has && !iterating) {
      int iters;
      const typename P::D d = P::template distance<FK>(e, fp, S.detail(), iters);
      de_n++;
      if constexpr (P::kTotal) it_n += (unsigned long long)e.total;  // the iterations of all orbits of the estimate
      else it_n += (unsigned long long)iters;
      typename Stage::Real qx, qy, qz;
      if (S.step(d, iters, qx, qy, qz)) {
        P::template start<FK>(e, Stage::kMulti ? S.params() : fpk, qx, qy, qz);
        iterating = true;
      } else {
        has = false;
      }
    }
  }
  *my_de += de_n;
  *my_iters += it_n;
}

// Adds this warp's counts to the launch stats (no block barrier: a warp of a
// persistent CTA leaves as soon as its queue is drained).
__device__ __forceinline__ void flush_counts(const DevOutputs &out, unsigned int my_de, unsigned long long my_iters,
                                             int slot_a, unsigned int val_a, int slot_b, unsigned int val_b) {
  if (!out.stats) return;
  const unsigned FULL = 0xffffffffu;
  unsigned long long *st = reinterpret_cast<unsigned long long *>(out.stats);
  const unsigned de = __reduce_add_sync(FULL, my_de);
  const unsigned a = __reduce_add_sync(FULL, val_a);
  const unsigned b = __reduce_add_sync(FULL, val_b);
  unsigned long long it = my_iters;
  for (int o = 16; o > 0; o >>= 1) it += __shfl_down_sync(FULL, it, o);
  if ((threadIdx.x & 31) == 0) {
    if (de) atomicAdd(st + K_DE, (unsigned long long)de);
    if (a) atomicAdd(st + slot_a, (unsigned long long)a);
    if (b) atomicAdd(st + slot_b, (unsigned long long)b);
    if (it) atomicAdd(st + K_ITERS, it);
  }
}

// Blocks of 256 per SM that a stage's registers have to leave room for.  The
// FP64 Mandelbox trades registers for warps (1080p deep zoom, stage P at
// 128 / 85 / 64 registers 3.14 / 2.87 / 2.74 ms, stage S 24.8 / 24.1 / 24.2 ms);
// its batch form holds the job's parameters in registers too, and stage S ends
// in a tail of single long orbits, which spills would lengthen (P 82 / 78 ms,
// S 67 / 82 ms at 128 / 85).  The reference-order kernels of few formulas are
// latency-bound: 1080p x 16 spp GI, stage GP at no bound (88 registers) / 85 /
// 64 / 51: 87.2 / 80.4 / 76.4 / 76.8 ms; an 800x600 Mandelbox with primitives,
// stage P at 107 / 128 / 85 / 64: 1.27 / 1.20 / 1.35 / 1.40 ms, stage S 2.46 /
// 2.33 / 2.00 / 2.14 ms.  The FP32 Mandelbox's stage P, from kFewPixels pixels:
// frames without AO over six views and scales from -2 to 3, time at no bound (89
// registers) over that at 85 / 64 / 51: 1920x1080 1.00 to 1.05 / 0.98 to 1.08 /
// 0.94 to 1.06, 1280x720 1.00 to 1.06 / 0.95 to 1.10 / 0.82 to 1.08, 640x360 0.99
// to 1.02 / 0.94 to 1.03 / 0.89 to 1.03.  64 registers are best on the view that
// fills the frame with short orbits and cost where orbits are long; 85 cost 1 %
// at most.  From kManyPixels 64, which there cost on no view more than no bound
// (the benchmark frame 5.94 ms, at 85 6.00); below kFewPixels no bound: 320x180
// 0.98 to 0.99 / 0.91 to 0.95 / 0.89 to 0.94.  (The Mandelbulb's is best
// unbounded, 512x512: 321 / 366 / 317 / 346 us.)
template <int FK, bool MULTI, class P>
struct kMinBlocks {
  static constexpr bool box64 = P::kWide && FK == FK_BOX_SIMPLE;
  static constexpr bool lean = P::kHyb && !P::kFastAO;  // a reference-order kernel of few formulas
  static constexpr bool box32 = !P::kWide && !P::kHyb && !MULTI && FK == FK_BOX_SIMPLE;
  static constexpr int primary = box64 ? (MULTI ? 3 : 4) : lean ? 2 : box32 ? 3 : 0;  // 0: none asked
  static constexpr int shade = box64 ? (MULTI ? 2 : 3) : lean ? 3 : 0;
  static constexpr int gi = lean ? 4 : 0;
};

// ============================================================================
// Stage P: primary march with binary refinement, one task per pixel.
// ============================================================================
template <bool MULTI, class P>
struct PrimaryStage {
  typedef double Real;
  static constexpr bool kMulti = MULTI;
  typedef typename P::D D;
  const DevFrame &fr;
  const Launch &L;
  const DevOutputs &out;
  const WJob *jb;
  typename StageParams<MULTI, P>::type fp;
  int kd;
  int job;
  // ray
  double dx, dy, dz, ox, oy, oz, t, stp, dir_len;
  double lx, ly, lz;  // previous request point (dead-ray check)
  D thr, c0, dist_prev, search_limit;
  int phase, sub, count, last_iters;
  unsigned int pm, ray, binary_de;
  long long pix;

  __device__ const typename P::Params &params() const { return fp; }
  __device__ int kind() const { return kd; }
  __device__ D detail() const { return thr; }

  // distThresh at the request point (render_worker.cpp:653-679): FP64 from
  // |camera - q| as the plain kernel computes it; FP32 from t
  // with the tail of thresh_tail: an equirectangular view halves it (in the
  // FP32 form inside c0 and `cthr`), advanced quality clamps it
  __device__ void set_thr(double qx, double qy, double qz) {
    if (P::kWide) {
      double v;
      if (fr.constant_de_threshold) {
        v = fr.de_thresh;
      } else {
        const double ax = jb->cam[0] - qx, ay = jb->cam[1] - qy, az = jb->cam[2] - qz;
        const double l = sqrt(ax * ax + ay * ay + az * az);
        v = l * jb->resolution * jb->fov / jb->detail;
      }
      thr = D(thresh_tail(fr, jb->persp, v));
    } else {
      float v = fr.constant_de_threshold ? jb->cthr : float(t) * float(c0);
      if (fr.adv_quality) {
        if (v > float(fr.detail_size_max)) v = float(fr.detail_size_max);
        if (v < float(fr.detail_size_min)) v = float(fr.detail_size_min);
      }
      thr = D(v);
    }
  }

  __device__ void point(double &qx, double &qy, double &qz) {
    qx = fma(dx, t, ox);
    qy = fma(dy, t, oy);
    qz = fma(dz, t, oz);
    set_thr(qx, qy, qz);
  }

  // The next march point; false when the ray is stuck: the point did not
  // move or is not finite (render_worker.cpp:747-756).
  __device__ bool advance(double &qx, double &qy, double &qz) {
    const double nx = fma(dx, t, ox), ny = fma(dy, t, oy), nz = fma(dz, t, oz);
    if ((nx == lx && ny == ly && nz == lz) || !(isfinite(nx) && isfinite(ny) && isfinite(nz))) return false;
    lx = nx;
    ly = ny;
    lz = nz;
    qx = nx;
    qy = ny;
    qz = nz;
    set_thr(qx, qy, qz);
    return true;
  }

  __device__ bool start(long long idx, double &qx, double &qy, double &qz) {
    if constexpr (MULTI) {
      job = job_of(L.jobs, L.njobs, idx);
      jb = &L.jobs[job];
      fp = P::job_params(L, job);
      kd = P::kind(fp);
    }
    const unsigned long long local = (unsigned long long)(idx - jb->first);
    int x, y;
    if (L.layout == 1) {
      const unsigned long long tile = local >> 5;
      const int w = int(local & 31);
      const unsigned long long ty = fdiv(tile, jb->div_tx);
      x = int(tile - ty * (unsigned long long)jb->tiles_x) * 8 + (w & 7);
      y = int(ty) * 4 + (w >> 3);
    } else {
      const unsigned long long yy = fdiv(local, jb->div_w);
      x = int(local - yy * (unsigned long long)jb->width);
      y = int(yy);
    }
    if (x >= jb->width || y >= jb->rows) return false;  // padding of the last tile row/column
    y += jb->row0;
    ray = unsigned(y) * unsigned(jb->width) + unsigned(x);
    pix = jb->pixel_offset + (long long)ray;
    // camera ray (render_worker.cpp:155-163, 247, 326-327)
    const double ix = (1.0 / double(jb->width) * double(x) + -0.5) * jb->aspect;
    const double iy = jb->legacy_y ? 1.0 / double(jb->height) * double(y) + -0.5
                                   : -1.0 / double(jb->height) * double(y) + 0.5;
    double vx = ix * jb->fov, vy = 1.0, vz = iy * jb->fov;
    if (jb->persp != MBR_PROJECTION_THREE_POINT) {
      if (hemisphere_cut(jb->persp, jb->fov, ix, iy)) {
        last_iters = 0;
        write_miss(true);
        return false;
      }
      const D3 v = projection_dir(jb->persp, jb->fov, ix, iy);
      vx = v.x;
      vy = v.y;
      vz = v.z;
    }
    double n = 1.0 / sqrt(vx * vx + vy * vy + vz * vz);
    vx *= n;
    vy *= n;
    vz *= n;
    if (!jb->mrot_zero) {
      const double *m = jb->mrot;
      const double rx = m[0] * vx + m[1] * vy + m[2] * vz;
      const double ry = m[3] * vx + m[4] * vy + m[5] * vz;
      const double rz = m[6] * vx + m[7] * vy + m[8] * vz;
      vx = rx;
      vy = ry;
      vz = rz;
    }
    n = 1.0 / sqrt(vx * vx + vy * vy + vz * vz);
    dx = vx * n;
    dy = vy * n;
    dz = vz * n;
    dir_len = sqrt(dx * dx + dy * dy + dz * dz);
    ox = jb->cam[0];
    oy = jb->cam[1];
    oz = jb->cam[2];
    c0 = D(jb->c0);
    t = 0.0;
    stp = 0.0;
    phase = 0;
    sub = 0;
    count = 0;
    last_iters = 0;
    thr = D(0);
    lx = ly = lz = 1e30;
    if (fr.jitter) pm = pm_for_ray(ray, fr.seed).s;
    if (!advance(qx, qy, qz)) {  // a camera that is not finite: stuck at once
      write_hit();
      return false;
    }
    return true;
  }

  // cut: a fish-eye-cut pixel, not traced and black
  __device__ void write_miss(bool cut = false) {
    float rgb[3] = {fr.background[0], fr.background[1], fr.background[2]};
    if (cut) rgb[0] = rgb[1] = rgb[2] = 0.0f;
    if (out.depth) out.depth[pix] = 1e20;
    if (out.iters) out.iters[pix] = last_iters;
    if (out.hit) out.hit[pix] = 0;
    if (out.normal) {
      out.normal[3 * pix + 0] = 0.f;
      out.normal[3 * pix + 1] = 0.f;
      out.normal[3 * pix + 2] = 0.f;
    }
    if (out.shade) out.shade[pix] = 0.f;
    if (out.ao) out.ao[pix] = 1.0f;
    if (out.rgb) {
      out.rgb[3 * pix + 0] = rgb[0];
      out.rgb[3 * pix + 1] = rgb[1];
      out.rgb[3 * pix + 2] = rgb[2];
    }
    if (out.rgb8) to_rgb8(fr, rgb, &out.rgb8[3 * pix]);
  }

  __device__ void write_hit() {
    const unsigned long long h = atomicAdd(&L.ctr->hits, 1ull);
    HitRec &r = L.hits[h];
    r.px = fma(dx, t, ox);
    r.py = fma(dy, t, oy);
    r.pz = fma(dz, t, oz);
    r.depth = t;
    r.pix = pix;
    r.thr = double(thr);
    r.iters = last_iters;
    r.nx = 1.f;
    r.ny = 0.f;
    r.nz = 0.f;
    r.shade = 0.f;
    r.shadow = 1.f;
    r.ao_q = 0ull;
    r.job = MULTI ? job : 0;
    r.ray = ray;
  }

  // reference binary search step (render_worker.cpp:854-912)
  __device__ bool binary_check(double &qx, double &qy, double &qz) {
    if (sub >= fr.binary_steps || (dist_prev < thr && dist_prev > thr * search_limit)) {
      write_hit();
      return false;
    }
    if (dist_prev > thr) t += stp;
    else if (dist_prev < thr * search_limit) t -= stp;
    point(qx, qy, qz);
    return true;
  }

  __device__ bool step(D d, int iters, double &qx, double &qy, double &qz) {
    last_iters = iters;
    if (phase == 1) {
      binary_de++;
      dist_prev = d;
      stp *= 0.5;
      sub++;
      return binary_check(qx, qy, qz);
    }
    count++;
    if (d < thr) {
      stp *= 0.5;
      sub = 0;
      dist_prev = d;
      phase = 1;
      return binary_check(qx, qy, qz);
    }
    double jit = 1.0;
    if (fr.jitter) {
      ParkMiller p;
      p.s = pm;
      jit = 1.0 - tenthousandths(p.random(1000));
      pm = p.s;
    }
    if (P::kWide) {
      stp = (double(d) - 0.5 * double(thr)) * fr.de_factor * jit;
      stp = step_limit(fr, stp, double(thr));
      t += stp / dir_len;
    } else {
      stp = double((float(d) - 0.5f * float(thr)) * float(fr.de_factor)) * jit;
      if (fr.adv_quality) stp = step_limit(fr, stp, double(thr));
      else if (stp > 3.0) stp = 3.0;
      t += stp;
    }
    if (t > fr.view_distance_max || count >= fr.max_steps) {
      write_miss();
      return false;
    }
    if (!advance(qx, qy, qz)) {  // stuck: a hit where it stands, without refinement
      write_hit();
      return false;
    }
    return true;
  }
};

template <int FK, bool MULTI, class P, int BLOCKS = kMinBlocks<FK, MULTI, P>::primary>
__global__ void __launch_bounds__(256, BLOCKS) primary_kernel(const __grid_constant__ DevFrame fr,
                                                      const __grid_constant__ typename P::Params fp0,
                                                      const __grid_constant__ WJob job0,
                                                      const __grid_constant__ Launch L, DevOutputs out) {
  if (gated_off(L)) return;
  PrimaryStage<MULTI, P> S{fr, L, out, &job0, fp0, P::kind(fp0), 0};
  S.search_limit = typename P::D(1.0 - 0.001 * fr.detail_level);
  S.binary_de = 0;
  unsigned int my_de = 0;
  unsigned long long my_iters = 0;
  run_stage<FK, P>(S, fp0, &L.ctr->pixels_next, L.total, L.refill_k, &my_de, &my_iters);
  flush_counts(out, my_de, my_iters, K_MARCH, my_de - S.binary_de, K_BINARY, S.binary_de);
}

// ============================================================================
// Stage N: normals + Lambert term, one task per hit.
// ============================================================================
template <bool MULTI, class P>
struct NormalStage {
  typedef double Real;
  static constexpr bool kMulti = MULTI;
  typedef typename P::D D;
  const DevFrame &fr;
  const Launch &L;
  typename StageParams<MULTI, P>::type fp;
  int kd;
  HitRec *r;
  double ox, oy, oz, delta;
  D thr, nx, ny, nz;
  int sub;

  __device__ const typename P::Params &params() const { return fp; }
  __device__ int kind() const { return kd; }
  __device__ D detail() const { return thr; }

  __device__ void point(double &qx, double &qy, double &qz) {
    const double dd = (sub & 1) ? -delta : delta;
    const int axis = sub >> 1;
    qx = ox + (axis == 0 ? dd : 0.0);
    qy = oy + (axis == 1 ? dd : 0.0);
    qz = oz + (axis == 2 ? dd : 0.0);
  }

  __device__ bool start(long long idx, double &qx, double &qy, double &qz) {
    r = &L.hits[idx];
    if constexpr (MULTI) {
      fp = P::job_params(L, r->job);
      kd = P::kind(fp);
    }
    ox = r->px;
    oy = r->py;
    oz = r->pz;
    thr = D(r->thr);
    delta = r->thr * fr.smoothness;
    sub = 0;
    nx = ny = nz = D(0);
    point(qx, qy, qz);
    return true;
  }

  __device__ bool step(D d, int, double &qx, double &qy, double &qz) {
    const bool neg = (sub & 1) != 0;
    const int axis = sub >> 1;
    D &comp = (axis == 0) ? nx : ((axis == 1) ? ny : nz);
    comp = neg ? comp - d : d;
    sub++;
    if (sub < 6) {
      point(qx, qy, qz);
      return true;
    }
    // CalculateNormals tail (shader_calculate_normals.cpp:111-123)
    float fx, fy, fz;
    float s = 0.f;
    if (P::kWide) {
      double ux = double(nx), uy = double(ny), uz = double(nz);
      if (fabs(ux) < 1e-50 && fabs(uy) < 1e-50 && fabs(uz) < 1e-50) {
        ux = 1.0;
        uy = uz = 0.0;
      } else {
        const double inv = 1.0 / sqrt(ux * ux + uy * uy + uz * uz);
        ux *= inv;
        uy *= inv;
        uz *= inv;
      }
      if (!(isfinite(ux) && isfinite(uy) && isfinite(uz))) {
        ux = 1.0;
        uy = uz = 0.0;
      }
      fx = float(ux);
      fy = float(uy);
      fz = float(uz);
      if (fr.shading_enable) s = float(ux * fr.light[0] + uy * fr.light[1] + uz * fr.light[2]);
    } else {
      fx = float(nx);
      fy = float(ny);
      fz = float(nz);
      if (fabsf(fx) < 1e-30f && fabsf(fy) < 1e-30f && fabsf(fz) < 1e-30f) {
        fx = 1.f;
        fy = fz = 0.f;
      } else {
        const float inv = rsqrtf(fx * fx + fy * fy + fz * fz);
        fx *= inv;
        fy *= inv;
        fz *= inv;
      }
      if (!(isfinite(fx) && isfinite(fy) && isfinite(fz))) {
        fx = 1.f;
        fy = fz = 0.f;
      }
      if (fr.shading_enable) s = fx * float(fr.light[0]) + fy * float(fr.light[1]) + fz * float(fr.light[2]);
    }
    r->nx = fx;
    r->ny = fy;
    r->nz = fz;
    // LightShading, directional light (shader_light_shading.cpp:61-72)
    if (fr.shading_enable) {
      if (s < 0) s = 0;
      s = 1.0f - fr.material_shading + s * fr.material_shading;
      s = s * fr.light_intensity;
      if (s > 500.0f) s = 500.0f;
    }
    r->shade = s;
    return false;
  }
};

template <int FK, bool MULTI, class P>
__global__ void __launch_bounds__(256) normal_kernel(const __grid_constant__ DevFrame fr,
                                                     const __grid_constant__ typename P::Params fp0,
                                                     const __grid_constant__ Launch L, DevOutputs out) {
  if (gated_off(L)) return;
  NormalStage<MULTI, P> S{fr, L, fp0, P::kind(fp0)};
  unsigned int my_de = 0;
  unsigned long long my_iters = 0;
  const long long total = (long long)L.ctr->hits;
  run_stage<FK, P>(S, fp0, &L.ctr->normals_next, total, L.refill_k, &my_de, &my_iters);
  const int slot = L.normal_slot ? L.normal_slot : K_NORMAL;
  flush_counts(out, my_de, my_iters, slot, my_de, slot, 0);
}

// ============================================================================
// Stage S: shadow march and AO marches, (shadow_tasks + ao_rays) tasks per hit.
// ============================================================================
// PCG32 jump-ahead by `delta` steps: Brown, "Random Number Generation with
// Arbitrary Strides" (Trans. Am. Nucl. Soc. 71, 1994), as in pcg32_advance_r.
__device__ __forceinline__ unsigned long long pcg_advance(unsigned long long state, unsigned long long inc,
                                                          unsigned long long delta) {
  unsigned long long cur_mult = 6364136223846793005ull, cur_plus = inc;
  unsigned long long acc_mult = 1ull, acc_plus = 0ull;
  while (delta > 0) {
    if (delta & 1) {
      acc_mult *= cur_mult;
      acc_plus = acc_plus * cur_mult + cur_plus;
    }
    cur_plus = (cur_mult + 1ull) * cur_plus;
    cur_mult *= cur_mult;
    delta >>= 1;
  }
  return acc_mult * state + acc_plus;
}

// The secondary marches run in the policy's precision: FP32 from the FP64
// hit point rounded once (no FP64 conversions in the loop), or FP64 from the
// hit point itself.  Their hit test uses the float-rounded distThresh, as the
// reference's shaders do.
// The march length of a penetrating directional light's shadow: delta /
// resolution at the hit, i.e. |camera - p| * fov (light.cpp:277-290), with
// the camera of the hit's own job
template <bool MULTI>
__device__ __forceinline__ double shadow_distance(const DevFrame &fr, const Launch &L, const HitRec &r) {
  const double *cam = MULTI ? L.jobs[r.job].cam : fr.camera;
  const double res = MULTI ? L.jobs[r.job].resolution : fr.resolution;
  const double fov = MULTI ? L.jobs[r.job].fov : fr.fov;
  const int persp = MULTI ? L.jobs[r.job].persp : fr.persp;
  const double ax = cam[0] - r.px, ay = cam[1] - r.py, az = cam[2] - r.pz;
  double delta = sqrt(ax * ax + ay * ay + az * az) * res * fov;  // CalcDelta
  if (persp == MBR_PROJECTION_EQUIRECTANGULAR) delta *= 0.5;
  return delta / res;
}

// FAST: the AO task is the fast AO (a separate instantiation, so the march
// kernels carry none of its code).
template <bool MULTI, class P, bool FAST>
struct ShadeStage {
  typedef typename P::D Real;
  static constexpr bool kMulti = MULTI;
  typedef typename P::D D;
  const DevFrame &fr;
  const Launch &L;
  typename StageParams<MULTI, P>::type fp;
  int kd;
  HitRec *r;
  D ox, oy, oz, t;
  D dx, dy, dz, end, vdm, dfac;
  // soft shadow: the largest 1 - angle / range so far (shader_aux_shadow.cpp:142-151);
  // fast AO: the previous (clamped) distance sample
  D maxsoft;
  float thr;
  int count, mode;  // mode 0 shadow, 1 AO march, 2 fast AO (end: its float sum)
  unsigned int shadow_de;
  unsigned int trips;  // AO marches that reached max_raymarching_steps (watchdog)

  __device__ const typename P::Params &params() const { return fp; }
  __device__ int kind() const { return kd; }
  __device__ D detail() const { return D(thr); }

  __device__ void point(D &qx, D &qy, D &qz) {
    qx = fmadd(dx, t, ox);
    qy = fmadd(dy, t, oy);
    qz = fmadd(dz, t, oz);
  }

  __device__ bool start(long long idx, D &qx, D &qy, D &qz) {
    // both start records are loaded before the first is tested: the origin's
    // address depends on the task index only, so the two loads overlap
    const long long h = (long long)fdiv((unsigned long long)idx, L.div_per);
    const float4 dv = L.sdir[idx];
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!P::kWide) o = L.sorg[h];
    if (dv.w == 0.0f) return false;  // resolved by the direction kernel
    r = &L.hits[h];
    if constexpr (MULTI) {
      fp = P::job_params(L, r->job);
      kd = P::kind(fp);
    }
    if (P::kWide) {
      ox = D(r->px);
      oy = D(r->py);
      oz = D(r->pz);
      thr = float(r->thr);
      t = D(r->thr);
    } else {
      ox = D(o.x);
      oy = D(o.y);
      oz = D(o.z);
      thr = o.w;
      t = D(thr);
    }
    dx = D(dv.x);
    dy = D(dv.y);
    dz = D(dv.z);
    mode = dv.w < 0.0f ? 0 : (FAST ? 2 : 1);
    end = mode == 1 ? D(dv.w) : vdm;
    if (!mode && fr.penetrating) end = D(shadow_distance<MULTI>(fr, L, *r));
    maxsoft = D(0);
    if (FAST && mode == 2) {  // first sample at 1 * distThresh along the normal
      end = D(0);
      maxsoft = D(1e20);
    }
    count = 0;
    point(qx, qy, qz);
    return true;
  }

  __device__ bool step(D d, int, D &qx, D &qy, D &qz) {
    count++;
    if (mode == 0) {
      shadow_de++;
      const bool soft = fr.soft_range > 0.0;
      bool outside = false;  // a soft shadow ignores samples outside the limit box (shader_aux_shadow.cpp:130-147)
      if constexpr (P::kHyb) {
        const DevScene &sc = fp.sc;
        if (soft && sc.limits) {
          D qx, qy, qz;
          point(qx, qy, qz);
          outside = qx < sc.flim_min[0] || qx > sc.flim_max[0] || qy < sc.flim_min[1] || qy > sc.flim_max[1] ||
                    qz < sc.flim_min[2] || qz > sc.flim_max[2];
        }
      }
      if (soft && !outside) {
        D angle = (d - D(thr)) / t;
        if (angle < D(0)) angle = D(0);
        if (d < D(thr)) angle = D(0);
        D sft = D(1) - angle / D(fr.soft_range);
        if (fr.penetrating) sft = sft * ((end - t) / end);
        if (sft < D(0)) sft = D(0);
        if (sft > maxsoft) maxsoft = sft;
      }
      if (d < D(thr)) {
        D v = D(0);
        if (fr.penetrating) {
          v = D(1) - (end - t) / end;
          if (v < D(0)) v = D(0);
        }
        r->shadow = float(soft ? D(1) - maxsoft : v);
        return false;
      }
      if (P::kWide) t += fmax(fmin(double(d), 1e6) * double(dfac), 1e-15);
      else t += fmaxf(fminf(float(d), 1e6f) * float(dfac), 1e-15f);
      if (count > fr.max_steps || t >= end) {
        r->shadow = soft ? float(D(1) - maxsoft) : 1.f;
        return false;
      }
    } else if (FAST && mode == 2) {
      // FastAmbientOcclusion (shader_fast_ambient_occlusion.cpp:40-65): sample
      // i = count at scan t = i^2 distThresh; the sum is kept in float
      D dist = d;
      if (dist > maxsoft * D(2)) dist = maxsoft * D(2);
      maxsoft = dist;
      const D delta = P::kWide ? D(r->thr) : D(thr);
      if (P::kWide)
        end = D(float(double(end) + ldexp(1.0, -count) * (double(t) - fr.ao_fast_tune * double(dist)) / double(delta)));
      else
        end = D(float(end) + ldexpf(1.0f, -count) * (float(t) - float(fr.ao_fast_tune) * float(dist)) / float(delta));
      const int i = count + 1;
      if (i >= fr.ao_quality * fr.ao_quality) {
        float ao = 1.0f - 0.2f * float(end);
        if (ao < 0.0f) ao = 0.0f;
        r->ao_q = (unsigned long long)__float_as_uint(ao);
        return false;
      }
      t = D(i * i) * delta;
    } else {
      if (d < D(thr)) {
        if (P::kWide) {
          const double s = 1.0 - (double(end) - double(t)) / double(end);
          ao_add(r, fmax(s, 0.0));
        } else {
          const float s = 1.0f - __fdividef(float(end) - float(t), float(end));
          ao_add(r, double(fmaxf(s, 0.0f)));
        }
        return false;
      }
      t = fmadd(D(2), d, t);
      if (t >= end || count >= fr.max_steps) {
        if (!(t >= end)) trips++;  // the cap ended it: a watchdog trip
        ao_add(r, 1.0);
        return false;
      }
    }
    point(qx, qy, qz);
    return true;
  }
};

// Stage D: the start records of stage S, one thread per task.  AO direction
// k of a hit: draws 2k, 2k+1 of PCG32(state ao_seed, stream pixel) mapped to
// a cosine-weighted direction about the normal; task 0 (when the shadow
// march runs) points at the light, or is resolved here when the surface faces
// away (LightShading, shade <= 0.001) or no room is left to march.
template <bool MULTI>
__global__ void __launch_bounds__(256) direction_kernel(const __grid_constant__ DevFrame fr,
                                                        const __grid_constant__ Launch L) {
  if (gated_off(L)) return;
  const long long nh = (long long)L.ctr->hits;
  const int per = L.shadow_tasks + L.ao_rays;
  const long long n = nh * per;
  const float vdm = float(fr.view_distance_max);
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long h = (long long)fdiv((unsigned long long)idx, L.div_per);
    const int k = int(idx - h * per);
    HitRec &r = L.hits[h];
    const float thr = float(r.thr);
    if (k == 0) L.sorg[h] = make_float4(float(r.px), float(r.py), float(r.pz), thr);
    float4 dv;
    if (k < L.shadow_tasks) {
      if (!(r.shade > 0.001f)) {
        r.shadow = 0.f;
        dv = make_float4(0.f, 0.f, 0.f, 0.f);
      } else if (!(thr < (fr.penetrating ? float(shadow_distance<MULTI>(fr, L, r)) : vdm))) {
        r.shadow = 1.f;
        dv = make_float4(0.f, 0.f, 0.f, 0.f);
      } else {
        dv = make_float4(float(fr.light[0]), float(fr.light[1]), float(fr.light[2]), -1.0f);
      }
    } else if (L.ao_fast) {
      dv = make_float4(r.nx, r.ny, r.nz, 1.0f);  // fast AO: samples along the normal
    } else {
      const int a = k - L.shadow_tasks;
      Pcg32 g = pcg_init(fr.ao_seed, (unsigned long long)r.ray);
      g.state = pcg_advance(g.state, g.inc, 2ull * (unsigned long long)a);
      const float u1 = float(g.uniform()), u2 = float(g.uniform());
      const float nx = r.nx, ny = r.ny, nz = r.nz;
      const float rr = sqrtf(u1);
      float sp, cp;
      __sincosf(6.28318530717958647692f * u2, &sp, &cp);
      const float lx = rr * cp, ly = rr * sp, lz = sqrtf(fmaxf(0.0f, 1.0f - u1));
      const float sg = nz >= 0.0f ? 1.0f : -1.0f;
      const float aa = -1.0f / (sg + nz);
      const float b = nx * ny * aa;
      const float end = float(r.depth) * (MULTI ? L.jobs[r.job].fovf : float(fr.fov));
      if (!(thr < end)) {
        ao_add(&r, 1.0);  // no room to march: unoccluded
        dv = make_float4(0.f, 0.f, 0.f, 0.f);
      } else {
        dv = make_float4(fmaf(1.0f + sg * nx * nx * aa, lx, fmaf(b, ly, nx * lz)),
                         fmaf(sg * b, lx, fmaf(sg + ny * ny * aa, ly, ny * lz)),
                         fmaf(-sg * nx, lx, fmaf(-ny, ly, nz * lz)), end);
      }
    }
    L.sdir[idx] = dv;
  }
}

template <int FK, bool MULTI, class P, bool FAST>
__device__ __forceinline__ void shade_body(const DevFrame &fr, const typename P::Params &fp0, const Launch &L,
                                           DevOutputs &out) {
  if (gated_off(L)) return;
  ShadeStage<MULTI, P, FAST> S{fr, L, fp0, P::kind(fp0)};
  S.shadow_de = 0;
  S.trips = 0;
  S.vdm = typename P::D(fr.view_distance_max);
  S.dfac = typename P::D(fr.de_factor);
  unsigned int my_de = 0;
  unsigned long long my_iters = 0;
  const long long total = (long long)L.ctr->hits * (long long)(L.shadow_tasks + L.ao_rays);
  run_stage<FK, P>(S, fp0, &L.ctr->shade_next, total, L.refill_k, &my_de, &my_iters);
  flush_counts(out, my_de, my_iters, K_AO, my_de - S.shadow_de, K_SHADOW, S.shadow_de);
  const unsigned int trips = __reduce_add_sync(0xffffffffu, S.trips);
  if ((threadIdx.x & 31) == 0 && trips) {
    if (out.stats) atomicAdd(reinterpret_cast<unsigned long long *>(out.stats) + K_WATCHDOG, (unsigned long long)trips);
    if (out.status) atomicOr(out.status, int(STATUS_AO_MARCH_CAP));
  }
}

template <int FK, bool MULTI, class P>
__global__ void __launch_bounds__(256, kMinBlocks<FK, MULTI, P>::shade) shade_kernel(const __grid_constant__ DevFrame fr,
                                                    const __grid_constant__ typename P::Params fp0,
                                                    const __grid_constant__ Launch L, DevOutputs out) {
  shade_body<FK, MULTI, P, false>(fr, fp0, L, out);
}

// Stage S when the AO is the fast AO.
template <int FK, bool MULTI, class P>
__global__ void __launch_bounds__(256) shade_fast_kernel(const __grid_constant__ DevFrame fr,
                                                         const __grid_constant__ typename P::Params fp0,
                                                         const __grid_constant__ Launch L, DevOutputs out) {
  shade_body<FK, MULTI, P, true>(fr, fp0, L, out);
}

// ============================================================================
// Stage F: colour and outputs of every hit.
// ============================================================================
static __global__ void __launch_bounds__(256) finish_kernel(const __grid_constant__ DevFrame fr,
                                                     const __grid_constant__ Launch L, DevOutputs out) {
  if (gated_off(L)) return;
  const long long nh = (long long)L.ctr->hits;
  for (long long h = (long long)blockIdx.x * blockDim.x + threadIdx.x; h < nh; h += (long long)gridDim.x * blockDim.x) {
    const HitRec &r = L.hits[h];
    const long long pix = r.pix;
    const float shade = r.shade * r.shadow;
    const float ao = L.ao_fast        ? __uint_as_float((unsigned int)r.ao_q)
                     : (L.ao_rays > 0) ? float(double(r.ao_q) * (1.0 / 4294967296.0) / double(L.ao_rays))
                                       : 1.0f;
    const float col = fr.albedo * (shade + fr.ambient * ao);
    float rgb[3] = {col, col, col};
    if (out.depth) out.depth[pix] = r.depth;
    if (out.iters) out.iters[pix] = r.iters;
    if (out.hit) out.hit[pix] = 1;
    const bool nrm = fr.shading_enable || L.ao_rays > 0 || L.want_normal;
    if (out.normal) {
      out.normal[3 * pix + 0] = nrm ? r.nx : 0.f;
      out.normal[3 * pix + 1] = nrm ? r.ny : 0.f;
      out.normal[3 * pix + 2] = nrm ? r.nz : 0.f;
    }
    if (out.shade) out.shade[pix] = shade;
    if (out.ao) out.ao[pix] = ao;
    if (out.rgb) {
      out.rgb[3 * pix + 0] = rgb[0];
      out.rgb[3 * pix + 1] = rgb[1];
      out.rgb[3 * pix + 2] = rgb[2];
    }
    if (out.rgb8) to_rgb8(fr, rgb, &out.rgb8[3 * pix]);
  }
}

// Counts pixels (misses + hits) once per launch, from the stage-P queue size.
static __global__ void pixel_count_kernel(const __grid_constant__ Launch L, DevOutputs out, long long pixels) {
  if (gated_off(L)) return;
  if (threadIdx.x == 0 && out.stats) atomicAdd(reinterpret_cast<unsigned long long *>(out.stats) + K_PIXELS,
                                               (unsigned long long)pixels);
}

// ============================================================================
// GI frames (single-frame launches).  Monte Carlo paths of GlobalIlumination
// (src/shader_global_illumination.cpp:41-209) with MonteCarloDOF
// (src/render_worker.cpp:1832-1862), as the plain kernel's gi_path restates
// them, split into stages like the frame pipeline:
//   stage GP  one task per path (pixel, sample), pixel-major: the jittered
//             thin-lens primary ray, the reference march and binary search;
//             a hit appends the path's first vertex to the level-0 list
//   per level b = 0 .. bounces:
//     stage N   the six normal samples of every vertex of level b
//     stage GV  per vertex: the hard sun-shadow march when the surface faces
//               the sun, its radiance term, then (b < bounces) the cosine
//               bounce marched with the GI step rule; a hit appends the next
//               vertex to the level-b+1 list, a miss adds the sky
//   stage GF  per pixel: the path radiances summed in sample order.
// Random numbers come from the same PCG32 stream per (pixel, sample) and the
// same Park-Miller jitter stream as the plain kernel's: the bounce of level b
// takes draws 4 + 2b and 5 + 2b, reached by jump-ahead.  A path's radiance
// terms are added in the plain kernel's order by one thread at a time.
// ============================================================================
enum { G_MARCH = 0, G_BINARY, G_SHADOW, G_BOUNCE };

// distThresh at q (render_worker.cpp:653-679), from the camera position
__device__ __forceinline__ double gi_thresh(const DevFrame &fr, double qx, double qy, double qz) {
  if (fr.constant_de_threshold) return thresh_tail(fr, fr.persp, fr.de_thresh);
  const double ax = fr.camera[0] - qx, ay = fr.camera[1] - qy, az = fr.camera[2] - qz;
  return thresh_tail(fr, fr.persp, sqrt(ax * ax + ay * ay + az * az) * fr.resolution * fr.fov / fr.detail_level);
}

template <class P>
struct GIPrimaryStage {
  typedef double Real;
  typedef typename P::D D;
  static constexpr bool kMulti = false;
  const DevFrame &fr;
  const Launch &L;
  const DevOutputs &out;
  const WJob *jb;
  typename StageParams<false, P>::type fp;
  int kd;
  unsigned long long ray;  // RNG stream id: frame pixel * samples + sample
  long long pix;           // output index of the pixel
  long long path;          // path of the launch: pixel of the launch * samples + sample
  int sample, phase, sub, count, last_iters;
  unsigned int pm;
  double ox, oy, oz, dx, dy, dz, t, stp, dir_len, thr;
  double lx, ly, lz;  // previous request point (dead-ray check)
  D dist_prev, search_limit;
  unsigned int n_march, n_binary;

  __device__ const typename P::Params &params() const { return fp; }
  __device__ int kind() const { return kd; }
  __device__ D detail() const { return D(thr); }
  __device__ void ray_point(double &qx, double &qy, double &qz) const {
    qx = ox + dx * t;
    qy = oy + dy * t;
    qz = oz + dz * t;
  }

  __device__ bool start(long long idx, double &qx, double &qy, double &qz) {
    const unsigned long long spp = (unsigned long long)fr.gi_samples;
    path = idx;
    const unsigned long long lpix = fdiv((unsigned long long)idx, L.div_spp);
    sample = int((unsigned long long)idx - lpix * spp);
    const unsigned long long yy = fdiv(lpix, jb->div_w);
    const int x = int(lpix - yy * (unsigned long long)jb->width);
    const int y = int(yy) + jb->row0;
    const unsigned long long pixel = (unsigned long long)y * (unsigned long long)jb->width + (unsigned long long)x;
    pix = jb->pixel_offset + (long long)pixel;
    ray = pixel * spp + (unsigned long long)sample;
    Pcg32 rng = pcg_init(fr.gi_seed, ray);
    const double ujx = rng.uniform(), ujy = rng.uniform(), ulr = rng.uniform(), ula = rng.uniform();
    double ix, iy;
    image_point(fr, double(x), double(y), &ix, &iy);
    if (hemisphere_cut(fr.persp, fr.fov, ix, iy)) {  // not traced: black, no hit
      last_iters = 0;
      if (sample == 0) {
        if (out.depth) out.depth[pix] = 1e20;
        if (out.iters) out.iters[pix] = 0;
        if (out.hit) out.hit[pix] = 0;
      }
      L.path_rad[path] = 0.0;
      return false;
    }
    ix = ix + (ujx - 0.5) / double(fr.width) * fr.aspect;
    iy = iy + (ujy - 0.5) / double(fr.height);
    D3 view = view_vector(fr, ix, iy);
    const D3 cam = camera_of(fr);
    D3 st = cam;
    if (fr.dof_aperture > 0.0) {
      const double randR = fr.dof_aperture * sqrt(ulr);
      const double randAngle = 2.0 * 3.14159265358979323846 * ula;
      double sa, ca;
      sincos(randAngle, &sa, &ca);
      const D3 rv = rotate(fr, D3{randR * sa, 0.0, randR * ca});
      view = d3sub(view, d3mul(rv, 1.0 / fr.dof_focus));
      st = d3add(cam, rv);
    }
    const D3 dir = d3norm(view);
    ox = st.x;
    oy = st.y;
    oz = st.z;
    dx = dir.x;
    dy = dir.y;
    dz = dir.z;
    dir_len = d3len(dir);
    pm = pm_for_ray(ray, fr.seed).s;
    phase = G_MARCH;
    t = 0.0;
    stp = 0.0;
    count = 0;
    sub = 0;
    last_iters = 0;
    thr = 0.0;
    ray_point(qx, qy, qz);
    if (!(isfinite(qx) && isfinite(qy) && isfinite(qz))) {  // stuck at once (render_worker.cpp:747-756)
      hit();
      return false;
    }
    lx = qx;
    ly = qy;
    lz = qz;
    thr = gi_thresh(fr, qx, qy, qz);
    return true;
  }

  __device__ bool miss() {
    if (sample == 0) {
      if (out.depth) out.depth[pix] = 1e20;
      if (out.iters) out.iters[pix] = last_iters;
      if (out.hit) out.hit[pix] = 0;
    }
    L.path_rad[path] = fr.gi_sky;
    return false;
  }

  // the primary ray found the surface at t: the path's first vertex
  __device__ bool hit() {
    if (sample == 0) {
      if (out.depth) out.depth[pix] = t;
      if (out.iters) out.iters[pix] = last_iters;
      if (out.hit) out.hit[pix] = 1;
    }
    L.path_rad[path] = 0.0;
    const unsigned long long h = atomicAdd(&L.ctr->hits, 1ull);
    HitRec &r = L.hits[h];
    ray_point(r.px, r.py, r.pz);
    r.depth = t;
    r.thr = thr;
    r.pix = path;
    r.iters = last_iters;
    r.nx = 1.f;
    r.ny = r.nz = 0.f;
    r.job = 0;
    return false;
  }

  // reference binary search step (render_worker.cpp:854-912)
  __device__ bool binary_check(double &qx, double &qy, double &qz) {
    if (sub >= fr.binary_steps || (double(dist_prev) < thr && double(dist_prev) > thr * double(search_limit)))
      return hit();
    if (double(dist_prev) > thr) t += stp;
    else if (double(dist_prev) < thr * double(search_limit)) t -= stp;
    ray_point(qx, qy, qz);
    thr = gi_thresh(fr, qx, qy, qz);
    return true;
  }

  __device__ bool step(D d, int iters, double &qx, double &qy, double &qz) {
    last_iters = iters;
    if (phase == G_BINARY) {
      n_binary++;
      dist_prev = d;
      stp *= 0.5;
      sub++;
      return binary_check(qx, qy, qz);
    }
    n_march++;
    count++;
    if (double(d) < thr) {
      stp *= 0.5;
      sub = 0;
      dist_prev = d;
      phase = G_BINARY;
      return binary_check(qx, qy, qz);
    }
    double jit = 1.0;
    if (fr.jitter) {
      ParkMiller p;
      p.s = pm;
      jit = 1.0 - tenthousandths(p.random(1000));
      pm = p.s;
    }
    stp = (double(d) - 0.5 * thr) * fr.de_factor * jit;
    stp = step_limit(fr, stp, thr);
    t += stp / dir_len;
    if (t > fr.view_distance_max || count >= fr.max_steps) return miss();
    ray_point(qx, qy, qz);
    if ((qx == lx && qy == ly && qz == lz) || !(isfinite(qx) && isfinite(qy) && isfinite(qz))) return hit();
    lx = qx;
    ly = qy;
    lz = qz;
    thr = gi_thresh(fr, qx, qy, qz);
    return true;
  }
};

template <class P>
struct GIVertexStage {
  typedef double Real;
  typedef typename P::D D;
  static constexpr bool kMulti = false;
  const DevFrame &fr;
  const Launch &L;
  typename StageParams<false, P>::type fp;
  int kd;
  long long path;
  int phase, count;
  double tp, vx, vy, vz, vthr, nx, ny, nz, ndl;
  double ox, oy, oz, dx, dy, dz, t, thr;
  unsigned int n_gi;

  __device__ const typename P::Params &params() const { return fp; }
  __device__ int kind() const { return kd; }
  __device__ D detail() const { return D(thr); }
  __device__ void ray_point(double &qx, double &qy, double &qz) const {
    qx = ox + dx * t;
    qy = oy + dy * t;
    qz = oz + dz * t;
  }

  __device__ bool start(long long idx, double &qx, double &qy, double &qz) {
    const HitRec &r = L.hits[idx];
    path = r.pix;
    vx = r.px;
    vy = r.py;
    vz = r.pz;
    vthr = r.thr;
    nx = double(r.nx);
    ny = double(r.ny);
    nz = double(r.nz);
    ndl = nx * fr.light[0] + ny * fr.light[1] + nz * fr.light[2];
    tp = 1.0;
    for (int b = 0; b < L.level; b++) tp *= double(fr.albedo);
    if (!(ndl > 0.0)) return after_shadow(0.0, qx, qy, qz);
    // hard AuxShadow toward the sun from the vertex (shader_aux_shadow.cpp:94-321)
    phase = G_SHADOW;
    t = vthr;
    count = 0;
    thr = vthr;
    if (!(t < fr.view_distance_max)) return after_shadow(1.0, qx, qy, qz);
    ox = vx;
    oy = vy;
    oz = vz;
    dx = fr.light[0];
    dy = fr.light[1];
    dz = fr.light[2];
    ray_point(qx, qy, qz);
    return true;
  }

  __device__ bool after_shadow(double sh, double &qx, double &qy, double &qz) {
    if (ndl > 0.0) L.path_rad[path] += tp * double(fr.albedo) * fr.gi_sun * ndl * sh;
    if (L.level >= fr.gi_bounces) return false;
    tp *= double(fr.albedo);
    // the bounce's two draws of the path's stream
    const unsigned long long spp = (unsigned long long)fr.gi_samples;
    const unsigned long long lpix = fdiv((unsigned long long)path, L.div_spp);
    const unsigned long long sample = (unsigned long long)path - lpix * spp;
    const unsigned long long ray = ((unsigned long long)L.row0 * (unsigned long long)fr.width + lpix) * spp + sample;
    Pcg32 rng = pcg_init(fr.gi_seed, ray);
    rng.state = pcg_advance(rng.state, rng.inc, 4ull + 2ull * (unsigned long long)L.level);
    const double u1 = rng.uniform(), u2 = rng.uniform();
    const D3 d = cosine_dir(D3{nx, ny, nz}, u1, u2);
    dx = d.x;
    dy = d.y;
    dz = d.z;
    ox = vx;
    oy = vy;
    oz = vz;
    phase = G_BOUNCE;
    t = vthr;
    count = 0;
    if (!(t < fr.view_distance_max) || count >= fr.max_steps) {
      L.path_rad[path] += tp * fr.gi_sky;
      return false;
    }
    ray_point(qx, qy, qz);
    thr = gi_thresh(fr, qx, qy, qz);
    return true;
  }

  __device__ bool step(D d, int, double &qx, double &qy, double &qz) {
    n_gi++;
    if (phase == G_SHADOW) {
      if (double(d) < double(float(vthr))) return after_shadow(0.0, qx, qy, qz);
      const double s = fmax(fmin(double(d), 1000000.0) * fr.de_factor, 1e-15);
      count++;
      if (count > fr.max_steps) return after_shadow(1.0, qx, qy, qz);
      t += s;
      if (!(t < fr.view_distance_max)) return after_shadow(1.0, qx, qy, qz);
      ray_point(qx, qy, qz);
      return true;
    }
    // G_BOUNCE: the GI march rule (shader_global_illumination.cpp:75-125)
    if (double(d) < thr) {
      if (t < thr * 2.0) return false;  // the bounce hit its own vertex
      const unsigned long long h = atomicAdd(L.next_hits, 1ull);
      HitRec &r = L.hits_next[h];
      ray_point(r.px, r.py, r.pz);
      r.depth = t;
      r.thr = thr;
      r.pix = path;
      r.iters = 0;
      r.nx = 1.f;
      r.ny = r.nz = 0.f;
      r.job = 0;
      return false;
    }
    count++;
    t += double(d) * fr.de_factor;
    if (!(t < fr.view_distance_max) || count >= fr.max_steps) {
      L.path_rad[path] += tp * fr.gi_sky;
      return false;
    }
    ray_point(qx, qy, qz);
    thr = gi_thresh(fr, qx, qy, qz);
    return true;
  }
};

template <int FK, class P>
__global__ void __launch_bounds__(256, kMinBlocks<FK, false, P>::gi) gi_primary_kernel(const __grid_constant__ DevFrame fr,
                                                         const __grid_constant__ typename P::Params fp0,
                                                         const __grid_constant__ WJob job0,
                                                         const __grid_constant__ Launch L, DevOutputs out) {
  if (gated_off(L)) return;
  GIPrimaryStage<P> S{fr, L, out, &job0, fp0, P::kind(fp0)};
  S.search_limit = typename P::D(1.0 - 0.001 * fr.detail_level);
  S.n_march = S.n_binary = 0;
  unsigned int my_de = 0;
  unsigned long long my_iters = 0;
  run_stage<FK, P>(S, fp0, &L.ctr->pixels_next, L.total, L.refill_k, &my_de, &my_iters);
  flush_counts(out, my_de, my_iters, K_MARCH, S.n_march, K_BINARY, S.n_binary);
}

// At most 64 registers (4 blocks of 256 per SM): the stage is latency-bound,
// and twice the resident warps outweigh its few spills (the 4K x 16 spp
// hybrid GI frame: 1.28 -> 1.18 s; at 80 registers 1.21 s).
template <int FK, class P>
__global__ void __launch_bounds__(256, 4) gi_vertex_kernel(const __grid_constant__ DevFrame fr,
                                                           const __grid_constant__ typename P::Params fp0,
                                                           const __grid_constant__ Launch L, DevOutputs out) {
  if (gated_off(L)) return;
  GIVertexStage<P> S{fr, L, fp0, P::kind(fp0)};
  S.n_gi = 0;
  unsigned int my_de = 0;
  unsigned long long my_iters = 0;
  const long long total = (long long)L.ctr->hits;
  run_stage<FK, P>(S, fp0, &L.ctr->shade_next, total, L.refill_k, &my_de, &my_iters);
  flush_counts(out, my_de, my_iters, K_GI, S.n_gi, K_GI, 0);
}

// Stage GF: the mean radiance of every pixel (its paths summed in sample
// order, as the plain kernel sums them), its colour and the outputs the plain
// kernel writes for GI (normal 0, shade 0, AO 1).
static __global__ void __launch_bounds__(256) gi_finish_kernel(const __grid_constant__ DevFrame fr,
                                                        const __grid_constant__ WJob job0,
                                                        const __grid_constant__ Launch L, DevOutputs out,
                                                        long long pixels) {
  if (gated_off(L)) return;
  const int spp = fr.gi_samples;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < pixels;
       p += (long long)gridDim.x * blockDim.x) {
    const long long pix = job0.pixel_offset + (long long)job0.row0 * job0.width + p;
    double acc = 0.0;
    for (int s = 0; s < spp; s++) acc += L.path_rad[p * spp + s];
    const float v = float(acc / double(spp));
    float rgb[3] = {v, v, v};
    if (out.normal) {
      out.normal[3 * pix + 0] = 0.f;
      out.normal[3 * pix + 1] = 0.f;
      out.normal[3 * pix + 2] = 0.f;
    }
    if (out.shade) out.shade[pix] = 0.f;
    if (out.ao) out.ao[pix] = 1.0f;
    if (out.rgb) {
      out.rgb[3 * pix + 0] = v;
      out.rgb[3 * pix + 1] = v;
      out.rgb[3 * pix + 2] = v;
    }
    if (out.rgb8) to_rgb8(fr, rgb, &out.rgb8[3 * pix]);
  }
}

// The instantiated pipelines (fk: the formula kind).
int pipeline_fp32(int fk, const mbr_tuning &tu, cudaStream_t st, const DevFrame &fr, const FastParams &fp, const WJob &j0,
                  const Launch &L, const DevOutputs &out, long long pixels);
int pipeline_fp64(int fk, const mbr_tuning &tu, cudaStream_t st, const DevFrame &fr, const WideParams &fp, const WJob &j0,
                  const Launch &L, const DevOutputs &out, long long pixels);
int pipeline_batch_fp32(int fk, const mbr_tuning &tu, cudaStream_t st, const DevFrame &fr, const FastParams &fp,
                        const WJob &j0, const Launch &L, const DevOutputs &out, long long pixels);
int pipeline_batch_fp64(int fk, const mbr_tuning &tu, cudaStream_t st, const DevFrame &fr, const WideParams &fp,
                        const WJob &j0, const Launch &L, const DevOutputs &out, long long pixels,
                        cudaEvent_t before_shade);
int pipeline_hybrid(const DevScene &sc, const mbr_tuning &tu, cudaStream_t st, const DevFrame &fr, const WJob &j0,
                    const Launch &L, const DevOutputs &out, long long pixels);

// ---- host side -------------------------------------------------------------------
static int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// The FP32 Mandelbox's stage P runs unbounded below the first number of pixels
// and at 64 registers from the second (see kMinBlocks).
const long long kFewPixels = 131072, kManyPixels = 1572864;

// The stage launches of one frame or batch under policy P, in stream order.
template <bool MULTI, class P>
static int launch_pipeline(int fk, const mbr_tuning &tu, cudaStream_t st, const DevFrame &fr,
                           const typename P::Params &fp0, const WJob &j0, const Launch &L0, const DevOutputs &out,
                           long long pixels, cudaEvent_t before_shade = nullptr) {
  Launch L = L0;
  L.div_per = make_fastdiv(std::max(1, L.shadow_tasks + L.ao_rays));
  L.gate_value = P::kWide;
  const int sms = sm_count();
  const int grid = std::max(1, sms * tu.ctas_per_sm);
  const int block = tu.block_size;
  if (P::kHyb) fk = FK_ANY;
  int e = int(cudaMemsetAsync(L.ctr, 0, sizeof(Counters4), st));
  if (e) return e;
  if constexpr (!MULTI && P::kGI) {
    if (fr.gi_samples > 0) {  // GI frame: stage GP, then per level stages N and GV, then GF
      L.div_spp = make_fastdiv(fr.gi_samples);
      L.row0 = fr.row0;
      Counters4 *ctrs = L.ctr;
      HitRec *lists[2] = {L.hits, L.hits_next};
      e = int(cudaMemsetAsync(ctrs, 0, sizeof(Counters4) * size_t(fr.gi_bounces + 2), st));
      if (e) return e;
#define GI_CASES(LAUNCH)         \
  switch (fk) {                  \
    LAUNCH(FK_BOX_SIMPLE)        \
    LAUNCH(FK_BOX)               \
    LAUNCH(FK_BULB)              \
    LAUNCH(FK_MENGER)            \
    LAUNCH(FK_ANY)               \
    default: return int(cudaErrorInvalidValue); \
  }
      {
        Launch Lp = L;
        Lp.ctr = &ctrs[0];
        Lp.hits = lists[0];
#define GP_LAUNCH(K) \
  case K:            \
    if constexpr (P::kHyb == (K == FK_ANY)) gi_primary_kernel<K, P><<<grid, block, 0, st>>>(fr, fp0, j0, Lp, out); \
    break;
        GI_CASES(GP_LAUNCH)
#undef GP_LAUNCH
        count_launches(1);
      }
      for (int b = 0; b <= fr.gi_bounces; b++) {
        Launch Lb = L;
        Lb.ctr = &ctrs[b];
        Lb.hits = lists[b & 1];
        Lb.hits_next = lists[(b + 1) & 1];
        Lb.next_hits = &ctrs[b + 1].hits;
        Lb.level = b;
        Lb.normal_slot = K_GI;
#define GV_LAUNCH(K)                                                                                   \
  case K:                                                                                              \
    if constexpr (P::kHyb == (K == FK_ANY)) {                                                           \
      normal_kernel<K, false, typename P::Normal><<<grid, block, 0, st>>>(fr, fp0, Lb, out);                             \
      gi_vertex_kernel<K, P><<<grid, block, 0, st>>>(fr, fp0, Lb, out);                                 \
    }                                                                                                  \
    break;
        GI_CASES(GV_LAUNCH)
#undef GV_LAUNCH
        count_launches(2);
      }
#undef GI_CASES
      gi_finish_kernel<<<sms * 4, 256, 0, st>>>(fr, j0, L, out, pixels);
      pixel_count_kernel<<<1, 32, 0, st>>>(L, out, pixels);
      count_launches(2);
      return int(cudaGetLastError());
    }
  }
#define STAGE_LAUNCH(PP, KERNEL, K, ...)                                                \
  case K:                                                                               \
    if constexpr (P::kHyb == (K == FK_ANY)) KERNEL<K, MULTI, PP><<<grid, block, 0, st>>>(__VA_ARGS__); \
    break;
#define STAGE(KERNEL, ...) STAGEP(P, KERNEL, __VA_ARGS__)
#define STAGEP(PP, KERNEL, ...)                                                         \
  switch (fk) {                                                                         \
    STAGE_LAUNCH(PP, KERNEL, FK_BOX_SIMPLE, __VA_ARGS__)                                \
    STAGE_LAUNCH(PP, KERNEL, FK_BOX, __VA_ARGS__)                                       \
    STAGE_LAUNCH(PP, KERNEL, FK_BULB, __VA_ARGS__)                                      \
    STAGE_LAUNCH(PP, KERNEL, FK_MENGER, __VA_ARGS__)                                    \
    STAGE_LAUNCH(PP, KERNEL, FK_ANY, __VA_ARGS__)                                       \
    default: return int(cudaErrorInvalidValue);                                         \
  }
  bool primary = false;
  if constexpr (kMinBlocks<FK_BOX_SIMPLE, MULTI, P>::box32) {
    primary = fk == FK_BOX_SIMPLE && (L.total < kFewPixels || L.total >= kManyPixels);
    if (primary && L.total < kFewPixels)
      primary_kernel<FK_BOX_SIMPLE, MULTI, P, 0><<<grid, block, 0, st>>>(fr, fp0, j0, L, out);
    else if (primary)
      primary_kernel<FK_BOX_SIMPLE, MULTI, P, 4><<<grid, block, 0, st>>>(fr, fp0, j0, L, out);
  }
  if (!primary) { STAGE(primary_kernel, fr, fp0, j0, L, out) }
  const bool need_normal = fr.shading_enable || L.ao_rays > 0 || L.want_normal;
  if (need_normal) { typedef typename P::Normal PN; STAGEP(PN, normal_kernel, fr, fp0, L, out) }
  const bool marches = L.ao_rays > 0 || L.shadow_tasks > 0;
  if (marches) direction_kernel<MULTI><<<sms * 8, 256, 0, st>>>(fr, L);
  if (before_shade) {
    e = int(cudaEventRecord(before_shade, st));
    if (e) return e;
  }
  if (marches) {
    if constexpr (P::kFastAO) {
      if (L.ao_fast) { STAGE(shade_fast_kernel, fr, fp0, L, out) }
    }
    if (!L.ao_fast) { STAGE(shade_kernel, fr, fp0, L, out) }
  }
#undef STAGE
#undef STAGEP
#undef STAGE_LAUNCH
  finish_kernel<<<sms * 4, 256, 0, st>>>(fr, L, out);
  pixel_count_kernel<<<1, 32, 0, st>>>(L, out, pixels);
  count_launches(3 + (need_normal ? 1 : 0) + (marches ? 2 : 0));
  return int(cudaGetLastError());
}

}  // namespace mbr
