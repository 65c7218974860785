// wavefront.cu - the wavefront engines' entry points: frames, batches, the
// precision policy, the autotuner and allocation-free rendering.  The kernels
// are in wavefront.cuh.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "wavefront.cuh"

namespace mbr {

// Views whose smallest hit threshold is below this many FP32 units (2^-24)
// of the camera coordinates iterate in FP64 under MBR_ENGINE_WAVEFRONT_AUTO.
// The FP32 depth error grows about as 0.01 / (threshold in FP32 units); 256
// keeps it near 1e-4 relative at the 99th percentile.
const double kWideRatio = 256.0;

// ============================================================================
// Precision policy
// ============================================================================
// 1 when the smallest hit threshold of a view, bounded below by
// DE(camera) * c0 (c0: threshold per unit distance), or the constant
// threshold, is below kWideRatio FP32 units of the camera coordinates.  The
// bound passes through the threshold's tail (equirectangular halving,
// advanced-quality clamps) as every threshold of the view does.
__device__ __forceinline__ int wide_needed(const DevScene &sc, const DevFrame &fr, const double cam[3], double c0,
                                           int persp) {
  double thr_min = fr.de_thresh;
  if (!fr.constant_de_threshold) {
    int it;
    const double d0 = calc_distance<double, F_EXT, false>(sc, cam[0], cam[1], cam[2], 0.0, false, &it);
    thr_min = d0 * c0;
  }
  thr_min = thresh_tail(fr, persp, thr_min);
  const double scale = fmax(fmax(fabs(cam[0]), fabs(cam[1])), fmax(fabs(cam[2]), 1.0));
  return (thr_min < kWideRatio * scale * 0x1p-24) ? 1 : 0;
}

__global__ void policy_kernel(const __grid_constant__ DevScene sc, const __grid_constant__ DevFrame fr, int *gate) {
  if (blockIdx.x == 0 && threadIdx.x == 0)
    *gate = wide_needed(sc, fr, fr.camera, fr.resolution * fr.fov / fr.detail_level, fr.persp);
}

__global__ void batch_policy_kernel(const DevScene *scenes, const int *scene_of, const WJob *jobs, int n,
                                    const __grid_constant__ DevFrame fr, int *flags) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n)
    flags[i] = wide_needed(scenes[scene_of[i]], fr, jobs[i].cam, jobs[i].resolution * jobs[i].fov / jobs[i].detail,
                           jobs[i].persp);
}

static WJob make_job(const DevFrame &fr, long long first, long long pixel_offset) {
  WJob j;
  std::memset(&j, 0, sizeof(j));
  for (int i = 0; i < 3; i++) j.cam[i] = fr.camera[i];
  for (int i = 0; i < 9; i++) j.mrot[i] = fr.mrot[i];
  j.mrot_zero = fr.mrot_zero;
  j.width = fr.width;
  j.height = fr.height;
  j.tiles_x = (fr.width + 7) / 8;
  j.row0 = fr.row0;
  j.rows = fr.row1 - fr.row0;
  j.first = first;
  j.pixel_offset = pixel_offset;
  j.fov = fr.fov;
  j.persp = fr.persp;
  j.legacy_y = fr.legacy_y;
  j.aspect = fr.aspect;
  j.resolution = fr.resolution;
  j.detail = fr.detail_level;
  // CalcDistThresh and CalcDelta halve both for an equirectangular view (render_worker.cpp:669, 688)
  const double half = fr.persp == MBR_PROJECTION_EQUIRECTANGULAR ? 0.5 : 1.0;
  j.c0 = float(fr.resolution * fr.fov / fr.detail_level * half);
  j.fovf = float(fr.fov * half);
  j.cthr = float(fr.de_thresh * half);
  j.div_w = make_fastdiv(j.width);
  j.div_tx = make_fastdiv(j.tiles_x);
  return j;
}

static long long job_items(const WJob &j, int layout) {
  if (layout == 1) return (long long)j.tiles_x * ((j.rows + 3) / 4) * 32;
  return (long long)j.width * j.rows;
}

static mbr_status check_supported(mbr_ctx *ctx, const DevScene &sc, const DevFrame &fr, bool batch) {
  if (batch && (sc.is_hybrid || sc.generic || fr.gi_samples > 0))
    return set_err(ctx, MBR_EUNSUPPORTED,
                   "wavefront batches: hybrid sequences, formulas without a specialised form and GI render one frame "
                   "at a time");
  if (sc.iter_thresh || sc.interior || sc.has_w)
    return set_err(ctx, MBR_EUNSUPPORTED,
                   "wavefront engine: iteration_threshold_mode, interior_mode and initial_waxis != 0 use the plain engines");
  if (sc.delta_de)
    return set_err(ctx, MBR_EUNSUPPORTED,
                   "wavefront engine: the delta DE offsets points by 1e-5 of the detail size, which FP32 points do "
                   "not resolve; it runs on the plain FP64 engines");
  if (fr.refine != MBR_REFINE_REFERENCE)
    return set_err(ctx, MBR_EUNSUPPORTED, "wavefront engine: root refinement uses the plain engines");
  if (sc.n_nodes > 0)
    return set_err(ctx, MBR_EUNSUPPORTED, "wavefront engine: explicit objects trees use the plain engines");
  for (int k = 0; k < MBR_MAX_FRACTALS; k++)
    if (sc.slot[k].add_bail || keyed_formula_has_state(sc.slot[k].formula))
      return set_err(ctx, MBR_EUNSUPPORTED,
                     "wavefront engine: formulas with a convergence bailout or orbit state (pseudo-Kleinian, "
                     "Abox mod 11, box fold bulb pow 2 V2) use the plain engines");
  if (fr.slow_shading)
    return set_err(ctx, MBR_EUNSUPPORTED, "wavefront engine: slow shading (iteration-count normals) uses the plain "
                                          "engines");
  return MBR_OK;
}

// Scratch of a launch over `pixels` work items with `per` stage-S tasks per
// hit: counters and the policy flag (256 B), hit records, FP32 origins and
// stage-S start records.  A HitRec is 88 bytes, so the hit region is rounded
// up to a multiple of 256 bytes: the float4 records after it then start on a
// 16-byte boundary for every pixel count, odd ones included.
static size_t hit_region_bytes(long long pixels) { return (size_t(pixels) * sizeof(HitRec) + 255) / 256 * 256; }

static size_t scratch_bytes(long long pixels, int per) {
  return 256 + hit_region_bytes(pixels) + size_t(pixels) * sizeof(float4) * (1 + size_t(per));
}

// Byte offsets of the hit records, the FP32 origins and the stage-S records.
static void scratch_offsets(long long pixels, size_t off[3]) {
  off[0] = 256;
  off[1] = 256 + hit_region_bytes(pixels);
  off[2] = off[1] + size_t(pixels) * sizeof(float4);
}

static void scratch_layout(Launch &L, void *base, long long pixels) {
  char *p = static_cast<char *>(base);
  size_t off[3];
  scratch_offsets(pixels, off);
  L.ctr = reinterpret_cast<Counters4 *>(p);
  L.gate = nullptr;
  L.hits = reinterpret_cast<HitRec *>(p + off[0]);
  L.sorg = reinterpret_cast<float4 *>(p + off[1]);
  L.sdir = reinterpret_cast<float4 *>(p + off[2]);
}

static int *scratch_gate(void *base) { return reinterpret_cast<int *>(static_cast<char *>(base) + 128); }

static bool is_wavefront(int engine) {
  return engine == MBR_ENGINE_WAVEFRONT_FP32 || engine == MBR_ENGINE_WAVEFRONT_FP64 ||
         engine == MBR_ENGINE_WAVEFRONT_AUTO;
}

mbr_status render_wavefront(mbr_ctx *ctx, const DevScene &sc, const DevFrame &fr, const DevOutputs &out, int engine,
                            void *stream) {
  if (!is_wavefront(engine)) return set_err(ctx, MBR_EINVAL, "not a wavefront engine: %d", engine);
  mbr_status stt = check_supported(ctx, sc, fr, false);
  if (stt != MBR_OK) return stt;
  // hybrids and formulas without a specialised form iterate in the reference's order (PrecHybT)
  const bool gi = fr.gi_samples > 0, hyb = sc.is_hybrid != 0 || sc.generic != 0;
  if (gi && fr.gi_bounces > 120)
    return set_err(ctx, MBR_EUNSUPPORTED, "wavefront engine: GI with more than 120 bounces uses the plain engines");
  if (hyb && engine == MBR_ENGINE_WAVEFRONT_FP64)
    return set_err(ctx, MBR_EUNSUPPORTED, "wavefront engine: hybrid sequences and formulas other than the Mandelbulb, "
                                          "Mandelbox and Menger sponge iterate in FP32 (MBR_ENGINE_WAVEFRONT_FP32 or "
                                          "_AUTO); in FP64 they use MBR_ENGINE_PLAIN_FP64");
  const mbr_tuning tu = ctx_tuning(ctx);
  const WJob j0 = make_job(fr, 0, out.pixel_offset);
  const long long pixels = (long long)fr.width * (fr.row1 - fr.row0);
  const long long total = gi ? pixels * (long long)fr.gi_samples : job_items(j0, tu.queue_layout);
  const int per = ((fr.shading_enable && fr.shadow_enable) ? 1 : 0) + ao_tasks(fr);
  // scratch: counters, then the GI accumulators or the hit records
  // GI: a counter block per bounce level (4 KiB), the auto-engine flag, the
  // path radiances and two vertex lists of one entry per path
  const size_t gi_head = 4096 + 256;
  const size_t bytes = gi ? gi_head + size_t(total) * (sizeof(double) + 2 * sizeof(HitRec)) : scratch_bytes(total, per);
  unsigned long long *work = nullptr;
  stt = ctx_work(ctx, (bytes + 7) / 8, &work);
  if (stt != MBR_OK) return stt;
  Launch L;
  std::memset(&L, 0, sizeof(L));
  L.jobs = nullptr;
  L.fps = nullptr;
  L.wps = nullptr;
  L.njobs = 1;
  L.total = total;
  if (gi) {
    char *w = reinterpret_cast<char *>(work);
    L.ctr = reinterpret_cast<Counters4 *>(w);
    L.path_rad = reinterpret_cast<double *>(w + gi_head);
    L.hits = reinterpret_cast<HitRec *>(w + gi_head + sizeof(double) * size_t(total));
    L.hits_next = L.hits + total;
  } else {
    scratch_layout(L, work, total);
  }
  L.refill_k = tu.refill_k;
  L.layout = tu.queue_layout;
  L.ao_rays = ao_tasks(fr);
  L.ao_fast = fr.ao_fast;
  L.shadow_tasks = (fr.shading_enable && fr.shadow_enable) ? 1 : 0;
  L.want_normal = fr.want_normal;
  const FastParams fp = load_fast_params(sc);
  const WideParams wp = load_wide_params(sc);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int e = 0;
  if (hyb)  // FP32 iteration in the reference's order
    return cuda_err(ctx, pipeline_hybrid(sc, tu, s, fr, j0, L, out, pixels), "wavefront launch");
  if (engine == MBR_ENGINE_WAVEFRONT_AUTO) {
    int *gate = gi ? reinterpret_cast<int *>(reinterpret_cast<char *>(work) + 4096) : scratch_gate(work);
    L.gate = gate;
    policy_kernel<<<1, 32, 0, s>>>(sc, fr, gate);
    count_launches(1);
    e = int(cudaGetLastError());
  }
  if (!e && engine != MBR_ENGINE_WAVEFRONT_FP64)
    e = pipeline_fp32(fast_kind(fp), tu, s, fr, fp, j0, L, out, pixels);
  if (!e && engine != MBR_ENGINE_WAVEFRONT_FP32)
    e = pipeline_fp64(wide_kind(wp), tu, s, fr, wp, j0, L, out, pixels);
  return cuda_err(ctx, e, "wavefront launch");
}

}  // namespace mbr

// ============================================================================
// Batches and the autotuner
// ============================================================================
using namespace mbr;

// One pipeline of a batch: the jobs of one formula kind and one precision.
struct BatchGroup {
  int wide;              // 1: Prec64
  int kind;              // FK_* of its jobs
  int offset, count;     // jobs [offset, offset + count) of the batch's job table
  long long items;       // work items of its pixel queue
  long long pixels;
};

struct mbr_batch {
  mbr_ctx *ctx = nullptr;
  WJob *d_jobs = nullptr;
  FastParams *d_params = nullptr;
  WideParams *d_wide = nullptr;
  void *d_scratch = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  long long total = 0;
  int launches = 0;  // kernels in the graph
  std::vector<BatchGroup> groups;
};

// Scratch of one group, a multiple of 256 bytes.
static size_t group_scratch(const BatchGroup &g, int per) { return (scratch_bytes(g.items, per) + 255) / 256 * 256; }

// Whether two jobs write a pixel in common.  Groups that run in turn then leave
// the last one's; side by side they would race.
static bool jobs_overlap(const std::vector<WJob> &jobs) {
  std::vector<std::pair<long long, long long>> span;
  for (const WJob &j : jobs) {
    const long long first = j.pixel_offset + (long long)j.row0 * j.width;
    span.push_back({first, first + (long long)j.rows * j.width});
  }
  std::sort(span.begin(), span.end());
  for (size_t i = 1; i < span.size(); i++)
    if (span[i].first < span[i - 1].second) return true;
  return false;
}

// Precision flag of every job (AUTO): the policy kernel over the job table.
static int batch_policy(const std::vector<DevScene> &dsc, const std::vector<int> &scene_of,
                        const std::vector<WJob> &wj, const DevFrame &fr0, std::vector<int> *flags) {
  const int n = int(wj.size());
  DevScene *d_sc = nullptr;
  int *d_of = nullptr, *d_fl = nullptr;
  WJob *d_wj = nullptr;
  int e = int(cudaMalloc(&d_sc, sizeof(DevScene) * dsc.size()));
  if (!e) e = int(cudaMalloc(&d_of, sizeof(int) * n));
  if (!e) e = int(cudaMalloc(&d_fl, sizeof(int) * n));
  if (!e) e = int(cudaMalloc(&d_wj, sizeof(WJob) * n));
  if (!e) e = int(cudaMemcpy(d_sc, dsc.data(), sizeof(DevScene) * dsc.size(), cudaMemcpyHostToDevice));
  if (!e) e = int(cudaMemcpy(d_of, scene_of.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
  if (!e) e = int(cudaMemcpy(d_wj, wj.data(), sizeof(WJob) * n, cudaMemcpyHostToDevice));
  if (!e) {
    batch_policy_kernel<<<(n + 127) / 128, 128>>>(d_sc, d_of, d_wj, n, fr0, d_fl);
    count_launches(1);
    e = int(cudaGetLastError());
  }
  flags->assign(n, 0);
  if (!e) e = int(cudaMemcpy(flags->data(), d_fl, sizeof(int) * n, cudaMemcpyDeviceToHost));
  cudaFree(d_sc);
  cudaFree(d_of);
  cudaFree(d_fl);
  cudaFree(d_wj);
  return e;
}

extern "C" {

mbr_status mbr_batch_create(mbr_ctx *ctx, const mbr_scene *scenes, int32_t n_scenes, const mbr_job *jobs,
                            int32_t n_jobs, const mbr_render_params *params, const mbr_outputs *outs, int engine,
                            void *stream, mbr_batch **batch) {
  if (!batch) return set_err(ctx, MBR_EINVAL, "null batch pointer");
  *batch = nullptr;
  if (!ctx || !scenes || !jobs || !params || !outs || n_scenes < 1 || n_jobs < 1)
    return set_err(ctx, MBR_EINVAL, "null argument or empty batch");
  if (!is_wavefront(engine)) return set_err(ctx, MBR_EUNSUPPORTED, "batches run on the wavefront engines");
  const mbr_tuning tu = ctx_tuning(ctx);
  std::vector<DevScene> dsc(n_scenes);
  for (int i = 0; i < n_scenes; i++) {
    mbr_status st = build_scene(ctx, scenes[i], &dsc[i]);
    if (st != MBR_OK) return st;
  }
  DevFrame fr0;
  std::vector<WJob> wj(n_jobs);
  std::vector<int> scene_of(n_jobs);
  std::vector<long long> job_pixels(n_jobs);
  for (int i = 0; i < n_jobs; i++) {
    const mbr_job &jb = jobs[i];
    if (jb.scene_index < 0 || jb.scene_index >= n_scenes)
      return set_err(ctx, MBR_EINVAL, "job %d: scene_index %d out of range", i, jb.scene_index);
    if (jb.pixel_offset < 0) return set_err(ctx, MBR_EINVAL, "job %d: negative pixel_offset", i);
    DevFrame fr;
    mbr_status st = build_frame(ctx, jb.camera, *params, &fr, stream);
    if (st != MBR_OK) return st;
    st = check_supported(ctx, dsc[jb.scene_index], fr, true);
    if (st != MBR_OK) return st;
    if (i == 0) fr0 = fr;
    wj[i] = make_job(fr, 0, jb.pixel_offset);
    scene_of[i] = jb.scene_index;
    job_pixels[i] = (long long)fr.width * (fr.row1 - fr.row0);
  }
  fr0.want_normal = outs->normal != nullptr;
  {  // the gamma table was copied on `stream`; the graph may be launched on another
    const int e = int(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
    if (e) return cuda_err(ctx, e, "cudaStreamSynchronize");
  }
  // precision of every job
  std::vector<int> wide(n_jobs, engine == MBR_ENGINE_WAVEFRONT_FP64 ? 1 : 0);
  if (engine == MBR_ENGINE_WAVEFRONT_AUTO) {
    const int e = batch_policy(dsc, scene_of, wj, fr0, &wide);
    if (e) return cuda_err(ctx, e, "batch precision policy");
  }
  // groups of one (precision, formula kind), each a contiguous run of the job table
  std::map<std::pair<int, int>, std::vector<int>> by_group;
  for (int i = 0; i < n_jobs; i++) {
    const DevScene &sc = dsc[scene_of[i]];
    const int kind = wide[i] ? wide_kind(load_wide_params(sc)) : fast_kind(load_fast_params(sc));
    by_group[{wide[i], kind}].push_back(i);
  }
  mbr_batch *b = new mbr_batch();
  b->ctx = ctx;
  std::vector<WJob> tab;
  std::vector<FastParams> fps;
  std::vector<WideParams> wps;
  tab.reserve(n_jobs);
  fps.reserve(n_jobs);
  wps.reserve(n_jobs);
  long long max_items = 0;
  for (const auto &kv : by_group) {
    BatchGroup g;
    g.wide = kv.first.first;
    g.kind = kv.first.second;
    g.offset = int(tab.size());
    g.count = int(kv.second.size());
    g.items = 0;
    g.pixels = 0;
    for (int i : kv.second) {
      WJob j = wj[i];
      j.first = g.items;
      g.items += job_items(j, tu.queue_layout);
      g.pixels += job_pixels[i];
      tab.push_back(j);
      fps.push_back(load_fast_params(dsc[scene_of[i]]));
      wps.push_back(load_wide_params(dsc[scene_of[i]]));
    }
    max_items = std::max(max_items, g.items);
    b->groups.push_back(g);
  }
  b->total = 0;
  for (const BatchGroup &g : b->groups) b->total += g.items;
  auto fail = [&](int e, const char *what) {
    mbr_batch_destroy(b);
    return cuda_err(ctx, e, what);
  };
  int e = int(cudaMalloc(&b->d_jobs, sizeof(WJob) * n_jobs));
  if (e) return fail(e, "cudaMalloc(jobs)");
  e = int(cudaMalloc(&b->d_params, sizeof(FastParams) * n_jobs));
  if (e) return fail(e, "cudaMalloc(params)");
  e = int(cudaMalloc(&b->d_wide, sizeof(WideParams) * n_jobs));
  if (e) return fail(e, "cudaMalloc(wide params)");
  const int per = ((fr0.shading_enable && fr0.shadow_enable) ? 1 : 0) + ao_tasks(fr0);
  // Scratch: one region that the groups use in turn, or, where together they
  // take at most an eighth of the device's free memory and no two jobs write the
  // same pixel, one region each, so that the groups run side by side.
  size_t each = 0;
  for (const BatchGroup &g : b->groups) each += group_scratch(g, per);
  size_t free_bytes = 0, total_bytes = 0;
  e = int(cudaMemGetInfo(&free_bytes, &total_bytes));
  if (e) return fail(e, "cudaMemGetInfo");
  bool side_by_side = b->groups.size() > 1 && each <= free_bytes / 8 && !jobs_overlap(wj);
  if (side_by_side && cudaMalloc(&b->d_scratch, each) != cudaSuccess) {
    cudaGetLastError();
    b->d_scratch = nullptr;
    side_by_side = false;
  }
  if (!side_by_side) {
    e = int(cudaMalloc(&b->d_scratch, scratch_bytes(max_items, per)));
    if (e) return fail(e, "cudaMalloc(scratch)");
  }
  e = int(cudaMemcpy(b->d_jobs, tab.data(), sizeof(WJob) * n_jobs, cudaMemcpyHostToDevice));
  if (e) return fail(e, "cudaMemcpy(jobs)");
  e = int(cudaMemcpy(b->d_params, fps.data(), sizeof(FastParams) * n_jobs, cudaMemcpyHostToDevice));
  if (e) return fail(e, "cudaMemcpy(params)");
  e = int(cudaMemcpy(b->d_wide, wps.data(), sizeof(WideParams) * n_jobs, cudaMemcpyHostToDevice));
  if (e) return fail(e, "cudaMemcpy(wide params)");
  // Capture the groups' pipelines of one batch into a graph, side by side or
  // in turn.  Side by side the FP64 groups begin: their stage S ends in a long
  // tail of single marches (jobs with the camera inside the solid), and the
  // FP32 groups, which wait until it can start, fill it (128 jobs: in turn
  // 195 ms, all groups at once 188 ms, FP32 after the FP64 stage P 182 ms, so
  // 173 ms).
  std::vector<cudaStream_t> streams(side_by_side ? b->groups.size() + 1 : 1, nullptr);
  std::vector<cudaEvent_t> events(side_by_side ? b->groups.size() + 1 : 1, nullptr);
  for (size_t i = 0; i < streams.size() && !e; i++) {
    e = int(cudaStreamCreateWithFlags(&streams[i], cudaStreamNonBlocking));
    if (!e) e = int(cudaEventCreateWithFlags(&events[i], cudaEventDisableTiming));
  }
  const cudaStream_t cs = streams[0];
  const DevOutputs d = dev_outputs(ctx, *outs);
  const char *failed = "cudaStreamCreate";
  if (!e) {
    failed = "graph capture";
    e = int(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
  }
  if (!e) {
    const int64_t before = mbr_kernel_launches();
    int le = side_by_side ? int(cudaEventRecord(events[0], cs)) : 0;
    char *scratch = static_cast<char *>(b->d_scratch);
    std::vector<size_t> order, forked;
    for (int wide = 1; wide >= 0; wide--)
      for (size_t i = 0; i < b->groups.size(); i++)
        if (b->groups[i].wide == wide) order.push_back(i);
    if (!side_by_side) std::sort(order.begin(), order.end());  // in turn: FP32 first, as the groups lie
    for (size_t i : order) {
      if (le) break;
      const BatchGroup &g = b->groups[i];
      const cudaStream_t gs = side_by_side ? streams[i + 1] : cs;
      if (side_by_side) {
        le = int(cudaStreamWaitEvent(gs, events[0], 0));
        if (!le) forked.push_back(i);
        for (size_t j : forked)
          if (!le && !g.wide && b->groups[j].wide) le = int(cudaStreamWaitEvent(gs, events[j + 1], 0));
        if (le) break;
      }
      Launch L;
      std::memset(&L, 0, sizeof(L));
      L.jobs = b->d_jobs + g.offset;
      L.fps = b->d_params + g.offset;
      L.wps = b->d_wide + g.offset;
      L.njobs = g.count;
      L.total = g.items;
      scratch_layout(L, scratch, g.items);
      if (side_by_side) scratch += group_scratch(g, per);
      L.refill_k = tu.refill_k;
      L.layout = tu.queue_layout;
      L.ao_rays = ao_tasks(fr0);
      L.ao_fast = fr0.ao_fast;
      L.shadow_tasks = (fr0.shading_enable && fr0.shadow_enable) ? 1 : 0;
      L.want_normal = fr0.want_normal;
      if (g.wide)
        le = pipeline_batch_fp64(g.kind, tu, gs, fr0, wps[g.offset], tab[g.offset], L, d, g.pixels,
                                 side_by_side ? events[i + 1] : nullptr);
      else
        le = pipeline_batch_fp32(g.kind, tu, gs, fr0, fps[g.offset], tab[g.offset], L, d, g.pixels);
    }
    // every branch that was forked has to join before the capture ends
    for (size_t i : forked) {
      int je = int(cudaEventRecord(events[i + 1], streams[i + 1]));
      if (!je) je = int(cudaStreamWaitEvent(cs, events[i + 1], 0));
      if (!le) le = je;
    }
    b->launches = int(mbr_kernel_launches() - before);  // recorded, not queued
    count_launches(-b->launches);
    cudaGraph_t gr = nullptr;
    e = int(cudaStreamEndCapture(cs, &gr));
    b->graph = gr;
    if (!e) e = le;
  }
  for (cudaStream_t st : streams)
    if (st) cudaStreamDestroy(st);
  for (cudaEvent_t ev : events)
    if (ev) cudaEventDestroy(ev);
  if (e) return fail(e, failed);
  e = int(cudaGraphInstantiate(&b->exec, b->graph, 0));
  if (e) return fail(e, "cudaGraphInstantiate");
  *batch = b;
  return MBR_OK;
}

mbr_status mbr_batch_launch(mbr_batch *b, void *stream) {
  if (!b) return MBR_EINVAL;
  const int e = int(cudaGraphLaunch(b->exec, static_cast<cudaStream_t>(stream)));
  if (!e) count_launches(b->launches);
  return cuda_err(b->ctx, e, "cudaGraphLaunch");
}

void mbr_batch_destroy(mbr_batch *b) {
  if (!b) return;
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  if (b->d_jobs) cudaFree(b->d_jobs);
  if (b->d_params) cudaFree(b->d_params);
  if (b->d_wide) cudaFree(b->d_wide);
  if (b->d_scratch) cudaFree(b->d_scratch);
  delete b;
}

mbr_status mbr_choose_precision(mbr_ctx *ctx, const mbr_camera *camera, const mbr_render_params *params,
                                int32_t *fp64) {
  if (!ctx || !camera || !params || !fp64) return set_err(ctx, MBR_EINVAL, "null argument");
  const DevScene *sc = ctx_scene(ctx);
  if (!sc) return set_err(ctx, MBR_EINVAL, "no scene set (call mbr_scene_set first)");
  if (cudaSetDevice(ctx_device(ctx)) != cudaSuccess) return set_err(ctx, MBR_ECUDA, "cudaSetDevice failed");
  DevFrame fr;
  mbr_status st = build_frame(ctx, *camera, *params, &fr, nullptr);
  if (st != MBR_OK) return st;
  int *d_flag = nullptr;
  int e = int(cudaMalloc(&d_flag, sizeof(int)));
  if (e) return cuda_err(ctx, e, "cudaMalloc(flag)");
  policy_kernel<<<1, 32>>>(*sc, fr, d_flag);
  count_launches(1);
  e = int(cudaGetLastError());
  int flag = 0;
  if (!e) e = int(cudaMemcpy(&flag, d_flag, sizeof(int), cudaMemcpyDeviceToHost));
  cudaFree(d_flag);
  if (e) return cuda_err(ctx, e, "precision policy");
  *fp64 = flag;
  return MBR_OK;
}

mbr_status mbr_wavefront_scratch_layout(int64_t pixels, int32_t tasks_per_hit, uint64_t offsets[3],
                                        uint64_t *total_bytes) {
  if (pixels < 0 || tasks_per_hit < 0 || !offsets || !total_bytes) return MBR_EINVAL;
  size_t off[3];
  scratch_offsets(pixels, off);
  for (int i = 0; i < 3; i++) offsets[i] = off[i];
  *total_bytes = scratch_bytes(pixels, tasks_per_hit);
  return MBR_OK;
}

int32_t mbr_batch_groups(const mbr_batch *b, int32_t *wide_jobs) {
  if (!b) return -1;
  int32_t w = 0;
  for (const BatchGroup &g : b->groups)
    if (g.wide) w += g.count;
  if (wide_jobs) *wide_jobs = w;
  return int32_t(b->groups.size());
}

// Times the wavefront pipeline on the given frame over block size x CTAs per
// SM x refill threshold x queue layout and keeps the fastest configuration.
mbr_status mbr_autotune(mbr_ctx *ctx, const mbr_camera *camera, const mbr_render_params *params,
                        const mbr_outputs *out, int engine, void *stream, mbr_tuning *best) {
  if (!ctx || !camera || !params || !out || !best) return set_err(ctx, MBR_EINVAL, "null argument");
  const mbr_tuning saved = ctx_tuning(ctx);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  mbr_tuning bt = saved;
  const int blocks[] = {128, 256};  // __launch_bounds__(256)
  const int ctas[] = {6, 8, 12};
  const int ks[] = {0, 2, 4, 8, 16, 24};
  const int layouts[] = {0, 1};
  mbr_status status = MBR_OK;
  // one timed frame per launch shape, then the four fastest re-timed three
  // times each: the median decides (a single frame can be lucky by several
  // per cent, more than the shapes differ)
  std::vector<std::pair<float, mbr_tuning>> cand;
  auto time_one = [&](const mbr_tuning &t, float *ms) {
    ctx_tuning(ctx) = t;
    mbr_status s2 = mbr_render(ctx, camera, params, out, engine, stream);  // warm-up
    if (s2 != MBR_OK) return s2;
    cudaEventRecord(e0, st);
    s2 = mbr_render(ctx, camera, params, out, engine, stream);
    cudaEventRecord(e1, st);
    if (s2 != MBR_OK) return s2;
    cudaEventSynchronize(e1);
    cudaEventElapsedTime(ms, e0, e1);
    return MBR_OK;
  };
  for (int b : blocks)
    for (int c : ctas) {
      if (b * c > 2048) continue;
      for (int k : ks)
        for (int l : layouts) {
          const mbr_tuning t{b, c, k, l};
          float ms = 0.f;
          status = time_one(t, &ms);
          if (status != MBR_OK) goto done;
          cand.push_back({ms, t});
        }
    }
  std::sort(cand.begin(), cand.end(),
            [](const std::pair<float, mbr_tuning> &a, const std::pair<float, mbr_tuning> &b) { return a.first < b.first; });
  {
    float best_ms = 1e30f;
    for (size_t i = 0; i < cand.size() && i < 4; i++) {
      float m[3];
      for (int r = 0; r < 3; r++) {
        status = time_one(cand[i].second, &m[r]);
        if (status != MBR_OK) goto done;
      }
      std::sort(m, m + 3);
      if (m[1] < best_ms) {
        best_ms = m[1];
        bt = cand[i].second;
      }
    }
  }
done:
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  ctx_tuning(ctx) = (status == MBR_OK) ? bt : saved;
  *best = ctx_tuning(ctx);
  return status;
}

}  // extern "C"

// ============================================================================
// Allocation-free rendering
//
// For callers that cannot allocate device memory: a host application whose
// device memory is owned by its own allocator or memory pool (which must not
// be bypassed), or a process running under a hard memory cap, where a
// cudaMalloc in the middle of a frame could fail or synchronise the device.
// The wavefront pipeline's scratch (hit records, stage-S start records,
// launch counters, the gamma table and the status word) lives in one
// file-scope device array, part of this library's device image: every GPU
// that loads the library holds it until the process exits.
// ============================================================================
namespace {

static __device__ __align__(256) unsigned char g_noalloc_scratch[MBR_NOALLOC_SCRATCH_BYTES];

const size_t kGammaBytes = 65536 * sizeof(uint16_t);
const size_t kHeadBytes = kGammaBytes + 256;  // gamma table, then the status word

struct NoallocDevice {
  bool ready = false;
  unsigned char *base = nullptr;  // device address of g_noalloc_scratch on this device
  double gamma_value = -1.0;      // gamma of the table currently in the array
};
const int kMaxDevices = 64;
NoallocDevice g_noalloc[kMaxDevices];
std::mutex g_noalloc_mutex;
uint16_t g_noalloc_gamma_host[65536];  // host staging table of the gamma copies

mbr_status noalloc_fail(char *err, size_t err_len, mbr_status st, const std::string &msg) {
  if (err && err_len) std::snprintf(err, err_len, "%s", msg.c_str());
  return st;
}

// The largest pixel count whose scratch fits in `have` bytes.
long long noalloc_max_pixels(int per, size_t have) {
  const size_t per_pixel = sizeof(HitRec) + sizeof(float4) * (1 + size_t(per));
  long long n = (long long)((have - 256 - 255) / per_pixel);  // the hit region rounds up by < 256 bytes
  while (scratch_bytes(n + 1, per) <= have) n++;
  return n;
}

}  // namespace

extern "C" mbr_status mbr_render_noalloc(const mbr_scene *scene, const mbr_camera *camera,
                                         const mbr_render_params *params, const mbr_outputs *out, void *stream,
                                         char *err, size_t err_len) {
  if (err && err_len) err[0] = '\0';
  if (!scene || !camera || !params || !out) return noalloc_fail(err, err_len, MBR_EINVAL, "null argument");
  int dev = 0;
  int e = int(cudaGetDevice(&dev));
  if (e || dev < 0 || dev >= kMaxDevices)
    return noalloc_fail(err, err_len, MBR_ECUDA, "no current CUDA device");
  // one-time set-up on this device: the device address of the scratch array
  // (host code may not use the array's name as a device address)
  NoallocDevice *nd = &g_noalloc[dev];
  {
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!nd->ready) {
      void *ptr = nullptr;
      e = int(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
      if (e || !ptr)
        return noalloc_fail(err, err_len, MBR_ECUDA,
                            std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(cudaError_t(e)));
      nd->base = static_cast<unsigned char *>(ptr);
      nd->ready = true;
    }
  }
  DevScene sc;
  mbr_status st = build_scene(nullptr, *scene, &sc);
  if (st != MBR_OK) return noalloc_fail(err, err_len, st, "invalid or unsupported scene (see mbr_scene_set)");
  DevFrame fr;
  std::string msg;
  {
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);  // the host staging table is shared
    st = build_frame_owned_gamma(*camera, *params, reinterpret_cast<uint16_t *>(nd->base), g_noalloc_gamma_host,
                                 &nd->gamma_value, &fr, stream, &msg);
  }
  if (st != MBR_OK) return noalloc_fail(err, err_len, st, msg);
  fr.want_normal = out->normal != nullptr;
  if (sc.is_hybrid || sc.generic || sc.iter_thresh || sc.interior || sc.has_w || fr.gi_samples > 0 ||
      fr.refine != MBR_REFINE_REFERENCE || fr.slow_shading)
    return noalloc_fail(err, err_len, MBR_EUNSUPPORTED,
                        "the wavefront engine renders non-hybrid Mandelbulb, Mandelbox and Menger scenes without GI, "
                        "root refinement, iteration threshold, interior mode, initial w or slow shading");
  const long long total = (long long)fr.width * (fr.row1 - fr.row0);  // row-linear queue: no tile padding
  const int per = ((fr.shading_enable && fr.shadow_enable) ? 1 : 0) + ao_tasks(fr);
  const size_t need = scratch_bytes(total, per);
  const size_t have = size_t(MBR_NOALLOC_SCRATCH_BYTES) - kHeadBytes;
  if (need > have) {
    char buf[320];
    std::snprintf(buf, sizeof(buf),
                  "frame of %lld pixels with %d shadow/AO tasks per hit needs %zu bytes of scratch; the "
                  "allocation-free entry point has %zu (at most %lld pixels at this setting)",
                  total, per, need, have, noalloc_max_pixels(per, have));
    return noalloc_fail(err, err_len, MBR_EINVAL, buf);
  }
  Launch L;
  std::memset(&L, 0, sizeof(L));
  L.njobs = 1;
  L.total = total;
  scratch_layout(L, nd->base + kHeadBytes, total);
  const mbr_tuning tu{128, 12, 2, 0};
  L.refill_k = tu.refill_k;
  L.layout = tu.queue_layout;
  L.ao_rays = ao_tasks(fr);
  L.ao_fast = fr.ao_fast;
  L.shadow_tasks = (fr.shading_enable && fr.shadow_enable) ? 1 : 0;
  L.want_normal = fr.want_normal;
  DevOutputs d;
  d.depth = out->depth;
  d.iters = out->iters;
  d.hit = out->hit;
  d.normal = out->normal;
  d.shade = out->shade;
  d.ao = out->ao;
  d.rgb = out->rgb;
  d.rgb8 = out->rgb8;
  d.stats = out->stats;
  d.status = reinterpret_cast<int32_t *>(nd->base + kGammaBytes);
  d.pixel_offset = 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the array keeps the previous call's contents: the status word starts at
  // zero here and the launch counters are zeroed at the head of the pipeline
  e = int(cudaMemsetAsync(d.status, 0, sizeof(int32_t), s));
  if (e) return noalloc_fail(err, err_len, MBR_ECUDA, std::string("cudaMemsetAsync: ") + cudaGetErrorString(cudaError_t(e)));
  const WJob j0 = make_job(fr, 0, 0);
  const FastParams fp = load_fast_params(sc);
  e = pipeline_fp32(fast_kind(fp), tu, s, fr, fp, j0, L, d, total);
  if (e) return noalloc_fail(err, err_len, MBR_ECUDA, std::string("wavefront launch: ") + cudaGetErrorString(cudaError_t(e)));
  return MBR_OK;
}
