// wavefront_batch.cu - batch pipelines (a job table), FP32 and FP64 iteration.
#include "wavefront.cuh"

namespace mbr {
int pipeline_batch_fp32(int fk, const mbr_tuning &tu, cudaStream_t st, const DevFrame &fr, const FastParams &fp, const WJob &j0,
                        const Launch &L, const DevOutputs &out, long long pixels) {
  return launch_pipeline<true, Prec32>(fk, tu, st, fr, fp, j0, L, out, pixels);
}

int pipeline_batch_fp64(int fk, const mbr_tuning &tu, cudaStream_t st, const DevFrame &fr, const WideParams &fp, const WJob &j0,
                        const Launch &L, const DevOutputs &out, long long pixels, cudaEvent_t before_shade) {
  return launch_pipeline<true, Prec64>(fk, tu, st, fr, fp, j0, L, out, pixels, before_shade);
}
}  // namespace mbr
