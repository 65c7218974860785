// wavefront32.cu - single-frame pipelines with FP32 iteration.
#include "wavefront.cuh"

namespace mbr {
int pipeline_fp32(int fk, const mbr_tuning &tu, cudaStream_t st, const DevFrame &fr, const FastParams &fp, const WJob &j0,
                  const Launch &L, const DevOutputs &out, long long pixels) {
  return launch_pipeline<false, Prec32>(fk, tu, st, fr, fp, j0, L, out, pixels);
}
}  // namespace mbr
