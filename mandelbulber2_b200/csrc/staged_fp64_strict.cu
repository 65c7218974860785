// staged_fp64_strict.cu - the staged frames of the plain FP64 engine, compiled with --fmad=false.
#define MBR_NO_FMA 1
#include "staged_plain.cuh"

namespace mbr {
int launch_staged_fp64_strict(const DevScene &sc, const DevFrame &fr, const DevOutputs &out, void *scratch, void *stream) {
  return launch_staged_plain_t<double, 1>(sc, fr, out, scratch, stream);
}
}  // namespace mbr
