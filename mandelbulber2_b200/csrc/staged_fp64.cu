// staged_fp64.cu - the staged frames of the plain FP64 engine.
#include "staged_plain.cuh"

namespace mbr {
int launch_staged_fp64(const DevScene &sc, const DevFrame &fr, const DevOutputs &out, void *scratch, void *stream) {
  return launch_staged_plain_t<double, 0>(sc, fr, out, scratch, stream);
}
size_t staged_plain_scratch(const DevScene &sc, const DevFrame &fr) {
  return staged_plain_takes(sc, fr) ? staged_plain_bytes(fr) : 0;
}
}  // namespace mbr
