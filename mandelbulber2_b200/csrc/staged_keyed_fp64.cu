// staged_keyed_fp64.cu - staged frames of one formula by settings key.
#include "staged_plain.cuh"

namespace mbr {
int ref_keyed_fp64(int formula, const DevScene &sc, const DevFrame &fr, const RefLaunch &L, const DevOutputs &out,
                cudaStream_t s, bool *taken) {
  return ref_keyed_stages<double, 0>(formula, sc, fr, L, out, s, taken);
}
}  // namespace mbr
