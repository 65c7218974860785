// staged_keyed_fp64_strict.cu - staged frames of one formula by settings key, compiled with --fmad=false.
#define MBR_NO_FMA 1
#include "staged_plain.cuh"

namespace mbr {
int ref_keyed_fp64_strict(int formula, const DevScene &sc, const DevFrame &fr, const RefLaunch &L, const DevOutputs &out,
                       cudaStream_t s, bool *taken) {
  return ref_keyed_stages<double, 1>(formula, sc, fr, L, out, s, taken);
}
}  // namespace mbr
