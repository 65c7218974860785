// wavefront_hybrid.cu - single-frame pipelines in the reference's order: hybrids and extended scenes.
#include "wavefront.cuh"

namespace mbr {

// The kernels by what the scene needs: single formulas of the three with
// extensions; sequences of the Mandelbulb and the Menger sponge, of the Mandelbox
// and the Menger sponge, and of all three; and a general kernel of each kind that
// also takes blended slots and fast AO (the extended one: GI and every other
// formula).  Sequences of the Mandelbulb and the Mandelbox alone take the
// three-formula kernel: in one of the two the compiler fused other operations of
// the Mandelbox, and its frames differed from the general kernel's in last bits.  The general kernels alone against this choice: an 800x600
// Mandelbox with primitives 8.46 / 4.12 ms (its parameters become constant
// operands and 16 formulas leave the loop), 1080p x 16 spp GI of a
// Mandelbulb and Menger sequence 187.5 / 154.5 ms.
int pipeline_hybrid(const DevScene &sc, const mbr_tuning &tu, cudaStream_t st, const DevFrame &fr, const WJob &j0,
                    const Launch &L, const DevOutputs &out, long long pixels) {
  const HybParams hp{sc};
#define HYBRID(FEAT) return launch_pipeline<false, PrecHybT<(FEAT)>>(FK_ANY, tu, st, fr, hp, j0, L, out, pixels)
  const bool blend = orbit_blends(sc);
  int forms = 0;
  for_orbit_slots(sc, [&](const DevSlot &s) {  // an empty slot blends, which takes the general kernel
    forms |= s.formula == MBR_FORMULA_MANDELBULB  ? HB_BULB
             : s.formula == MBR_FORMULA_MANDELBOX ? HB_BOX
             : s.formula == MBR_FORMULA_MENGER_SPONGE ? HB_MENGER
             : s.formula == MBR_FORMULA_NONE ? 0
                                             : HB_ALL;
  });
  if (scene_extended(sc)) {
    // (the pseudo-Kleinian DE function's x^2 + y^2 shares products with the lean
    // kernels' |z|^2, and the compiler fuses it otherwise than in the general one)
    if (!sc.is_hybrid && !blend && fr.gi_samples == 0 && !L.ao_fast && sc.de_final != DEF_PSEUDO_KLEINIAN) {
      if (forms == HB_BOX) HYBRID(HB_EXT | HB_BOX);
      if (forms == HB_BULB) HYBRID(HB_EXT | HB_BULB);
      if (forms == HB_MENGER) HYBRID(HB_EXT | HB_MENGER);
    }
    HYBRID(HB_EXT | HB_ALL | HB_SEQ | HB_BLEND);
  }
  if (!blend && !L.ao_fast && !(forms & HB_ALL)) {
    if (!(forms & HB_BOX)) HYBRID(HB_BULB | HB_MENGER | HB_SEQ);
    if (!(forms & HB_BULB)) HYBRID(HB_BOX | HB_MENGER | HB_SEQ);
    HYBRID(HB_BULB | HB_BOX | HB_MENGER | HB_SEQ);
  }
  HYBRID(HB_BULB | HB_BOX | HB_MENGER | HB_SEQ | HB_BLEND);
#undef HYBRID
}
}  // namespace mbr
