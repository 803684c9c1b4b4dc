// fb_kernels.h — host-side entry points of the pass kernels (internal).
#pragma once
#include <cuda_runtime.h>

#include "fb_passes.cuh"

namespace fb {

enum PassKind { kPassTransmittance = 0, kPassSingle = 1, kPassDensity = 2, kPassMultiple = 3 };

// Kernel of (mode, pass, texels-per-thread, variant, order 2). Multiple
// scattering: the variants of ms_variant (by the row's layout; 0 / 1 and 4 / 5
// = registers for 4 / 3 CTAs per SM). Density: occupancy variant 0-2, +
// kDensClamped with exact-size interval tables; order2 selects the launch of
// order 2 (it reads the single-scattering tables); from kDensArcs, orders >= 3
// by arcs, by the nu texels of a thread.
const void* kernel_plain(int pass, int tpt, int variant, bool order2);
const void* kernel_mixed(int pass, int tpt, int variant, bool order2);

inline const void* kernel_for(bool mixed, int pass, int tpt, int variant = 0, bool order2 = false) {
  return mixed ? kernel_mixed(pass, tpt, variant, order2) : kernel_plain(pass, tpt, variant, order2);
}

}  // namespace fb
