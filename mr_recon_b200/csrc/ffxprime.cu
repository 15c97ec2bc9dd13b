// Direct FFT passes of lengths with prime factors 7, 11, 13, 17 or 19 (ffx.cu
// chooses them per axis).
#include <algorithm>

#include "ffx_pass.cuh"

namespace mrn {

int launch_ffx_primes(const FfxSet& S, const FfxGrid& G, const FfxStep& step, bool inv, int source, bool to_image,
                      const float2* src, const float2* mps, float2* out, float scale, cudaStream_t st) {
#define MRN_FFXP(II, SS, TT)                                                                                  \
  do {                                                                                                        \
    if (step.w == 16) return launch_ffx_pass<II, SS, TT, 16, true, true>(S, G, step, src, mps, out, scale, st); \
    if (step.w == 8) return launch_ffx_pass<II, SS, TT, 8, true, true>(S, G, step, src, mps, out, scale, st);   \
    return launch_ffx_pass<II, SS, TT, 4, true, true>(S, G, step, src, mps, out, scale, st);                    \
  } while (0)
  if (inv) {
    if (to_image) MRN_FFXP(true, kFfxGrid, true);
    MRN_FFXP(true, kFfxGrid, false);
  }
  if (source == kFfxGrid) MRN_FFXP(false, kFfxGrid, false);
  if (source == kFfxImage) MRN_FFXP(false, kFfxImage, false);
  MRN_FFXP(false, kFfxSense, false);
#undef MRN_FFXP
}

}  // namespace mrn
