// Paths per wavefront of a render (plain C++).
#ifndef RX_WAVE_H
#define RX_WAVE_H
#include <algorithm>

namespace rx {

// Each extend launch ends in a tail where the last, longest rays run on an
// emptying GPU; larger waves amortise it (measured on the 1080p 64-spp
// icosphere scene, extend / frame time: 16 M paths 43.7 / 58.2 ms, 32 M
// 35.1 / 47.6 ms, 64 M 30.7 / 42.7 ms, 128 M (the whole frame in one wave)
// 28.0 / 39.9 ms).  By default the wave is the largest power of two from
// 32 M to 128 M paths whose state (path SoA, queues, hit and shadow records:
// ~120 B + 48 B per shadow record slot) fits in a quarter of the free device
// memory; 128 M paths hold ~22 GB.
//
// `frames` frames of `P` pixels, `per_shadow` shadow records a path; cap and
// shadow_cap: what the wave buffers hold by now.  free_bytes() asks for the
// free memory, which takes 70 us, and tens of milliseconds while another
// process of the machine holds the driver: it is called only when the answer
// can matter, that is for a wave of more than 32 M paths that the buffers do
// not hold yet.
template <class Free>
inline long long default_wave_paths(long long frames, long long P, long long cap, long long shadow_cap,
                                    long long per_shadow, Free free_bytes) {
  long long target = 1LL << 27;
  // the wave of that target: whole frames, so mostly less than the target
  const long long want = std::max(1LL, std::min(frames, target / std::max(P, 1LL))) * P;
  if (want > (1LL << 25) && (cap < want || shadow_cap < want * per_shadow)) {
    const long long quarter = free_bytes() / 4, per_path = 120 + 48 * per_shadow;
    while (target > (1LL << 25) && quarter < target * per_path) target >>= 1;
  }
  return target;
}

}  // namespace rx
#endif
