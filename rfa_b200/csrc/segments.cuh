// How a causal sequence is cut into segments that different CTAs work on.
#pragma once

#include <stdint.h>

namespace rfa {

struct CausalPlan {
  int nseg;        // segments per (batch, head)
  int64_t tseg;    // tokens per segment (multiple of every kernel's chunk length)
};

constexpr int64_t kSms = 148;
// n chunks in segments of m, as short as `fit` segments a sequence (one wave) allow, where that saves a sequence `min_saved` chunks
inline CausalPlan cut_segments(int64_t T, int64_t chunk, int64_t fit, int64_t min_saved) {
  const int64_t n = (T + chunk - 1) / chunk;
  if (fit >= 2 && n >= 2) {
    const int64_t s = fit < n ? fit : n, m = (n + s - 1) / s;
    if (n - m >= min_saved) return CausalPlan{(int)((n + m - 1) / m), m * chunk};
  }
  return CausalPlan{1, n * chunk};
}

}  // namespace rfa
