// Where an exact truncated SVD (block subspace iteration) looks at its residuals.
#pragma once

#include <algorithm>
#include <cmath>

namespace tg {

// A check (orthonormalisation, Jacobi, host read) costs three to five
// iterations, so a solve should need one or two of them.  `ratio` is the largest
// kept residual over the tolerance: the solve is done at ratio <= 1.
//
// fixed: the first check at 1 (from the basis of the last solve) or 3, the next
// three later, the others from the decay of the last two, for contexts whose
// results depend on where a solve ends (EngineT::keep_order).
//
// Otherwise the first check is where the projector's last solve in this
// environment ended, the next ones come from the decay seen between two checks
// or, before there are two, expected from the block's spectrum, with one iteration
// in hand: without it the first sweeps' solves ended close below the tolerance,
// and the density matrices of 2 x 2, D = 3 complex environments of chi = 25, 27 and
// 29 were 1.2e-13, 2.5e-13 and 2.3e-13 off those in 64 bits (geometric means of 8);
// with it 0.8e-13, 1.6e-13 and 1.3e-13, at fixed places 0.7e-13, 0.8e-13 and 1.9e-13
// (a second run of a context 2.0e-13, 1.3e-13 and 3.3e-13), in 0.8 of the time.
struct ExactSteps {
  static constexpr int kMaxIters = 80;

  bool fixed = false;
  int prev_it = 0;  // the last check, 0: none
  double prev_ratio = 0.0;

  // the first check; hint: hint() of the projector's last solve, 0: none
  int first(bool warm, int hint) const { return !fixed && hint > 0 ? hint : warm ? 1 : 3; }
  bool falling(double ratio) const { return prev_it > 0 && ratio < prev_ratio; }
  // the residuals' decay an iteration; edge: the same expected from the spectrum
  double decay(int it, double ratio, double edge) const {
    return falling(ratio) ? std::pow(ratio / prev_ratio, 1.0 / (it - prev_it)) : std::min(0.5, edge);
  }
  // After a check at `it` with ratio > 1: iterations to the next one, or 0 for a
  // solve to be given up (for the dense SVD).
  int next(int it, double ratio, double edge) {
    const double f = decay(it, ratio, edge);
    const double need = f > 0.0 ? std::max(1.0, std::ceil(std::log(ratio) / -std::log(f))) : 3.0;
    const int left = kMaxIters - it;
    int gap = 3;
    if (falling(ratio)) gap = static_cast<int>(std::min(16.0, need));
    else if (prev_it == 0 && !fixed) gap = static_cast<int>(std::min(16.0, need + 1.0));
    if (fixed) {
      if (prev_it > 0 && it > 12 && ratio > 0.5 * prev_ratio) return 0;
    } else {
      // stalled is what cannot end in the iterations left, by the decay of an
      // iteration: a late first check can be followed by a gap of one, over which a
      // sound decay is 0.8.  (Judged by a ratio of 0.5 between two checks, solves of
      // 30 iterations at D = 4, chi = 60 went to the dense SVD.)
      if (falling(ratio) && it > 12 && need > left) return 0;
      if (prev_it > 0 && !falling(ratio) && it > 12 && it - prev_it >= 3) return 0;
      if (left > 0) gap = std::min(gap, left);
    }
    if (gap > left) return 0;
    prev_it = it;
    prev_ratio = ratio;
    return gap;
  }
  // After the last check, at `it`: where the next solve looks first, one or two
  // iterations earlier where the residual shows them to spare.
  int hint(int it, double ratio, double edge) const {
    const double f = decay(it, ratio, edge);
    int spare = 0;
    while (spare < 2 && f > 0.0 && ratio * std::pow(f, -(spare + 1)) <= 1.0) ++spare;
    return std::max(1, it - spare);
  }
};

}  // namespace tg
