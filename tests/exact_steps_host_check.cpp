// Runs ExactSteps (exact_steps.hpp) on residuals that fall by a given factor an
// iteration.  stdin: lines of fixed, warm, hint, first ratio, decay, edge;
// stdout: iterations (0: given up), checks, last ratio, next hint.
#include <cstdio>

#include "exact_steps.hpp"

int main() {
  int fixed, warm, hint;
  double ratio0, decay, edge;
  while (std::scanf("%d %d %d %lf %lf %lf", &fixed, &warm, &hint, &ratio0, &decay, &edge) == 6) {
    tg::ExactSteps s{fixed != 0};
    int it = s.first(warm != 0, hint), checks = 1, gap = 1;
    double ratio = ratio0 * std::pow(decay, it);
    while (ratio > 1.0 && (gap = s.next(it, ratio, edge)) > 0) {
      it += gap;
      ++checks;
      ratio = ratio0 * std::pow(decay, it);
    }
    std::printf("%d %d %.17g %d\n", gap > 0 ? it : 0, checks, ratio, s.hint(it, ratio, edge));
  }
}
