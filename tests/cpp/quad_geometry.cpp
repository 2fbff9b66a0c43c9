// Reads "W rows cols pitch" lines, prints whether the four-slice kernel may serve them.
#include <cstdio>

#include "../../ctas_b200/csrc/bp_quad_rule.hpp"

int main() {
  long long W, R, C;
  double p;
  while (std::scanf("%lld %lld %lld %lf", &W, &R, &C, &p) == 4)
    std::printf("%d\n", ctas::quad_sharing_exact(W, R, C, p) ? 1 : 0);
}
