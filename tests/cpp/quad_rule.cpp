// The stack rule (bp_quad_rule.hpp): reads "form width slices SMs" lines, prints the
// slices that go through groups, the tiles of a slice and the count from which groups
// always pay.
#include <cstdio>

#include "../../ctas_b200/csrc/bp_quad_rule.hpp"

int main() {
  int form, sms;
  long long W, S;
  while (std::scanf("%d %lld %lld %d", &form, &W, &S, &sms) == 4) {
    const ctas::SliceTiles t = ctas::slice_tiles(W, W, W, 0.0, 0.0, 1.0);
    const long long n = ctas::quad_slices((ctas::QuadForm)form, t, S, sms);
    std::printf("%lld %lld %lld %lld %lld\n", n, (long long)t.all64, (long long)t.in64,
                (long long)t.in32, (long long)ctas::quad_always(t, sms));
  }
}
