// Which launches share a tuned tile: prints nothing and returns 0 when every field that
// decides the kernel, its grid or how full the device is separates two launches.
#include "../../ctas_b200/csrc/bp_fast.hpp"

int main() {
  ctas::BpLaunch a{};
  a.W = 2560;
  a.N = 1800;
  a.out_rows = a.out_cols = 2560;
  a.S = 9;
  const auto key = ctas::bp_fast_tune_key(a, 0, false);
  ctas::BpLaunch same = a;
  same.S = 5;
  same.center = 3.5f;
  if (!(ctas::bp_fast_tune_key(same, 0, false) == key)) return 1;
  ctas::BpLaunch b[7] = {a, a, a, a, a, a, a};
  b[0].wide = 1;
  b[1].W = 2048;
  b[2].N = 900;
  b[3].store = 1;
  b[4].interp = 1;
  b[5].out_rows = 2048;
  b[6].out_cols = 2048;
  for (int i = 0; i < 7; i++)
    if (ctas::bp_fast_tune_key(b[i], 0, false) == key) return 10 + i;
  if (ctas::bp_fast_tune_key(a, 1, false) == key) return 20;
  if (ctas::bp_fast_tune_key(a, 0, true) == key) return 21;
  // fill: slices of 700 x 700 (121 tiles of 64 x 64) on 148 SMs
  ctas::BpLaunch c = a;
  c.W = c.out_rows = c.out_cols = 700;
  auto at = [&](int slices) {
    c.S = slices;
    return ctas::bp_fast_tune_key(c, 0, false, 148);
  };
  const float centre = 0.f;
  c.centers = &centre;
  if (!(at(1) == at(33)) || !(at(8) == at(33))) return 31;
  c.centers = nullptr;
  if (at(3) == at(5) || at(8) == at(9) || !(at(10) == at(40))) return 30;
  return 0;
}
