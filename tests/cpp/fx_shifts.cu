// Values of the fixed-point shifts (mwf_fx.cuh) for tests/test_fixed_point_shifts.py: reads lines "x r", writes
// fx_down(x, r).
#include <cstdio>

#include "mwf_fx.cuh"

int main() {
  long long x;
  int r;
  while (scanf("%lld %d", &x, &r) == 2) printf("%lld\n", (long long)mwf::fx_down(x, r));
  return 0;
}
