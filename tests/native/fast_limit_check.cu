// Host check, no GPU needed: the fast step's kernels index cells with 32 bits,
// so its launchers refuse fields of 2^31 cells or more before they launch
// anything.
#include <cstdio>

#include "rt_kernels.h"

int main() {
  rt::Dims d{};
  const int n[6] = {64, 64, 64, 16, 16, 32};   // 2^31
  long long s = 1;
  for (int a = 0; a < 6; a++) {
    d.n[a] = n[a];
    d.s[a] = s;
    s *= n[a];
  }
  d.ncell = s;
  d.nvol3 = d.s[3];
  d.nspec = s / d.nvol3;
  int launches = -1;
  const long long off[6] = {0, 0, 0, 0, 0, 0};
  cudaError_t e = rt::launch_fast_prepare(d, rt::Grid{}, 1.0, rt::FastFields{}, nullptr, off, &launches, nullptr);
  if (e != cudaErrorInvalidValue || launches != 0) {
    printf("prepare: %s, %d launches\n", cudaGetErrorName(e), launches);
    return 1;
  }
  e = rt::launch_step_fast(d, rt::FastFields{}, nullptr, nullptr, &launches, nullptr);
  if (e != cudaErrorInvalidValue || launches != 0) {
    printf("step: %s, %d launches\n", cudaGetErrorName(e), launches);
    return 1;
  }
  if (!rt::fast_ok(d)) {
    d.ncell -= 1;
    if (rt::fast_ok(d)) return 0;
  }
  printf("fast_ok\n");
  return 1;
}
