// Host check, no GPU needed: the members of a binary32 batch are split over
// launches by what a launch's arguments hold and by the CTAs a grid may have.
#include <cstdio>
#include <vector>

#include "rt_kernels.h"
#include "rt_step.cuh"

static rt::StepArgs<float> field(int nx, int ny, int nz, int nk, int nl, int nm) {
  rt::StepArgs<float> S{};
  const int n[6] = {nx, ny, nz, nk, nl, nm};
  long long s = 1;
  for (int a = 0; a < 6; a++) {
    S.d.n[a] = n[a];
    S.d.s[a] = s;
    s *= n[a];
  }
  S.d.ncell = s;
  S.d.nvol3 = S.d.s[3];
  S.d.nspec = s / S.d.nvol3;
  return S;
}

static int fails = 0;
static void expect(const char* what, const std::vector<rt::StepArgs<float>>& S, int take, int launches) {
  const int n = (int)S.size(), t = rt::march_batch_take(S.data(), n), l = rt::march_batch_launches(S.data(), n);
  if (t == take && l == launches) return;
  printf("%s: %d of %d in the first launch (%d), %d launches (%d)\n", what, t, n, take, l, launches);
  fails++;
}

int main() {
  const auto small = field(8, 8, 8, 8, 8, 8);
  expect("one", {small}, 1, 1);
  expect("80", std::vector<rt::StepArgs<float>>(80, small), 80, 1);
  expect("81", std::vector<rt::StepArgs<float>>(81, small), 80, 2);
  expect("161", std::vector<rt::StepArgs<float>>(161, small), 80, 3);
  const auto large = field(32, 32, 32, 32, 32, 32);
  expect("large", {large, large, large, large, large}, 5, 1);
  // a CTA per (l,m): 2^30 of them in a field
  const auto point = field(1, 1, 1, 1, 32768, 32768), half = field(1, 1, 1, 1, 16384, 32768);
  expect("point", {point}, 1, 1);
  expect("points", {point, point, point}, 1, 3);
  expect("halves", {half, half, half, half, half}, 3, 2);
  expect("mixed", {small, point, small, point, small}, 3, 2);
  return fails;
}
