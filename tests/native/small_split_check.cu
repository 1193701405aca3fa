// Host check of the one-launch binary64 step's split into CTAs: over shapes of
// up to 65,536 cells and GPUs of 1 to 200 multiprocessors the face lists of a
// CTA fit the 48 KB of shared memory that a launch may have without raising
// the kernel's limit, beside the kernel's own few bytes, and the CTAs are one
// per multiprocessor wherever that fits.
#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "rt_kernels.h"

int main() {
  srand(7);
  long long seen = 0;
  for (int t = 0; t < 20000; t++) {
    rt::Dims d{};
    long long s = 1;
    for (int a = 0; a < 6; a++) {
      const long long room = 65536 / s;
      int n = rand() % 3 == 0 ? 1 : 1 + (int)(rand() % (a == 5 ? room : std::min<long long>(room, 1 + rand() % 40)));
      if (t < 200 && a == t % 6) n = (int)room;   // the largest fields
      d.n[a] = n;
      d.s[a] = s;
      s *= n;
    }
    d.ncell = s;
    d.lower_refl = rand() & 1;
    for (int sms = 1; sms <= 200; sms += 1 + rand() % 9) {
      const int C = rt::exact_small_cells(d, sms);
      long long jobs = d.n[2] > 1 && d.lower_refl ? C : 0, most = 1;
      for (int a = 0; a < 6; a++)
        if (d.n[a] > 1) jobs += C + std::min<long long>(C, d.s[a]), most += 2;
      const bool even = C == (d.ncell + sms - 1) / sms;
      if (C < 1 || jobs * 8 + 64 > 48 * 1024 || (!even && (C + 1) * most * 8 + 64 <= 48 * 1024) ||
          (sms >= 139 && !even)) {
        printf("%d %d %d %d %d %d on %d: C %d, %lld slots\n", d.n[0], d.n[1], d.n[2], d.n[3], d.n[4], d.n[5], sms, C, jobs);
        return 1;
      }
      seen++;
    }
  }
  printf("%lld splits\n", seen);
  return 0;
}
