// The windows of ntk_r2n.cu, enumerated: prints "layouts accepted wrong", wrong
// counting accepted ones whose windows are not what the kernel takes them for
// (all but the last full, consecutive ones overlapping by two halos, every row
// central in exactly one).
#include <cstdio>

#include "ntk_r2n_windows.h"

int main() {
  long layouts = 0, accepted = 0, wrong = 0;
  for (int H = 4; H <= 40; H += 2)
    for (int sg = 8; sg <= 16; sg *= 2)
      for (int n = 96; n < 60000; n += n < 8000 ? 1 : 37) {
        const ntk::r2n::Windows y = ntk::r2n::choose_windows(n, H, sg);
        if (!y.P) continue;
        ++layouts;
        if (!ntk::r2n::last_window_ok(y)) continue;
        ++accepted;
        bool ok = y.Wr % 16 == 0 && y.Wr <= 512 && y.Wr / 16 * sg <= 512;
        int row = 0;  // the next row to be stored
        for (int w = 0; w < y.P; ++w) {
          const int start = w * (y.Wr - 2 * y.H), nv = n - start < y.Wr ? n - start : y.Wr;
          const int lo = w == 0 ? 0 : y.H, hi = w == y.P - 1 ? nv : y.Wr - y.H;
          ok = ok && (w == y.P - 1 ? nv == y.last : nv == y.Wr) && start + lo == row && hi > lo;
          row = start + hi;
        }
        wrong += !(ok && row == n);
      }
  std::printf("%ld %ld %ld\n", layouts, accepted, wrong);
  return 0;
}
