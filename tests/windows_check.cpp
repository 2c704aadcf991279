// The overlapping windows of csrc/ntk_windows.h, enumerated over lengths,
// window lengths and every halo that the plans accept (L >= Lw / 4): prints
// "layouts long_halos wrong", long_halos counting those with H > L, wrong those
// with a window outside the system, a row not central in exactly one window, or
// a central row nearer than H to a cut end.
#include <cstdio>

#include "ntk_windows.h"

int main() {
  long layouts = 0, long_halos = 0, wrong = 0;
  for (int Lw = 128; Lw <= 512; Lw *= 2)
    for (int H = 2; Lw - 2 * H >= Lw / 4; H += 2)
      for (int n = Lw + 1; n < 6 * Lw; n += Lw < 512 ? 1 : 3) {
        const int L = Lw - 2 * H, P = (n - Lw + H + L - 1) / L + 1;
        ++layouts;
        long_halos += H > L;
        bool ok = P >= 2;
        int row = 0;
        for (int w = 0; w < P && ok; ++w) {
          const ntk::WinRows r = ntk::window_of(n, Lw, L, H, P, w);
          ok = r.start >= 0 && r.start + Lw <= n && r.lo >= 0 && r.hi <= Lw && r.start + r.lo == row && r.hi > r.lo;
          ok = ok && (r.kind == 0 ? r.start == 0 : r.lo >= H) && (r.kind == 2 ? r.start + Lw == n : r.hi <= Lw - H);
          row = r.start + r.hi;
        }
        wrong += !(ok && row == n);
      }
  std::printf("%ld %ld %ld\n", layouts, long_halos, wrong);
  return 0;
}
