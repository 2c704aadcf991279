// ntk_r2n_windows.h -- how ntk_r2n.cu cuts systems into windows.  Plain C++:
// tests/r2n_windows_check.cpp enumerates it on the host.
#pragma once
#include <algorithm>

namespace ntk {
namespace r2n {

constexpr int MAX_NC = 32;  // 16-row chunks of a window

struct Windows {
  int P = 0, Wr = 0, H = 0;  // windows (0: none found), rows of each, halo (0 with one window)
  int last = 0;              // rows of the last window
};

// Windows of n rows each overlapping by H-row halos, sg systems per CTA: the
// fewest rows solved for the share of the 1024 threads (64 registers each)
// that whole CTAs can fill; several small CTAs overlap their phases better
// than two large ones.
inline Windows choose_windows(int n, int H, int sg) {
  Windows y;
  double best = 0.0;
  for (int P = 1; P <= 4096; ++P) {
    const int Wr = (int)(((long long)n + 2LL * H * (P - 1) + 16 * P - 1) / (16 * P)) * 16;
    if (P > 1 && Wr < 4 * H + 64) break;  // halos would be half of the work
    if (Wr > 16 * MAX_NC) continue;
    const int threads = Wr / 16 * sg, ctas = std::min(1024 / threads, 32);
    const double cost = (double)P * Wr / (ctas * threads * (1.0 - 0.1 / ctas));
    if (best == 0.0 || cost < best) {
      best = cost;
      y.P = P;
      y.Wr = Wr;
    }
    if (P > 1 && P * (long long)(512 - 2 * H) > 4LL * n) break;
  }
  y.H = y.P > 1 ? H : 0;
  y.last = n - (y.P - 1) * (y.Wr - 2 * y.H);
  return y;
}

// The last window holds two chunks with tables of their own and an interior
// one, and reaches over both halos: every window before it is then full.
inline bool last_window_ok(const Windows& y) { return y.last >= std::max(48, 2 * y.H) && y.last <= y.Wr; }

}  // namespace r2n
}  // namespace ntk
