// ntk_windows.h -- overlapping windows of one system: Lw rows each, L = Lw -
// 2 H central ones written back, H of halo beside them (ntk_adi_refine.cu,
// ntk_adi_f64.cu, ntk_long_refine.cu).  Plain C++ for the host too:
// tests/windows_check.cpp enumerates it.
#pragma once

#ifdef __CUDACC__
#define WINDOWS_HD __host__ __device__ __forceinline__
#else
#define WINDOWS_HD inline
#endif

namespace ntk {

// Window w: first row, rows written back [lo, hi) (counted from it), and its
// kind (the matrix and tables it uses): 0 begins with the system's first row,
// 1 is cut at both ends, 2 ends with the system's last row, 3 is the system.
struct WinRows {
  int start, lo, hi, kind;
};

// Windows of a system of n > Lw rows; P = ceil((n - Lw + H) / L) + 1, at least 2.
WINDOWS_HD WinRows window_of(int n, int Lw, int L, int H, int P, int w) {
  if (w == P - 1) return {n - Lw, w * L - (n - Lw), Lw, 2};
  // where the halo is longer than the central rows (slow decay), the second
  // window's would begin before the system: it begins with the system instead,
  // its central rows still H or more from its cut end
  const int start = w * L - H;
  if (start <= 0) return {0, w * L, w * L + L, 0};
  return {start, H, H + L, 1};
}

}  // namespace ntk
