// ntk_chunk_f64.cu -- FP64 solves of few systems, T threads per system.
//
// One thread per system (ntk_solve_f64.cu) needs the fewest FP64
// instructions, but a 256 x 256 field has 256 systems and an ADI sweep of a
// 2048 x 2048 one 2046: 8 and 64 warps for 152 SMs, each walking 2 n
// dependent rows through global memory.  Here a CTA keeps S whole systems in
// shared memory and gives every system T threads of C consecutive rows:
//   forward   y_i = d_i - l_i y_{i-1} over the chunk from zero, for its end
//             value only; the chunks' carries are an exact affine scan over the
//             T ends (log2 T steps through shared memory, the products of the
//             multipliers tabulated on the host: one FMA a step); then the
//             sweep again from the carry, in place
//   backward  x_i = g_i y_i - (c_i / u_i) x_{i+1} likewise from the other end,
//             the second time straight to the results
// Sweeping twice costs an FMA a row, as adding the carries' responses to the
// rows of one sweep would, and rounds as the sequential sweeps do (2046 systems
// of 2048 rows: error against 64 bits 1.07e-16, with added responses 1.34e-16;
// 1 - 7% slower).  Nothing is truncated, so any matrix that factors is served,
// at 5 operations a row (+1 for the compact difference) against 3 (+1): the
// FP64 pipe (one warp instruction per ~76 clocks and sub-partition) bounds both
// kernels, and this one wins where one thread per system leaves the pipe idle
// (chunk_f64_pick).
// Rows stay in shared memory between the sweeps, not in registers, so a
// chunk may be long: the scans' 2 log2 T instructions a thread are spread
// over C rows.  A contiguous system's chunks lie C + 1 doubles apart (odd: the
// threads of a half-warp touch 16 different bank pairs); strided systems lie
// side by side, S to a row, and a half-warp reads whole row segments.
// The scaling g y, off the dependent chain, runs on the integer pipes
// (ntk_soft_f64.cuh), which leaves 4 (+1) FP64 instructions a row.
// Threads whose chunks see bitwise equal factors share one table (the head's
// few chunks before the pivots reach their fixed point, the interior, the
// tail), so the factors stay in L1.
// Measured, one thread per system against this kernel: 2046 systems of 2048
// rows 754 -> 47 us (67 with g y on the FP64 pipe; the pipe alone: 34 us),
// compact derivative of a 256 x 256 field 97 -> 8.2 us (most of it the call).
// A system with a value that is not finite, or that overflows on the way, is
// solved again row by row, so that inf and nan spread exactly as in the
// one-thread sweeps: from its input where the first sweeps or the scans show
// it (before anything is stored), from the rows' g y where only the second
// backward sweep, with the carry, goes beyond the range.  A nan in the input
// reaches every row of a sequential solve, so such systems (masked or diverged
// fields) are filled instead: 32768 compact lines of 2048 rows, each with a
// nan, 17500 -> 1330 us (one thread per system: 1110).
#include "ntk_chunk_f64.h"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "ntk_device.cuh"

namespace ntk {

namespace {

constexpr int RB = 4;  // rows per batch of a sweep: their loads are issued ahead of the dependent FMAs

struct ChunkParams {
  int n, S, T, C, P, steps, shift;  // P: pitch of a contiguous system; shift: log2 S (strided) or log2 T
  unsigned invC;       // ceil(2^32 / C): r / C = umulhi(r, invC) for the rows of a system
  const double* tab;      // [ncls][2][C]: -l, -w
  const double* g;        // [ncls][C]
  const SoftFactor* sg;   // the same, prepared
  const double* scan;  // [2][steps][T]
  const int* cls;      // [T]
  TablesF64 plain;
};

__device__ __forceinline__ bool finite(double x) { return ((unsigned)__double2hiint(x) & 0x7ff00000u) != 0x7ff00000u; }

// One system row by row from global memory, four rows' loads ahead of their
// dependent FMAs, the forward values parked in out (which may be in: the
// compact difference keeps its neighbours in registers).
template <int RHS>
__device__ __noinline__ void plain_system(const double* in, double* out, long long base, long long es, int n,
                                          long long s, const RhsParams& rp, const TablesF64& t) {
  constexpr int B = 4;
  const double* a = in + base;
  double* o = out + base;
  double y = 0.0, fm = 0.0, fc = a[0], d0 = fc, dn = 0.0;
  if (RHS == RHS_COMPACT) {
    const double* e = a + (long long)(n - 1) * es;
    d0 = rp.sigma0 * ((-5.0 * a[0] + 4.0 * a[es]) + a[2 * es]);
    dn = rp.sigmaN * ((-5.0 * e[0] + 4.0 * e[-es]) + e[-2 * es]);
  }
  if (RHS == RHS_CROSS) {
    d0 = rp.bnd[s * rp.bnd_ss];
    dn = rp.bnd[s * rp.bnd_ss + (long long)(n - 1) * rp.bnd_es];
  }
  for (int i0 = 0; i0 < n; i0 += B) {
    double d[B], l[B];  // compact: f of the row behind
#pragma unroll
    for (int q = 0; q < B; ++q) {
      const int i = i0 + q;
      const double* p = a + (long long)i * es;
      d[q] = 0.0;
      l[q] = i < n ? t.l[i] : 0.0;
      if (RHS == RHS_COMPACT) {
        if (i < n - 1) d[q] = p[es];
      } else if (RHS == RHS_CROSS) {
        if (i > 0 && i < n - 1)
          d[q] = rp.center == 0.0 ? -p[-rp.cs] - p[rp.cs]
                                  : fma(rp.top, p[rp.cs], fma(rp.center, p[0], rp.bottom * p[-rp.cs]));
      } else {
        if (i < n) d[q] = p[0];
      }
    }
#pragma unroll
    for (int q = 0; q < B; ++q) {
      const int i = i0 + q;
      if (i >= n) break;
      double r = d[q];
      if (RHS == RHS_COMPACT) {
        r = d[q] - fm;
        fm = fc;
        fc = d[q];
      }
      if (RHS != RHS_IDENTITY && i == n - 1) r = dn;
      if (RHS != RHS_IDENTITY && i == 0) r = d0;
      y = i == 0 ? r : fma(-l[q], y, r);
      o[(long long)i * es] = y;
    }
  }
  double x = t.g[n - 1] * y;
  o[(long long)(n - 1) * es] = x;
  for (int i0 = n - 2; i0 >= 0; i0 -= B) {
    double e[B], g[B], w[B];
#pragma unroll
    for (int q = 0; q < B; ++q) {
      const int i = max(i0 - q, 0);
      e[q] = o[(long long)i * es];
      g[q] = t.g[i];
      w[q] = t.w[i];
    }
#pragma unroll
    for (int q = 0; q < B; ++q) {
      if (i0 - q < 0) break;
      x = fma(-w[q], x, g[q] * e[q]);
      o[(long long)(i0 - q) * es] = x;
    }
  }
}

// Whether rows t, t + T .. of a system show that its sequential solve meets a
// nan in the forward sweep: a right-hand side that is a nan, or an infinite
// f_i, 2 <= i <= n - 3, of a compact difference (rows i - 1 and i + 1 then hold
// infinities of opposite signs, and y_{i+1} is inf - inf whatever the sign of
// the multipliers).
template <int RHS>
__device__ __noinline__ bool meets_nan(const double* a, long long es, int n, int t, int T, long long s,
                                       const RhsParams& rp) {
  auto nan = [](double x) { return ((uint64_t)__double_as_longlong(x) & ~(1ull << 63)) > 0x7ffull << 52; };
  bool seen = false;
#pragma unroll 1
  for (int i = t; i < n && !seen; i += T) {
    const double* q = a + (long long)i * es;
    if (RHS == RHS_COMPACT)
      seen = nan(q[0]) || (i > 1 && i < n - 2 && !finite(q[0]));
    else if (RHS == RHS_CROSS)
      seen = i == 0 || i == n - 1 ? nan(rp.bnd[s * rp.bnd_ss + (long long)i * rp.bnd_es])
                                  : nan(q[-rp.cs]) || nan(q[rp.cs]) || (rp.center != 0.0 && nan(q[0]));
    else
      seen = nan(q[0]);
  }
  return seen;
}

template <int RHS, bool STRIDED>
__global__ void __launch_bounds__(512, 2) chunk_f64_kernel(const double* in, double* out, Batch b,
                                                        const __grid_constant__ RhsParams rp,
                                                        const __grid_constant__ ChunkParams c) {
  extern __shared__ __align__(16) double smem[];
  const int nt = c.S * c.T;
  double* tile = smem;
  double* ex = smem + (STRIDED ? c.S * c.n : c.S * c.P);  // [2][nt]
  const int tid = threadIdx.x;
  const int s = STRIDED ? tid & (c.S - 1) : tid >> c.shift;
  const int t = STRIDED ? tid >> c.shift : tid & (c.T - 1);
  const int xs = STRIDED ? c.S : 1;  // one chunk on in ex
  const int rs = STRIDED ? c.S : 1;  // one row on in the tile
  const long long sys = (long long)blockIdx.x * c.S + s;
  const bool on = sys < b.nsys;
  const long long base = !on ? 0 : b.ni >= b.nsys ? sys * b.is : (sys / b.ni) * b.os + (sys % b.ni) * b.is;
  double* col = tile + (STRIDED ? s : s * c.P);  // row r of this system: col[slot(r)]
  auto slot = [&](int r) { return STRIDED ? r * c.S : r + (int)__umulhi((unsigned)r, c.invC); };

  // ---- stage the system's rows (the ADI stencil is formed on the way) ----
  if (on) {
    const double* src = in + base;
    if (RHS == RHS_CROSS) {
#pragma unroll 4
      for (int r = t; r < c.n; r += c.T) {
        const double* q = src + (long long)r * b.es;
        double v;
        if (r == 0 || r == c.n - 1) v = rp.bnd[sys * rp.bnd_ss + (long long)r * rp.bnd_es];
        else if (rp.center == 0.0) v = -q[-rp.cs] - q[rp.cs];
        else v = fma(rp.top, q[rp.cs], fma(rp.center, q[0], rp.bottom * q[-rp.cs]));
        col[slot(r)] = v;
      }
    } else {
#pragma unroll 4
      for (int r = t; r < c.n; r += c.T) cp_async8(col + slot(r), src + (long long)r * b.es, 8u);
      cp_async_wait_all();
    }
  }
  __syncthreads();

  const int r0 = t * c.C;
  const int len = on ? max(0, min(c.C, c.n - r0)) : 0;
  double* row = col + (STRIDED ? r0 * c.S : t * (c.C + 1));  // row r0 + k: row[k * rs]
  const int cls = __ldg(c.cls + t);
  const double* ml = c.tab + (size_t)cls * 2 * c.C;
  const double* mw = ml + c.C;
  const double* g = c.g + (size_t)cls * c.C;
  const SoftFactor* sg = c.sg + (size_t)cls * c.C;

  // ---- forward over the chunk from zero, for its end value only (the compact
  // difference is left in the rows) ----
  double y = 0.0;
  {
    // the neighbours' edge rows, and the end rows' one-sided stencils
    double fm = 0.0, fr = 0.0, be = 0.0;
    if (RHS == RHS_COMPACT) {
      if (len > 0) {
        fm = r0 > 0 ? col[slot(r0 - 1)] : 0.0;
        fr = r0 + len < c.n ? col[slot(r0 + len)] : 0.0;
        const bool tail = r0 + len == c.n;
        if (r0 == 0 || tail) {
          const int e = tail ? c.n - 1 : 0, d = tail ? -1 : 1;
          be = one_sided(tail ? rp.sigmaN : rp.sigma0, col[slot(e)], col[slot(e + d)], col[slot(e + 2 * d)]);
        }
      }
      __syncthreads();  // the neighbours' edge rows are read before any row is overwritten
    }
    double v[RB];
#pragma unroll
    for (int q = 0; q < RB; ++q) v[q] = q < len ? row[q * rs] : 0.0;
    for (int k = 0; k < len; k += RB) {
      double nx[RB], m[RB];
#pragma unroll
      for (int q = 0; q < RB; ++q) {
        nx[q] = k + RB + q < len ? row[(k + RB + q) * rs] : 0.0;
        m[q] = __ldg(ml + k + q);
      }
#pragma unroll
      for (int q = 0; q < RB; ++q) {
        if (k + q < len) {
          double d = v[q];
          if (RHS == RHS_COMPACT) {
            const double fn = k + q + 1 == len ? fr : q + 1 < RB ? v[(q + 1) % RB] : nx[0];
            d = fn - fm;
            fm = v[q];
            if (r0 + k + q == 0 || r0 + k + q == c.n - 1) d = be;
            row[(k + q) * rs] = d;
          }
          y = fma(m[q], y, d);
        }
      }
#pragma unroll
      for (int q = 0; q < RB; ++q) v[q] = nx[q];
    }
  }
  // ---- inclusive scan of the chunk ends: y becomes the value of the
  // chunk's last row with all carries ----
  int cur = 0;
  ex[tid] = y;
  for (int k = 0; k < c.steps; ++k) {
    const int o = 1 << k;
    __syncthreads();
    if (t >= o) y = fma(__ldg(c.scan + k * c.T + t), ex[cur * nt + tid - o * xs], y);
    cur ^= 1;
    ex[cur * nt + tid] = y;
  }
  __syncthreads();
  const double cin = t > 0 ? ex[cur * nt + tid - xs] : 0.0;

  // ---- forward again from the carry ----
  {
    double z = cin, v[RB];
#pragma unroll
    for (int q = 0; q < RB; ++q) v[q] = q < len ? row[q * rs] : 0.0;
    for (int k = 0; k < len; k += RB) {
      double nx[RB], m[RB];
#pragma unroll
      for (int q = 0; q < RB; ++q) {
        nx[q] = k + RB + q < len ? row[(k + RB + q) * rs] : 0.0;
        m[q] = __ldg(ml + k + q);
      }
#pragma unroll
      for (int q = 0; q < RB; ++q)
        if (k + q < len) {
          z = fma(m[q], z, v[q]);
          row[(k + q) * rs] = z;
        }
#pragma unroll
      for (int q = 0; q < RB; ++q) v[q] = nx[q];
    }
  }
  // ---- backward over the chunk from zero, for its start value; the rows keep
  // g y ----
  double x = 0.0;
  {
    const int k0 = (len - 1) & ~(RB - 1);
    double v[RB];
#pragma unroll
    for (int q = 0; q < RB; ++q) v[q] = len > 0 && k0 + q < len ? row[(k0 + q) * rs] : 0.0;
    for (int k = k0; k >= 0; k -= RB) {
      double nx[RB], gy[RB];
      SoftFactor f[RB];
      bool in_range = true;
#pragma unroll
      for (int q = 0; q < RB; ++q) {
        nx[q] = k >= RB ? row[(k - RB + q) * rs] : 0.0;
        f[q] = load_factor(sg + k + q);
      }
#pragma unroll
      for (int q = 0; q < RB; ++q) {
        in_range = in_range && (k + q >= len || soft_in_range(v[q], f[q], SOFT_SPAN));
        gy[q] = soft_product(v[q], f[q]);
      }
      if (!in_range)
        rare_rows(
            v, gy, [&](int q) { return __ldg(g + k + q); },
            [&](int q) { return k + q >= len || soft_in_range(v[q], load_factor(sg + k + q), SOFT_SPAN); });
#pragma unroll
      for (int q = RB - 1; q >= 0; --q)
        if (k + q < len) {
          x = fma(__ldg(mw + k + q), x, gy[q]);
          row[(k + q) * rs] = gy[q];
        }
#pragma unroll
      for (int q = 0; q < RB; ++q) v[q] = nx[q];
    }
  }
  // ---- the same scan from the other end; the buffer read for cin is left
  // alone until the first barrier ----
  cur ^= 1;
  ex[cur * nt + tid] = x;
  for (int k = 0; k < c.steps; ++k) {
    const int o = 1 << k;
    __syncthreads();
    if (t + o < c.T) x = fma(__ldg(c.scan + (c.steps + k) * c.T + t), ex[cur * nt + tid + o * xs], x);
    cur ^= 1;
    ex[cur * nt + tid] = x;
  }
  __syncthreads();
  const double xin = t < c.T - 1 ? ex[cur * nt + tid + xs] : 0.0;
  // what is not finite after these sweeps and scans, anywhere in the system,
  // has reached row 0
  bool ok = finite(ex[cur * nt + tid - t * xs]);

  // ---- backward again from the carry, results out ----
  bool over = false;  // a row beyond the range with the carry only: it has reached the chunk's first row
  {
    double* dst = out + base + (long long)r0 * b.es;
    const int k0 = (len - 1) & ~(RB - 1);
    double z = xin, v[RB];
#pragma unroll
    for (int q = 0; q < RB; ++q) v[q] = len > 0 && k0 + q < len ? row[(k0 + q) * rs] : 0.0;
    for (int k = k0; k >= 0; k -= RB) {
      double nx[RB], m[RB];
#pragma unroll
      for (int q = 0; q < RB; ++q) {
        nx[q] = k >= RB ? row[(k - RB + q) * rs] : 0.0;
        m[q] = __ldg(mw + k + q);
      }
#pragma unroll
      for (int q = RB - 1; q >= 0; --q)
        if (k + q < len) {
          z = fma(m[q], z, v[q]);
          if (!STRIDED) row[k + q] = z;
          else if (ok) dst[(long long)(k + q) * b.es] = z;
        }
#pragma unroll
      for (int q = 0; q < RB; ++q) v[q] = nx[q];
    }
    over = ok && len > 0 && !finite(z);
  }
  if (__syncthreads_or(over || (on && !ok))) {
    // over: chunks beyond the range; where !ok, threads that see a nan
    if (on && !ok) over = meets_nan<RHS>(in + base, b.es, c.n, t, c.T, sys, rp);
    ex[tid] = over ? 1.0 : 0.0;
    __syncthreads();
    if (on && !ok) {
      for (int j = 0; j < c.T; ++j) over = over || ex[tid + (j - t) * xs] != 0.0;
      double* dst = out + base;
      if (over) {
        const double x = c.plain.g[0] * __longlong_as_double(0x7ff8ll << 48);
        for (int r = t; r < c.n; r += c.T) dst[(long long)r * b.es] = x;
      } else if (t == 0) {
        plain_system<RHS>(in, out, base, b.es, c.n, sys, rp, c.plain);
      }
    } else if (on) {
      for (int j = 0; j < c.T; ++j) over = over || ex[tid + (j - t) * xs] != 0.0;
      if (STRIDED && over && t == 0) {  // the rows still hold g y
        double* dst = out + base;
        double z = col[slot(c.n - 1)];
        dst[(long long)(c.n - 1) * b.es] = z;
        for (int r = c.n - 2; r >= 0; --r) {
          z = fma(-c.plain.w[r], z, col[slot(r)]);
          dst[(long long)r * b.es] = z;
        }
      }
      if (!STRIDED && over) {  // nothing is stored yet
        ok = false;
        if (t == 0) plain_system<RHS>(in, out, base, b.es, c.n, sys, rp, c.plain);
      }
    }
  }
  if (!STRIDED && on && ok) {
    double* dst = out + base;
#pragma unroll 4
    for (int r = t; r < c.n; r += c.T) dst[r] = col[slot(r)];
  }
}

// Pitch of a contiguous system in the tile, in doubles: C + 1, odd, for each
// chunk.
int pitch(const ChunkF64::Cfg& cfg) { return cfg.T * (cfg.C + 1); }
size_t smem_bytes(const ChunkF64::Cfg& cfg, int n, int S, bool strided) {
  const size_t tile = (size_t)S * (strided ? n : pitch(cfg));
  return (tile + 2 * (size_t)S * cfg.T) * sizeof(double);
}

int log2_of(int v) {
  int k = 0;
  while ((1 << k) < v) ++k;
  return k;
}

constexpr size_t SMEM_MAX = 220 * 1024;
constexpr size_t SMEM_SM = 228 * 1024;
constexpr int SMS = 152;
constexpr int MAXT = 256;

template <int RHS, bool STRIDED>
int launch_one(const double* in, double* out, const Batch& b, const RhsParams& rp, const ChunkParams& c, size_t smem,
               cudaStream_t st) {
  auto k = chunk_f64_kernel<RHS, STRIDED>;
  int rc = allow_smem(k, smem, "cudaFuncSetAttribute(chunk_f64_kernel)");
  if (rc) return rc;
  const long long blocks = (b.nsys + c.S - 1) / c.S;
  k<<<(unsigned)blocks, c.S * c.T, smem, st>>>(in, out, b, rp, c);
  return cuda_status(cudaGetLastError(), "chunk_f64_kernel");
}

}  // namespace

std::vector<double> ChunkF64::init(int n_, const double* l, const double* u, const double* w) {
  n = n_;
  std::vector<double> tab;
  for (int T = 4; T <= MAXT; T *= 2) {
    Cfg f;
    f.T = T;
    f.C = ((n + T - 1) / T + RB - 1) / RB * RB;
    if (n < 5 * T || smem_bytes(f, n, std::max(1, 32 / T), false) > SMEM_MAX) continue;
    f.tab = tab.size();
    f.g = g_count;
    std::vector<double> Phi(T, 0.0), Psi(T, 0.0);
    std::vector<int> cls(T);
    for (int t = 0; t < T; ++t) {
      const int r0 = t * f.C, len = std::max(0, std::min(f.C, n - r0));
      int id = -1;  // a chunk seen before with bitwise equal factors in all rows
      for (int j = 0; j < f.ncls && id < 0; ++j) {
        const int q0 = f.rep[j] * f.C, qlen = std::max(0, std::min(f.C, n - q0));
        const size_t bytes = sizeof(double) * len;
        if (qlen == len && (len == 0 || (std::memcmp(l + q0, l + r0, bytes) == 0 &&
                                         std::memcmp(u + q0, u + r0, bytes) == 0 &&
                                         std::memcmp(w + q0, w + r0, bytes) == 0)))
          id = j;
      }
      if (id < 0) {
        id = f.ncls++;
        f.rep.push_back(t);
        // its columns; rows past the system's end hold zeros
        const size_t at = tab.size();
        tab.resize(at + 2 * (size_t)f.C, 0.0);
        double* q = tab.data() + at;
        double pl = 1.0, pw = 1.0;  // the responses of its end (start) to the carry entering it
        for (int k = 0; k < len; ++k) {
          q[k] = -l[r0 + k];
          q[f.C + k] = -w[r0 + k];
          pl *= q[k];
        }
        for (int k = len - 1; k >= 0; --k) pw *= q[f.C + k];
        Phi[t] = len ? pl : 0.0;
        Psi[t] = len ? pw : 0.0;
      } else {
        Phi[t] = Phi[f.rep[id]];
        Psi[t] = Psi[f.rep[id]];
      }
      cls[t] = id;
    }
    // scan multipliers: step k combines chunk t with the result of chunk
    // t - 2^k (t + 2^k from the other end)
    f.scan = tab.size();
    const int steps = log2_of(T);
    tab.resize(tab.size() + 2 * (size_t)steps * T, 0.0);
    double* sf = tab.data() + f.scan;
    double* sb = sf + (size_t)steps * T;
    for (int k = 0; k < steps; ++k)
      for (int t = 0; t < T; ++t) {
        const int o = 1 << k >> 1;
        if (k == 0) sf[t] = Phi[t], sb[t] = Psi[t];
        else {
          sf[k * T + t] = t >= o ? sf[(k - 1) * T + t] * sf[(k - 1) * T + t - o] : 0.0;
          sb[k * T + t] = t + o < T ? sb[(k - 1) * T + t] * sb[(k - 1) * T + t + o] : 0.0;
        }
      }
    f.cls = tab.size();
    tab.resize(tab.size() + (T + 1) / 2, 0.0);
    std::memcpy(tab.data() + f.cls, cls.data(), sizeof(int) * T);
    g_count += (size_t)f.ncls * f.C;
    cfgs.push_back(f);
  }
  return tab;
}

bool ChunkF64::serves_both_layouts() const {
  for (const Cfg& f : cfgs)  // contiguous systems fit every configuration kept by init
    if (4 * f.T >= 32 && smem_bytes(f, n, 4, true) <= SMEM_MAX) return true;
  return false;
}

void ChunkF64::g_rows(const double* g, double* out) const {
  SoftFactor* sg = reinterpret_cast<SoftFactor*>(out);
  double* plain = out + 2 * g_count;
  for (const Cfg& f : cfgs)
    for (int j = 0; j < f.ncls; ++j)
      for (int k = 0; k < f.C; ++k) {
        const int r = f.rep[j] * f.C + k;
        const size_t at = f.g + (size_t)j * f.C + k;
        plain[at] = r < n ? g[r] : 0.0;
        sg[at] = soft_factor(plain[at], SOFT_SPAN);
      }
}

// Costs in FP64 warp instructions of one sub-partition (~76 clocks each).
// Chunks: C (4 + extra) row instructions and the two scans for each CTA of an
// SM's share, plus twice the length of one CTA's dependent chain (the first
// CTAs fill the pipe and the last ones drain it; more where a second wave
// starts late); row segments of strided systems below 128 bytes cost up to an
// eighth.  One thread per system: n (2 + extra) instructions a warp times the
// measured distance from the pipe's rate, which falls as more warps hide each
// other's loads (contiguous systems, whose tiles take most of the time: as
// measured with one instruction more).  Measured, us, one thread a system
// against chunks: 512 rows contiguous, 4096 systems 161 : 23, 16384 163 : 75,
// 65536 291 : 273, compact with 262144 1143 : 1272; strided compact, 13472
// systems of 333 rows 79 : 56, 79990 207 : 275.
const ChunkF64::Cfg* chunk_f64_pick(const ChunkF64& c, const Batch& b, int rhs, int* S, bool always) {
  const bool strided = b.es != 1;
  const int extra = rhs == RHS_COMPACT ? 1 : 0;
  const ChunkF64::Cfg* best = nullptr;
  double best_cost = 0.0;
  for (const ChunkF64::Cfg& f : c.cfgs)
    for (int s = strided ? 4 : std::max(1, 32 / f.T); s <= 16; s *= 2) {
      const int nt = s * f.T;
      const size_t smem = smem_bytes(f, c.n, s, strided);
      const long long ctas = (b.nsys + s - 1) / s;
      if (nt < 32 || nt > 512 || smem > SMEM_MAX || ctas > 0x7fffffffLL) continue;
      const double per_sm = std::max(1.0, (double)ctas / SMS + 0.5);
      const double resident = std::min<double>(std::min(32, 2048 / nt), SMEM_SM / (smem + 1024));
      const double work = f.C * (4 + extra) + 2 * log2_of(f.T) + 2;
      const double cost = (work * per_sm * nt / 128 + (work + 12) * (per_sm > resident ? 2.5 : 2.0)) *
                          (!strided || s == 16 ? 1.0 : s == 8 ? 1.05 : 1.12);
      if (!best || cost < best_cost) {
        best_cost = cost;
        best = &f;
        *S = s;
      }
    }
  if (always) return best;
  const double load = std::ceil((double)((b.nsys + 31) / 32) / (4 * SMS));
  const double plain = strided ? (2 + extra) * (0.92 + 1.2 / load) : (3 + extra) * (0.95 + 1.5 / load);
  return best && best_cost < load * c.n * plain ? best : nullptr;
}

int launch_chunk_f64(const ChunkF64& cf, const ChunkF64::Cfg& cfg, int S, const double* in, double* out,
                     const Batch& b, const RhsParams& rp, const TablesF64& t, cudaStream_t st) {
  const bool strided = b.es != 1;
  ChunkParams c;
  c.n = cf.n;
  c.S = S;
  c.T = cfg.T;
  c.C = cfg.C;
  c.P = pitch(cfg);
  c.invC = 0xffffffffu / (unsigned)cfg.C + 1u;
  c.steps = log2_of(cfg.T);
  c.shift = strided ? log2_of(S) : c.steps;
  c.tab = cf.d_tab + cfg.tab;
  const double* rows = t.g + ChunkF64::g_offset(cf.n);
  c.sg = reinterpret_cast<const SoftFactor*>(rows) + cfg.g;
  c.g = rows + 2 * cf.g_count + cfg.g;
  c.scan = cf.d_tab + cfg.scan;
  c.cls = reinterpret_cast<const int*>(cf.d_tab + cfg.cls);
  c.plain = t;
  const size_t smem = smem_bytes(cfg, cf.n, S, strided);
  switch (rp.kind) {
    case RHS_COMPACT:
      return strided ? launch_one<RHS_COMPACT, true>(in, out, b, rp, c, smem, st)
                     : launch_one<RHS_COMPACT, false>(in, out, b, rp, c, smem, st);
    case RHS_CROSS:
      return strided ? launch_one<RHS_CROSS, true>(in, out, b, rp, c, smem, st)
                     : launch_one<RHS_CROSS, false>(in, out, b, rp, c, smem, st);
    default:
      return strided ? launch_one<RHS_IDENTITY, true>(in, out, b, rp, c, smem, st)
                     : launch_one<RHS_IDENTITY, false>(in, out, b, rp, c, smem, st);
  }
}

}  // namespace ntk
