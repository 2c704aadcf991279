// ntk_r2n.cu -- FP32 + refinement for systems of any length: the paired-chunk
// arithmetic of ntk_r2.cuh (16 rows a thread as 8 packed FP32x2 pairs) with
// as many chunks as the system has.
//
// The kernels of ntk_r2.cu need n = 512.  The chunked kernel that served
// every other length (ntk_refine.cuh) gives a system one warp of 4, 8, 16 or
// 32 rows a lane: 385 rows pay for 512, 700 for 1024 (with a register file's
// worth of rows per lane), 240 for 256 in 8-row chunks whose carries need
// scans, at 110-124 instructions a row.  Here a CTA takes 16 systems (8
// contiguous ones) and one thread per system and 16-row chunk, nc = ceil(n / 16) chunks: nothing is
// paid for beyond the last chunk.  Systems longer than 512 rows are cut into
// P equal windows of Wr rows overlapping by H-row halos (as in
// ntk_long_refine.cu: the product of the multipliers over H rows is below
// 2^-56), P chosen for the fewest rows solved per resident thread.
//
//  * Factors.  The interior chunks use the constants of the Toeplitz factors
//    (kernel parameters, as in ntk_r2.cu).  The first chunk (pivots not yet
//    converged) and the last one (the last row, and identity rows beyond it)
//    have tables of their own in shared memory, used by the first warp and the
//    warp of the last chunk only, so no end corrections are needed and the
//    last row may sit anywhere in its chunk.
//  * Tiles.  Strided systems: [row][16] in shared memory, by TMA boxes where
//    the layout allows tensor maps, else 8-byte cp.async; results straight
//    from registers, 128 bytes a half-warp.  Contiguous systems: one after
//    the other, Wr + 2 doubles apart, by one bulk copy each way per system
//    where 16-byte alignment allows (else cp.async and plain stores, lanes
//    walking a system's rows); the solve's accesses, two rows (16 bytes) a
//    thread and eight systems a quarter-warp, are free of bank conflicts.
//  * In place, P > 1: a window must not overwrite rows that its neighbours
//    still read as halos.  A CTA solves all windows of its systems in order
//    and keeps the H rows that the next window shares in a side buffer
//    (ntk_long_refine.cu copies the whole input first: 82 of 281 us for 16384
//    systems of 2048 rows).
// Measured against the chunked kernels, us: derivatives of a 240 x 385 x 700
// field along x (700 rows) 814 -> 304, y (385) 448 -> 341, z (240) 439 -> 277;
// 16384 systems of 2048 rows in place 281 -> 185, 65536 of 100 rows 60 -> 37,
// 2600 of 300 rows 12.6 -> 10.5.  Smaller batches stay with the chunked
// kernels (r2n_serves).
#include "ntk_r2n.h"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "ntk_device.cuh"
#include "ntk_r2_host.h"
#include "ntk_r2_tma.cuh"
#include "ntk_r2n_windows.h"

namespace ntk {
namespace r2n {

using namespace r2;

// systems per CTA: strided 16 (128-byte row segments); contiguous 8, which
// fills an SM's threads better (384 rows: 5 CTAs of 192 threads, not 2 of 384)
template <bool CONTIG>
constexpr int group_size = CONTIG ? 8 : 16;
// exchange values, [chunk][value][system] floats: a neighbour's are a constant
// distance away, and the chunks of a warp use different banks
enum { X_E1 = 0, X_S1, X_A0, X_B0, X_B7, X_E2, X_S2, X_COUNT };

// Factors of one chunk as pairs (row k, row k + 8).
struct Tab {
  float2 nl[8], g[8], nw[8], phi[8], psi[8];
};
// One window kind: its first and last chunk, its end rows (a, b, c).
struct Kind {
  Tab head, tail;
  DWc hd[3], td[3];
};
enum { FIRST = 0, MIDDLE, LAST, WHOLE, KINDS };
struct Tables {
  Tab plain;  // an interior chunk
  Kind kind[KINDS];
};

struct Geom {
  int n, Wr, nc, H, P;  // rows, window rows, its chunks, halo, windows
  int ni;               // systems per plane
  int gpp;              // groups per plane
  int boxr;             // strided: rows of a TMA box (0: cp.async staging)
  int bulk;             // contiguous: bulk copies (else cp.async staging, plain stores)
  int pf;               // prefetch distance in CTAs (0: none)
  long long is, os, es;
};

// ---------------------------------------------------------------------------
// chunk arithmetic with the factors of a provider: the kernel's constants, or
// a chunk's table (functions as in ntk_r2.cuh)
// ---------------------------------------------------------------------------
struct ByConst {
  const Consts& c;
  __device__ __forceinline__ float2 nl(int) const { return c.nl; }
  __device__ __forceinline__ float2 g(int) const { return c.g; }
  __device__ __forceinline__ float2 nw(int) const { return c.nw; }
  __device__ __forceinline__ float2 phi(int k) const { return c.phi[k]; }
  __device__ __forceinline__ float2 psi(int k) const { return c.psi[k]; }
};
struct ByTab {
  const Tab* t;
  __device__ __forceinline__ float2 nl(int k) const { return t->nl[k]; }
  __device__ __forceinline__ float2 g(int k) const { return t->g[k]; }
  __device__ __forceinline__ float2 nw(int k) const { return t->nw[k]; }
  __device__ __forceinline__ float2 phi(int k) const { return t->phi[k]; }
  __device__ __forceinline__ float2 psi(int k) const { return t->psi[k]; }
};
template <class F>
__device__ __forceinline__ float forward(float2 (&v)[8], const F& f) {
  float2 y = v[0];
#pragma unroll
  for (int k = 1; k < 8; ++k) {
    y = ffma2(f.nl(k), y, v[k]);
    v[k] = y;
  }
  return fma_(f.phi(7).y, v[7].x, v[7].y);
}
// Returns the chunk's start value without the carry entering at its end.
template <class F>
__device__ __forceinline__ float backward(float2 (&v)[8], float CA, const F& f) {
  const float CB = fma_(f.phi(7).x, CA, v[7].x);
  const float2 C = pair(CA, CB);
  float2 x = fmul2(f.g(7), ffma2(f.phi(7), C, v[7]));
  v[7] = x;
#pragma unroll
  for (int k = 6; k >= 0; --k) {
    const float2 y = ffma2(f.phi(k), C, v[k]);
    x = ffma2(f.nw(k), x, fmul2(f.g(k), y));
    v[k] = x;
  }
  return fma_(f.psi(0).x, v[0].y, v[0].x);
}
template <class F>
__device__ __forceinline__ void carry_in(float2 (&v)[8], float XB, const F& f) {
  const float2 X = pair(fma_(f.psi(0).y, XB, v[0].y), XB);
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = ffma2(f.psi(k), X, v[k]);
}

// ---------------------------------------------------------------------------
// the kernel
// ---------------------------------------------------------------------------
// Doubles of the tile: strided [row][16], contiguous [8][Wr + 2].
template <bool CONTIG>
__host__ __device__ constexpr size_t tile_elems(int Wr) {
  return (size_t)group_size<CONTIG> * (CONTIG ? Wr + 2 : Wr);
}
template <bool CONTIG>
__host__ __device__ constexpr size_t smem_of(int Wr, int nc, int stash_rows) {
  return 128 + (tile_elems<CONTIG>(Wr) + (size_t)stash_rows * group_size<CONTIG>)*8 +
         (size_t)X_COUNT * nc * group_size<CONTIG> * 4 + 3 * sizeof(Tab) + 16;
}

// Untiled bulk copies (both addresses 16-byte aligned, whole 16-byte units).
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void bulk_store(void* dst, const void* src, unsigned bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(src)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_prefetch_l2(const void* src, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

template <int RHS, bool CONTIG, bool GEN, bool SEQ>
__global__ void __launch_bounds__(512, 2)
    r2n_kernel(const __grid_constant__ CUtensorMap tin, const double* in, double* out, const __grid_constant__ Geom g,
               const __grid_constant__ Args a, const Tables* __restrict__ tables) {
  extern __shared__ unsigned char smem_raw[];
  // row r of a system: col[r * RS]; contiguous systems lie Wr + 2 doubles
  // apart, so the 16-byte accesses of a quarter-warp (eight systems, the same
  // two rows) touch all 32 banks
  constexpr int SG = group_size<CONTIG>;
  constexpr int RS = CONTIG ? 1 : SG;
  double* tile = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
  double* stash = tile + tile_elems<CONTIG>(g.Wr);  // [H][SG], SEQ
  float* xch = reinterpret_cast<float*>(stash + (SEQ ? (size_t)g.H * SG : 0));
  Tab* tabs = reinterpret_cast<Tab*>(xch + (size_t)X_COUNT * g.nc * SG);  // head, tail, interior
  uint64_t* bar = reinterpret_cast<uint64_t*>(tabs + 3);
  const Consts& K = a.k;
  const int t = threadIdx.x, nt = blockDim.x;
  const int s = t & (SG - 1), c = t / SG;
  const int r0 = ROWS * c;
  const int grp = SEQ ? (int)blockIdx.x : (int)(blockIdx.x / g.P);
  const int plane = grp / g.gpp;
  const int x0 = (grp - plane * g.gpp) * SG;
  const int live = min(SG, g.ni - x0);  // systems of this group
  const long long base = (long long)plane * g.os + (long long)x0 * g.is;
  float* xc = xch + c * (X_COUNT * SG) + s;
  auto X = [&](int which, int d) -> float& { return xc[(d * X_COUNT + which) * SG]; };  // chunk c + d
  double* col = tile + (CONTIG ? s * (g.Wr + 2) : s);
  const long long mine = base + (long long)s * g.is;  // this system's row 0
  if (t == 0) mbar_init(bar, 1);

  int w = SEQ ? 0 : (int)(blockIdx.x - grp * g.P);
  int old_kind = -1;
  unsigned rmax = 0, phase = 0;
  for (;;) {
    const int start = w * (g.Wr - 2 * g.H);
    const int nv = min(g.Wr, g.n - start);  // rows of the system in this window
    const int lo = w == 0 ? 0 : g.H, hi = w == g.P - 1 ? nv : g.Wr - g.H;
    const int last = (nv - 1) >> 4, kt = (nv - 1) & 15;  // the last row's chunk and place
    const int kind = g.P == 1 ? WHOLE : w == 0 ? FIRST : w == g.P - 1 ? LAST : MIDDLE;
    if (kind != old_kind) {
      const float* th = reinterpret_cast<const float*>(&tables->kind[kind].head);  // head, then tail
      const float* tp = reinterpret_cast<const float*>(&tables->plain);
      constexpr int NF = (int)(sizeof(Tab) / sizeof(float));
      float* dst = reinterpret_cast<float*>(tabs);
      for (int i = t; i < 3 * NF; i += nt) dst[i] = i < 2 * NF ? __ldg(th + i) : __ldg(tp + i - 2 * NF);
      old_kind = kind;
    }
    if (SEQ) fence_proxy_async();
    __syncthreads();  // barrier and tables ready; in later windows, the tile free

    // ---- stage rows start .. start + Wr - 1 (zeros beyond the system) ----
    if (!CONTIG && g.boxr > 0) {
      if (t == 0) {
        mbar_expect_tx(bar, (unsigned)(g.Wr * SG * 8));
        for (int r = 0; r < g.Wr; r += g.boxr) tma_load(tile + (size_t)r * SG, &tin, x0, start + r, plane, 0, bar);
        if (g.pf > 0) {
          const long long bn = (long long)blockIdx.x + g.pf;
          if (bn < (long long)gridDim.x) {
            const int gn = SEQ ? (int)bn : (int)(bn / g.P);
            const int pn = gn / g.gpp, wn = SEQ ? 0 : (int)(bn - (long long)gn * g.P);
            if (w == 0 || !SEQ)
              for (int r = 0; r < g.Wr; r += g.boxr)
                tma_prefetch_l2(&tin, (gn - pn * g.gpp) * SG, wn * (g.Wr - 2 * g.H) + r, pn, 0);
          }
        }
      }
    } else if (CONTIG) {
      if (g.bulk) {
        if (t == 0) mbar_expect_tx(bar, (unsigned)(live * nv * 8));
        if (t < 32) __syncwarp();
        if (t < live) {
          bulk_load(col, in + mine + start, (unsigned)(nv * 8), bar);
          const long long bn = (long long)blockIdx.x + g.pf;
          if (g.pf > 0 && w == 0 && bn < (long long)gridDim.x) {
            const int gn = SEQ ? (int)bn : (int)(bn / g.P);
            const int pn = gn / g.gpp, wn = SEQ ? 0 : (int)(bn - (long long)gn * g.P);
            const int xn = (gn - pn * g.gpp) * SG + t, sn = wn * (g.Wr - 2 * g.H);
            if (xn < g.ni)
              bulk_prefetch_l2(in + (long long)pn * g.os + (long long)xn * g.is + sn,
                               (unsigned)(min(g.Wr, g.n - sn) * 8));
          }
        }
      } else {
        // a system per warp turn, lanes walk its rows
        const int warps = nt >> 5, lane = t & 31;
        if (t < warps * 32)
          for (int sy = t >> 5; sy < live; sy += warps) {
            const double* src = in + base + (long long)sy * g.is + start;
            for (int q = lane; q < nv; q += 32) cp_async8(tile + sy * (g.Wr + 2) + q, src + q, 8u);
          }
      }
      // rows beyond the system, systems beyond the group
      if (s >= live || r0 + ROWS > nv) {
        for (int k = s < live ? max(nv - r0, 0) : 0; k < ROWS; ++k) col[r0 + k] = 0.0;
      }
    } else {
#pragma unroll 4
      for (int r = c; r < g.Wr; r += g.nc) {
        const bool ok = s < live && r < nv;
        cp_async8(col + (size_t)r * RS, ok ? in + mine + (long long)(start + r) * g.es : in, ok ? 8u : 0u);
      }
    }
    // neighbours of the window's rows and the tail's one-sided stencil, from
    // global memory while the tile arrives
    double fl = 0.0, fr = 0.0;
    float bh = 0.f, bl = 0.f;
    if (RHS == RHS_COMPACT && s < live) {
      const double* f = in + mine;
      if (c == 0 && start > 0) fl = f[(long long)(start - 1) * g.es];
      if (c == g.nc - 1 && start + g.Wr < g.n) fr = f[(long long)(start + g.Wr) * g.es];
      if (c == last && w == g.P - 1) {
        const double* e = f + (long long)(g.n - 1) * g.es;
        boundary_rhs(e[0], e[-g.es], e[-2 * g.es], a.sigmaN, bh, bl, rmax);
      }
    }
    bool there = true;
    if (CONTIG ? g.bulk : g.boxr > 0)
      there = mbar_wait(bar, phase);
    else
      cp_async_wait_all();
    phase ^= 1u;
    if (!__syncthreads_and(there)) {
      if (t == 0 && a.status) atomicOr(a.status, STATUS_TIMEOUT);
      return;
    }
    if (SEQ && w > 0) {  // rows that the window before has overwritten
      for (int r = c; r < g.H; r += g.nc) col[(size_t)r * RS] = stash[r * SG + s];
      __syncthreads();
    }

    // ---- right-hand side as (hi, lo) pairs in place; v: the high parts ----
    float2 v[8];
    float2 edge0 = make_float2(0.f, 0.f), edge15 = edge0;
    auto put = [&](int k, float h, float l) {  // row r0 + k
      reinterpret_cast<float2*>(col + (size_t)(r0 + k) * RS)[0] = make_float2(h, l);
    };
    if (RHS == RHS_COMPACT) {
      if (c > 0) fl = col[(size_t)(r0 - 1) * RS];
      if (c < g.nc - 1) fr = col[(size_t)(r0 + ROWS) * RS];
      const bool head = c == 0 && start == 0, tail = c == last && w == g.P - 1;
      if (head) boundary_rhs(col[0], col[RS], col[2 * RS], a.sigma0, bh, bl, rmax);
      double prev = fl, cur = col[(size_t)r0 * RS];
      double2 two = make_double2(0.0, 0.0);
      float h0 = 0.f, l0 = 0.f;  // the even row before
#pragma unroll
      for (int k = 0; k < ROWS; ++k) {
        double nxt = fr;
        if (k < ROWS - 1) {
          if (CONTIG) {
            if ((k & 1) || k == 0) two = *reinterpret_cast<const double2*>(col + r0 + ((k + 1) & ~1));
            nxt = (k & 1) ? two.x : two.y;
          } else {
            nxt = col[(size_t)(r0 + k + 1) * RS];
          }
        }
        float h, l;
        r2::split_f64(dsub_(nxt, prev), h, l, rmax);
        if (k == 0 && head) {
          h = bh;
          l = bl;
        }
        if (k == 0) edge0 = make_float2(h, l);
        else if (k == ROWS - 1) edge15 = make_float2(h, l);
        else if (!CONTIG || k == 1 || k == ROWS - 2) put(k, h, l);
        else if (k & 1) *reinterpret_cast<float4*>(col + r0 + k - 1) = make_float4(h0, l0, h, l);
        h0 = h;
        l0 = l;
        if (k < HALF) v[k].x = h;
        else v[k - HALF].y = h;
        prev = cur;
        cur = nxt;
      }
      if (tail) {  // the last row's stencil, zeros beyond it
#pragma unroll
        for (int k = 0; k < ROWS; ++k)
          if (k >= kt) {
            const float h = k == kt ? bh : 0.f, l = k == kt ? bl : 0.f;
            if (k == 0) edge0 = make_float2(h, l);
            else if (k == ROWS - 1) edge15 = make_float2(h, l);
            else put(k, h, l);
            if (k < HALF) v[k % HALF].x = h;
            else v[k % HALF].y = h;
          }
      }
    } else {
      const bool keep = SEQ && w < g.P - 1 && r0 + ROWS > hi - g.H && r0 < hi;
      auto row = [&](int k, double d, float& h, float& l) {
        if (keep && r0 + k >= hi - g.H && r0 + k < hi) stash[(r0 + k - (hi - g.H)) * SG + s] = d;
        r2::split_f64(d, h, l, rmax);
        if (k < HALF) v[k % HALF].x = h;
        else v[k % HALF].y = h;
      };
#pragma unroll
      for (int k = 0; k < ROWS; k += 2) {
        double d0, d1;
        if (CONTIG) {
          const double2 q = *reinterpret_cast<const double2*>(col + r0 + k);
          d0 = q.x;
          d1 = q.y;
        } else {
          d0 = col[(size_t)(r0 + k) * RS];
          d1 = col[(size_t)(r0 + k + 1) * RS];
        }
        float ha, la, hb, lb;
        row(k, d0, ha, la);
        row(k + 1, d1, hb, lb);
        if (CONTIG) {
          *reinterpret_cast<float4*>(col + r0 + k) = make_float4(ha, la, hb, lb);
        } else {
          put(k, ha, la);
          put(k + 1, hb, lb);
        }
      }
    }

    // ---- FP32 solve ----
    constexpr int CW = 32 / SG;  // chunks of a warp
    const bool tab = c / CW == 0 || c / CW == last / CW;
    const bool dead = c > last;                   // rows beyond the system only
    const ByConst fc{K};
    const ByTab ft{tabs + (c == 0 ? 0 : c == last ? 1 : 2)};
    if (dead) {
#pragma unroll
      for (int k = 0; k < HALF; ++k) v[k] = make_float2(0.f, 0.f);
    }
    X(X_E1, 0) = tab ? forward(v, ft) : forward(v, fc);
    __syncthreads();  // carries published; every halo row has been read
    if (RHS == RHS_COMPACT) {
      put(0, edge0.x, edge0.y);
      put(ROWS - 1, edge15.x, edge15.y);
    }
    const bool from_left = c > 0 && !dead;
    {
      const float CA = from_left ? X(X_E1, -1) : 0.f;
      X(X_S1, 0) = tab ? backward(v, CA, ft) : backward(v, CA, fc);
    }
    X(X_A0, 0) = v[0].x;
    X(X_B0, 0) = v[0].y;
    X(X_B7, 0) = v[7].y;
    __syncthreads();
    {
      const float XB = c < last ? X(X_S1, 1) : 0.f;
      if (tab) carry_in(v, XB, ft);
      else carry_in(v, XB, fc);
    }
    // ---- residual: the neighbours' edge rows as their owners have them ----
    float xl = 0.f, xr = 0.f;
    if (from_left) xl = fma_(c == 1 ? tabs[0].psi[7].y : K.psi[7].y, X(X_S1, 0), X(X_B7, -1));
    if (c < last) {
      const float XA = c + 1 < last ? fma_(K.psi[0].y, X(X_S1, 2), X(X_B0, 1)) : X(X_B0, 1);
      xr = fma_(c + 1 == last ? tabs[1].psi[0].x : K.psi[0].x, XA, X(X_A0, 1));
    }
    float2 r[8];
    auto residual = [&](int k, float2 da, float2 db) {
      const float2 xm = (k == 0) ? pair(xl, v[HALF - 1].x) : v[(k + HALF - 1) % HALF];
      const float2 xp = (k == HALF - 1) ? pair(v[0].y, xr) : v[(k + 1) % HALF];
      r[k] = res_interior<GEN>(pair(da.x, db.x), pair(da.y, db.y), xm, v[k], xp, a);
    };
#pragma unroll
    for (int k = 0; k < HALF; k += 2) {
      if (CONTIG) {
        const float4 qa = *reinterpret_cast<const float4*>(col + r0 + k);
        const float4 qb = *reinterpret_cast<const float4*>(col + r0 + k + HALF);
        residual(k, pair(qa.x, qa.y), pair(qb.x, qb.y));
        residual(k + 1, pair(qa.z, qa.w), pair(qb.z, qb.w));
      } else {
#pragma unroll
        for (int q = 0; q < 2; ++q)
          residual(k + q, reinterpret_cast<const float2*>(col + (size_t)(r0 + k + q) * RS)[0],
                   reinterpret_cast<const float2*>(col + (size_t)(r0 + k + q + HALF) * RS)[0]);
      }
    }
    if (c == 0) {
      const Kind& q = tables->kind[kind];
      const float2 d = reinterpret_cast<const float2*>(col)[0];
      r[0].x = res_row(d.x, d.y, 0.f, v[0].x, v[1].x, q.hd[0], q.hd[1], q.hd[2]);
    }
    if (c == last) {
      const Kind& q = tables->kind[kind];
      const float2 d = reinterpret_cast<const float2*>(col + (size_t)(r0 + kt) * RS)[0];
      float xm = xl, x = v[0].x;
#pragma unroll
      for (int k = 1; k < ROWS; ++k) {
        const float here = k < HALF ? v[k % HALF].x : v[k % HALF].y;
        const float before = k - 1 < HALF ? v[(k - 1) % HALF].x : v[(k - 1) % HALF].y;
        x = k == kt ? here : x;
        xm = k == kt ? before : xm;
      }
      const float rt = res_row(d.x, d.y, xm, x, 0.f, q.td[0], q.td[1], q.td[2]);
#pragma unroll
      for (int k = 0; k < HALF; ++k) {
        r[k].x = k == kt ? rt : k > kt ? 0.f : r[k].x;
        r[k].y = k + HALF == kt ? rt : k + HALF > kt ? 0.f : r[k].y;
      }
    }
    if (dead) {
#pragma unroll
      for (int k = 0; k < HALF; ++k) r[k] = make_float2(0.f, 0.f);
    }
    // ---- FP32 correction solve ----
    X(X_E2, 0) = tab ? forward(r, ft) : forward(r, fc);
    __syncthreads();
    {
      const float CA = from_left ? X(X_E2, -1) : 0.f;
      X(X_S2, 0) = tab ? backward(r, CA, ft) : backward(r, CA, fc);
    }
    __syncthreads();
    {
      const float XB = c < last ? X(X_S2, 1) : 0.f;
      if (tab) carry_in(r, XB, ft);
      else carry_in(r, XB, fc);
    }
    // ---- s (x + delta) as FP64 ----
    if (CONTIG) {
#pragma unroll
      for (int k = 0; k < HALF; k += 2) {
        double2 oa, ob;
        out_pair(v[k], r[k], a, oa.x, ob.x);
        out_pair(v[k + 1], r[k + 1], a, oa.y, ob.y);
        *reinterpret_cast<double2*>(col + r0 + k) = oa;
        *reinterpret_cast<double2*>(col + r0 + k + HALF) = ob;
      }
      if (g.bulk) {
        fence_proxy_async();
        __syncthreads();
        if (t < live) {
          bulk_store(out + mine + start + lo, col + lo, (unsigned)((hi - lo) * 8));
          tma_store_commit_and_wait();
        }
      } else {
        __syncthreads();
        const int warps = nt >> 5, lane = t & 31;
        if (t < warps * 32)
          for (int sy = t >> 5; sy < live; sy += warps) {
            double* dst = out + base + (long long)sy * g.is + start;
            for (int q = lo + lane; q < hi; q += 32) dst[q] = tile[sy * (g.Wr + 2) + q];
          }
      }
    } else {
      double* dst = out + mine + (long long)(start + r0) * g.es;
      // rows of this chunk to store: bits lo - r0 .. hi - r0 - 1
      const unsigned below = (1u << min(max(lo - r0, 0), ROWS)) - 1u;
      const unsigned rows = s < live ? ((1u << min(max(hi - r0, 0), ROWS)) - 1u) & ~below : 0u;
#pragma unroll
      for (int k = 0; k < HALF; ++k) {
        double oa, ob;
        out_pair(v[k], r[k], a, oa, ob);
        if (rows >> k & 1u) dst[(long long)k * g.es] = oa;
        if (rows >> (k + HALF) & 1u) dst[(long long)(k + HALF) * g.es] = ob;
      }
    }
    if (!SEQ || ++w == g.P) break;
  }
  if (__any_sync(__activemask(), rmax >= RANGE_MAG) && (t & 7) == 0 && a.status) atomicOr(a.status, 1u);
}

}  // namespace r2n

struct R2N {
  struct Layout : r2n::Windows {
    int nc = 0;  // chunks of a window
  };
  int n = 0;
  Layout lay[2];  // strided, contiguous
  bool gen = false;
  int device = 0, sms = 152;
  r2::Args args;
  r2n::Tables* d_tables = nullptr;  // [2]
  unsigned* d_status = nullptr;     // behind them
  ~R2N() {
    if (d_tables) cudaFree(d_tables);
  }
};

void r2n_destroy(R2N* r) { delete r; }

void r2n_status_words(const R2N* r, std::vector<unsigned*>& out) {
  if (r && r->d_status) out.push_back(r->d_status);
}

namespace {

using r2n::Kind;
using r2n::Tab;

// The factors of rows r0 .. r0 + 15 (identity rows from n on).
Tab table_of(const std::vector<double>& l, const std::vector<double>& u, const std::vector<double>& w, int r0) {
  const int n = (int)l.size();
  Tab t;
  for (int half = 0; half < 2; ++half) {
    double p = 1.0;
    for (int k = 0; k < 8; ++k) {
      const int i = r0 + 8 * half + k;
      const bool in = i < n;
      const float nl = in ? (float)-l[i] : 0.f, g = in ? (float)(1.0 / u[i]) : 1.f, nw = in ? (float)-w[i] : 0.f;
      p *= in ? -l[i] : 0.0;
      if (half == 0) t.nl[k].x = nl, t.g[k].x = g, t.nw[k].x = nw, t.phi[k].x = (float)p;
      else t.nl[k].y = nl, t.g[k].y = g, t.nw[k].y = nw, t.phi[k].y = (float)p;
    }
    p = 1.0;
    for (int k = 7; k >= 0; --k) {
      const int i = r0 + 8 * half + k;
      p *= i < n ? -w[i] : 0.0;
      if (half == 0) t.psi[k].x = (float)p;
      else t.psi[k].y = (float)p;
    }
  }
  return t;
}

bool near(double a, double b) { return std::fabs(a - b) <= std::ldexp(1.0, -24) * std::fabs(b); }

}  // namespace

int r2n_create(R2N** out, const Plan& p) {
  using namespace r2n;
  *out = nullptr;
  const int n = p.n;
  const Matrix& m = p.mat;
  // (64 rows: the two chunks with tables are half of each system, 64^3 along x
  // 10.5 us against the chunked kernel's 8.9; from 100 on this one is faster)
  if (n < 96 || m.nh != 1 || m.nt != 1) return NTK_OK;
  // pivot fixed point of the interior
  double u = m.bi;
  for (int it = 0; it < 4096; ++it) {
    const double un = m.bi - m.ai * m.ci / u;
    if (!std::isfinite(un) || un == 0.0) return NTK_OK;
    if (un == u) break;
    u = un;
  }
  if (!(std::fabs(m.bi - m.ai * m.ci / u - u) <= 1e-15 * std::fabs(u))) return NTK_OK;
  const double l = m.ai / u, w = m.ci / u, mult = std::max(std::fabs(l), std::fabs(w));
  // the carry across two sub-chunks is dropped, as in ntk_r2.cu
  if (!(std::pow(mult, 16) <= std::ldexp(1.0, -26))) return NTK_OK;
  R2N* r = new (std::nothrow) R2N();
  if (!r) {
    set_error("out of host memory");
    return NTK_ERR_ALLOC;
  }
  r->n = n;
  int H = 0;
  for (double q = 1.0; q > std::ldexp(1.0, -56); q *= mult) ++H;
  H = (H + 3) & ~1;  // even: window starts stay 16-byte aligned
  for (int lay = 0; lay < 2; ++lay) {
    R2N::Layout& y = r->lay[lay];
    static_cast<Windows&>(y) = choose_windows(n, H, lay ? group_size<true> : group_size<false>);
    if (!y.P || !last_window_ok(y)) {
      delete r;
      return NTK_OK;
    }
    y.nc = y.Wr / 16;
  }
  r->gen = !(r2::pow2_or_zero(m.ai) && r2::pow2_or_zero(m.bi) && r2::pow2_or_zero(m.ci));
  // constants of the interior, and its residual
  r2::Args& a = r->args;
  std::memset(&a, 0, sizeof(a));
  r2::Consts& k = a.k;
  k.nl = r2::splat((float)-l);
  k.g = r2::splat((float)(1.0 / u));
  k.nw = r2::splat((float)-w);
  for (int i = 0; i < 8; ++i) {
    k.phi[i] = r2::splat((float)std::pow(-l, i + 1));
    k.psi[i] = r2::splat((float)std::pow(-w, 8 - i));
  }
  a.ca = r2::splat((float)m.ai);
  a.cb = r2::splat((float)m.bi);
  a.cc = r2::splat((float)m.ci);
  a.cal = r2::splat(r2::to_dwc(m.ai).l);
  a.cbl = r2::splat(r2::to_dwc(m.bi).l);
  a.ccl = r2::splat(r2::to_dwc(m.ci).l);
  a.nca = r2::splat(-(float)m.ai);
  a.ncb = r2::splat(-(float)m.bi);
  a.ncc = r2::splat(-(float)m.ci);
  // both layouts' tables and, behind them, the status word
  std::vector<unsigned char> host(2 * sizeof(Tables) + 16, 0);
  for (int lay = 0; lay < 2; ++lay) {
    const R2N::Layout& y = r->lay[lay];
    Tables tb;
    std::memset(&tb, 0, sizeof(tb));
    for (int i = 0; i < 8; ++i) {
      tb.plain.nl[i] = k.nl;
      tb.plain.g[i] = k.g;
      tb.plain.nw[i] = k.nw;
      tb.plain.phi[i] = k.phi[i];
      tb.plain.psi[i] = k.psi[i];
    }
    bool ok = true;
    for (int kind = 0; kind < KINDS && ok; ++kind) {
      if ((kind == WHOLE) != (y.P == 1) || (kind == MIDDLE && y.P < 3)) continue;
      const bool cut_head = kind == MIDDLE || kind == LAST, cut_tail = kind == FIRST || kind == MIDDLE;
      const int rows = kind == WHOLE || kind == LAST ? y.last : y.Wr;
      Matrix q;
      q.n = rows;
      const double co[7] = {cut_head ? m.bi : m.b(0),     cut_head ? m.ci : m.c(0),     m.ai, m.bi, m.ci,
                            cut_tail ? m.ai : m.a(n - 1), cut_tail ? m.bi : m.b(n - 1)};
      q.set_reference(co);
      std::vector<double> fl, fu, fw(rows);
      ok = factor_host(q, fl, fu);
      if (!ok) break;
      for (int i = 0; i < rows; ++i) fw[i] = q.c(i) / fu[i];
      // every chunk but the first and the last has the interior's factors
      const int last = (rows - 1) / 16;
      for (int i = 16; i < 16 * last && ok; ++i) ok = near(fl[i], l) && near(fu[i], u) && near(fw[i], w);
      Kind& kd = tb.kind[kind];
      kd.head = table_of(fl, fu, fw, 0);
      kd.tail = table_of(fl, fu, fw, 16 * last);
      for (int e = 0; e < 3; ++e) {
        kd.hd[e] = r2::to_dwc(e == 0 ? 0.0 : e == 1 ? co[0] : co[1]);
        kd.td[e] = r2::to_dwc(e == 0 ? co[5] : e == 1 ? co[6] : 0.0);
      }
    }
    if (!ok) {
      delete r;
      return NTK_OK;
    }
    std::memcpy(host.data() + lay * sizeof(Tables), &tb, sizeof(tb));
  }
  cudaGetDevice(&r->device);
  cudaDeviceGetAttribute(&r->sms, cudaDevAttrMultiProcessorCount, r->device);
  int rc = cuda_status(cudaMalloc(&r->d_tables, host.size()), "cudaMalloc(window tables)");
  if (!rc)
    rc = cuda_status(cudaMemcpy(r->d_tables, host.data(), host.size(), cudaMemcpyHostToDevice),
                     "cudaMemcpy(window tables)");
  if (rc) {
    delete r;
    return rc;
  }
  r->d_status = reinterpret_cast<unsigned*>(r->d_tables + 2);
  *out = r;
  return NTK_OK;
}

namespace {

// Whether tensor maps address the strided systems of a batch.
bool maps_apply(const double* in, const Batch& b, long long planes) {
  return r2::aligned16(in) && b.es % 2 == 0 && (planes == 1 || b.os % 2 == 0);
}

}  // namespace

// Which batches take this kernel rather than the chunked ones (one warp a
// system), by the threads it gives an SM: a CTA's time is mostly latency, and
// staging without tensor maps (8-byte copies) adds to it, so it takes several
// a SM to win.  Measured, us, this kernel : the chunked ones, with threads an
// SM: contiguous 2432 systems of 128 rows (128) 5.7 : 4.0, 8192 (431) 8.3 :
// 8.5, 4868 of 256 (513) 8.6 : 9.2, 8191 of 97, odd (377) 10.4 : 9.1, 12001
// (553) 12.0 : 12.5; strided with tensor maps 2560 of 256 (269) 7.4 : 7.1, 4868
// (514) 9.2 : 10.0; without 4867 of 500 (1027) 20.2 : 18.0, 8191 (1725) 27.6 :
// 26.7, 12001 of 385 (2372) 31.8 : 34.8; windows in place, in order, strided
// 2432 of 1024 (256) 24.4 : 18.5, 4868 (514) 42.2 : 40.7, 6400 (674) 42.9 :
// 50.1; contiguous 2437 of 2048 (401) 45.7 : 43.8, 3600 of 1024 (568) 23.5 :
// 25.6.
bool r2n_serves(const R2N* r, const double* in, const double* out, const Batch& b, const RhsParams& rp,
                bool always) {
  if (!r || b.nsys < 1 || (rp.kind != RHS_IDENTITY && rp.kind != RHS_COMPACT)) return false;
  if (b.nsys > b.ni && b.nsys % b.ni != 0) return false;
  const long long planes = b.nsys > b.ni ? b.nsys / b.ni : 1, ni = b.nsys / planes;
  if (ni >= (1LL << 30) || planes >= (1LL << 30)) return false;
  // contiguous systems apart from each other, or adjacent strided ones
  const long long plane = b.es == 1 ? (ni - 1) * b.is + r->n : (long long)(r->n - 1) * b.es + ni;
  if (b.es == 1 ? b.is < r->n : (b.is != 1 || b.es < ni)) return false;
  if (planes > 1 && b.os < plane) return false;
  const R2N::Layout& y = r->lay[b.es == 1];
  const int sg = b.es == 1 ? r2n::group_size<true> : r2n::group_size<false>;
  const long long groups = (ni + sg - 1) / sg * planes;
  if (groups * y.P > 0x7fffffffLL) return false;
  const long long extent = (planes - 1) * b.os + plane;
  if (in != out && in < out + extent && out < in + extent) return false;
  // windows in place: all of a system's windows in one CTA
  const bool seq = in == out && y.P > 1;
  if (seq && rp.kind != RHS_IDENTITY) return false;
  if (always) return true;
  const bool contig = b.es == 1;
  int least = seq ? (contig ? 448 : 640) : 384;
  if (!contig && !maps_apply(in, b, planes)) least = r->n <= 512 ? 1280 : seq ? 1024 : 768;
  return (seq ? groups : groups * y.P) * (sg * y.nc) >= (long long)least * r->sms;
}

namespace {

template <int RHS, bool CONTIG, bool GEN, bool SEQ>
int r2n_launch(const R2N* r, const CUtensorMap& map, const double* in, double* out, const r2n::Geom& g,
               const r2::Args& a, long long groups, cudaStream_t st) {
  auto k = r2n::r2n_kernel<RHS, CONTIG, GEN, SEQ>;
  const size_t smem = r2n::smem_of<CONTIG>(g.Wr, g.nc, SEQ ? g.H : 0);
  int rc = allow_smem(k, smem, "cudaFuncSetAttribute(r2n_kernel)");
  if (rc) return rc;
  const long long grid = SEQ ? groups : groups * g.P;
  k<<<(unsigned)grid, r2n::group_size<CONTIG> * g.nc, smem, st>>>(map, in, out, g, a, r->d_tables + CONTIG);
  return cuda_status(cudaGetLastError(), "r2n_kernel");
}

template <int RHS, bool CONTIG, bool SEQ>
int r2n_gen(const R2N* r, const CUtensorMap& map, const double* in, double* out, const r2n::Geom& g,
            const r2::Args& a, long long groups, cudaStream_t st) {
  return r->gen ? r2n_launch<RHS, CONTIG, true, SEQ>(r, map, in, out, g, a, groups, st)
                : r2n_launch<RHS, CONTIG, false, SEQ>(r, map, in, out, g, a, groups, st);
}

}  // namespace

int r2n_run(R2N* r, const double* in, double* out, const Batch& b, const RhsParams& rp, double s, int prefetch,
            cudaStream_t st) {
  const long long planes = b.nsys > b.ni ? b.nsys / b.ni : 1, ni = b.nsys / planes;
  const bool contig = b.es == 1;
  const R2N::Layout& y = r->lay[contig];
  const bool seq = in == out && y.P > 1;
  const int sg = contig ? r2n::group_size<true> : r2n::group_size<false>;
  r2n::Geom g;
  g.n = r->n;
  g.Wr = y.Wr;
  g.nc = y.nc;
  g.H = y.H;
  g.P = y.P;
  g.ni = (int)ni;
  g.gpp = (int)((ni + sg - 1) / sg);
  g.is = b.is;
  g.os = planes > 1 ? b.os : 0;
  g.es = b.es;
  g.boxr = 0;
  g.bulk = contig && r2::aligned16(in) && r2::aligned16(out) && r->n % 2 == 0 && b.is % 2 == 0 &&
           (planes == 1 || b.os % 2 == 0);
  g.pf = 0;
  const long long groups = (long long)g.gpp * planes;
  CUtensorMap map;
  std::memset(&map, 0, sizeof(map));
  if (!contig && maps_apply(in, b, planes)) {
    g.boxr = y.Wr > 256 ? y.Wr / 2 : y.Wr;
    const cuuint64_t dims[4] = {(cuuint64_t)ni, (cuuint64_t)r->n, (cuuint64_t)planes, 1};
    const long long ps = planes > 1 ? b.os : (long long)b.es * r->n;
    const cuuint64_t strides[3] = {(cuuint64_t)b.es * 8, (cuuint64_t)ps * 8, (cuuint64_t)ps * planes * 8};
    const cuuint32_t box[4] = {(cuuint32_t)sg, (cuuint32_t)g.boxr, 1, 1};
    int rc = r2::encode(&map, in, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (rc) return rc;
  }
  if (g.boxr || g.bulk) g.pf = prefetch * r->sms * std::min(1024 / (sg * y.nc), 32) / 2;
  r2::Args a = r->args;
  r2::set_scales(&a, rp.kind == RHS_COMPACT ? rp.sigma0 : 1.0, rp.kind == RHS_COMPACT ? rp.sigmaN : 1.0, s);
  a.status = r->d_status;
  if (rp.kind == RHS_COMPACT)
    return contig ? r2n_gen<RHS_COMPACT, true, false>(r, map, in, out, g, a, groups, st)
                  : r2n_gen<RHS_COMPACT, false, false>(r, map, in, out, g, a, groups, st);
  if (seq)
    return contig ? r2n_gen<RHS_IDENTITY, true, true>(r, map, in, out, g, a, groups, st)
                  : r2n_gen<RHS_IDENTITY, false, true>(r, map, in, out, g, a, groups, st);
  return contig ? r2n_gen<RHS_IDENTITY, true, false>(r, map, in, out, g, a, groups, st)
                : r2n_gen<RHS_IDENTITY, false, false>(r, map, in, out, g, a, groups, st);
}

}  // namespace ntk
