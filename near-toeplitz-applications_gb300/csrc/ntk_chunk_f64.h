// ntk_chunk_f64.h -- FP64 solves of few systems, T threads per system
// (kernel and rationale in ntk_chunk_f64.cu).
#pragma once
#include <vector>

#include "ntk_internal.h"
#include "ntk_soft_f64.cuh"

namespace ntk {

// Tables of one matrix for every thread count it is offered with.
struct ChunkF64 {
  struct Cfg {
    int T = 0;             // threads per system
    int C = 0;             // rows per thread, a multiple of the sweeps' row batch
    int ncls = 0;          // distinct chunks (threads with bitwise equal factors share one)
    size_t tab = 0;        // offset of the classes' tables in d_tab
    size_t scan = 0;       // offset of [2][log2 T][T] scan multipliers in d_tab
    size_t cls = 0;        // offset of the T class numbers (ints) in d_tab
    size_t g = 0;          // offset of [ncls][C] rows of g among the g rows
    std::vector<int> rep;  // representative thread of each class
  };
  int n = 0;
  std::vector<Cfg> cfgs;
  const double* d_tab = nullptr;  // the plan's copy of init's tables
  size_t g_count = 0;      // rows of g of all configurations

  // l, u: the matrix's LU factors, w = c / u.  Returns the tables for the
  // device; leaves cfgs empty where no thread count applies.
  std::vector<double> init(int n, const double* l, const double* u, const double* w);
  // whether some configuration fits contiguous and some strided systems
  bool serves_both_layouts() const;
  // A g table holds g[n] and, from g_offset(n) on, the rows of g in chunk
  // order for every configuration, prepared for soft_product and plain
  // (g_elems() doubles, filled by g_rows).
  static size_t g_offset(int n) { return ((size_t)n + 1) & ~(size_t)1; }
  size_t g_elems() const { return 3 * g_count; }
  void g_rows(const double* g, double* out) const;
};

// The configuration for a batch, or null where one thread per system
// (ntk_solve_f64.cu) is the faster and `always` is not set, or where none
// fits; S: systems per CTA.
const ChunkF64::Cfg* chunk_f64_pick(const ChunkF64& c, const Batch& b, int rhs, int* S, bool always = false);

// rp.kind: RHS_IDENTITY, RHS_COMPACT or RHS_CROSS (with rp.center == 0 the
// stencil is -(lo + hi): rows divided by -rp.top).  t: the matrix's plain
// tables (systems whose values overflow or are not finite are solved with
// them, row by row), t.g a g table.
int launch_chunk_f64(const ChunkF64& c, const ChunkF64::Cfg& cfg, int S, const double* in, double* out,
                     const Batch& b, const RhsParams& rp, const TablesF64& t, cudaStream_t st);

}  // namespace ntk
