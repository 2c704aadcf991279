// ntk_chunk_f64.h -- FP64 solves of few systems, T threads per system
// (kernel and rationale in ntk_chunk_f64.cu).
#pragma once
#include <vector>

#include "ntk_internal.h"

namespace ntk {

// Tables of one matrix for every thread count it is offered with.
struct ChunkF64 {
  struct Cfg {
    int T = 0;             // threads per system
    int C = 0;             // rows per thread (odd: conflict-free in a dense shared-memory row)
    int CP = 0;            // C rounded up to the row batch of the sweeps
    int ncls = 0;          // distinct chunks (threads with bitwise equal factors share one)
    size_t tab = 0;        // offset of [ncls][4][CP] -l, phi, -w, psi in d_tab
    size_t scan = 0;       // offset of [2][log2 T][T] scan multipliers in d_tab
    size_t cls = 0;        // offset of the T class numbers (ints) in d_tab
    size_t g = 0;          // offset of [ncls][CP] rows of g among the g rows
    std::vector<int> rep;  // representative thread of each class
  };
  int n = 0;
  std::vector<Cfg> cfgs;
  double* d_tab = nullptr;
  size_t g_elems = 0;      // values of the g rows of all configurations

  ~ChunkF64();
  // l, u: the matrix's LU factors, w = c / u.  Leaves cfgs empty where no
  // thread count applies; fails only where an allocation or a copy does.
  int init(int n, const double* l, const double* u, const double* w);
  // rows of g[n] in chunk order for every configuration (g_elems values)
  void g_rows(const double* g, double* out) const;
};

// The configuration for a batch, or null where one thread per system
// (ntk_solve_f64.cu) is the faster; S: systems per CTA.
const ChunkF64::Cfg* chunk_f64_pick(const ChunkF64& c, const Batch& b, int rhs, int* S);

// rp.kind: RHS_IDENTITY, RHS_COMPACT or RHS_CROSS (with rp.center == 0 the
// stencil is -(lo + hi): rows divided by -rp.top).  t: the matrix's plain
// tables (systems whose values overflow or are not finite are solved with
// them, row by row); g: the g rows of chunk order in device memory.
int launch_chunk_f64(const ChunkF64& c, const ChunkF64::Cfg& cfg, int S, const double* in, double* out,
                     const Batch& b, const RhsParams& rp, const TablesF64& t, const double* g, cudaStream_t st);

}  // namespace ntk
