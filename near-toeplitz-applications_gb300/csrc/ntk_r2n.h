// ntk_r2n.h -- FP32 + refinement for systems of any length on the
// paired-chunk arithmetic (kernel and rationale in ntk_r2n.cu).
#pragma once
#include "ntk_plan.h"

namespace ntk {

struct R2N;

// Tables for a plan's matrix, or *out = null where this solve does not apply
// (slow decay, a head that converges too slowly, n < 96); an error only where
// an allocation or a copy fails.
int r2n_create(R2N** out, const Plan& p);
void r2n_destroy(R2N* r);
void r2n_status_words(const R2N* r, std::vector<unsigned*>& out);

// Whether r2n_run serves this batch (one refinement sweep) and is the faster.
bool r2n_serves(const R2N* r, const double* in, const double* out, const Batch& b, const RhsParams& rp,
                bool always = false);
int r2n_run(R2N* r, const double* in, double* out, const Batch& b, const RhsParams& rp, double s, int prefetch,
            cudaStream_t st);

}  // namespace ntk
