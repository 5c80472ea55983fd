// Whole block-RHS solves in one launch of thread-block clusters
// (solve_cluster.cu).
#pragma once

#include "plan.h"

namespace aosb {
// Both sweeps of one solve (tile 128, split-BF16 updates) for every pencil of
// the batch; `status` holds a word per pencil.  Returns false, with nothing
// done, where one launch per step is expected to be faster; otherwise *rc is
// the result.
bool solve_cluster(const aosb_plan* P, const aosb_solve_args_v1* a, int32_t* status, int* rc,
                   char* err, size_t cap);
}  // namespace aosb
