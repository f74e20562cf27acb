// Whole HEOM time loop of small blocks with site couplings in one launch, FP32
// (heom_site.cu).
#pragma once
#include "qsx_common.cuh"

namespace qsx {

// Runs the loop of `a` (FP32) into saves [batch][nsave][save_nodes * E] and
// returns true, or returns false when the shape is not this form's: blocks
// that are not n x n with 3 <= n <= 8, aki_temp_corr terms, or hierarchies
// that do not fit a cluster.  *st is the status when it ran;
// `low` (16-byte aligned) is scratch for batch x nnodes x (n rounded up to
// even)^2 complex words, `order` for 2 nnodes ints.
bool heom_site_run(const qsx_heom_args* a, double2* saves, float2* low, int* order,
                   cudaStream_t s, int* st);

}  // namespace qsx
