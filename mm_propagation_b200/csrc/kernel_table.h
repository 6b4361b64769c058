// kernel_table.h — host-visible handles to the kernels instantiated for one
// (precision, log2 NT) pair by kern_inst.cu.
#pragma once

#include "radix_plan.h"

namespace mmp {

struct KernelSet {
  const void* prime = nullptr;
  const void* pair = nullptr;
  const void* nu = nullptr;          // k_nu for any stage
  const void* nu_mid[6] = {};        // ... for intermediate stages reading n stored N_hat_j
  const void* nu_last[5] = {};       // ... for last stages reading n (null: not built)
  const void* result = nullptr;
  const void* dft_fwd = nullptr;
  const void* dft_inv = nullptr;
  int C = 0;      // CTAs per row (cluster size)
  int nthr = 0;   // threads per CTA
  int smem = 0;   // dynamic shared memory per CTA, bytes
  int logn = 0;
  int fp64 = 0;
  int xc = 0;     // rows split over 2^xc times the minimal number of CTAs
  int resident = 0;  // rows resident at once with one CTA per SM (0: not asked)
};

// Row splits built for rows of 2^logn samples: xc = 0 .. max_split, clusters of 2^xc times the
// minimal number of CTAs, up to 8 CTAs and down to 32 threads each.
constexpr int max_split(bool fp64, int logn) {
  return logn < 11 ? 0 : logn == 11 ? 2 : logn <= 13 ? 3 : fp64 ? 16 - logn : logn == 14 ? 3 : 17 - logn;
}

// Defined in the kern_inst.cu objects; returns an empty set for variants not built.
KernelSet kernels_for(int fp64, int logn, int xc = 0);

}  // namespace mmp
