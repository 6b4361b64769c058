// radix_plan.h — how a row of 2^logn samples is factored into the passes of its transform
// (fft.cuh), shared by the kernels, which take it at compile time, and the host, which
// builds the twiddle tables and the spectrum's storage order from it.
#pragma once

#include <cstddef>

namespace mmp {

constexpr int kMinLogN = 6;
constexpr int kMaxLogN = 16;
constexpr int kMaxPasses = 6;

// log2 of the radices: r[0] = A, the first pass over the whole row (stride B = N / A), then
// the row passes of the A sub-rows of B samples.
struct RadixPlan {
  int n;
  int r[kMaxPasses];
};

// A thread holds E = A samples: 16 from 8192 samples on (64 registers in FP32, so 1024 threads
// share an SM), 8 below, where a solve has few rows and a warp's own instruction stream is
// what it waits for. Radices of 32 took a pass less, but their unrolled bodies outgrew the
// instruction cache: k_nu on 32 x 6 rows of 16384 stalled on instruction fetches first of all
// (1.5-1.8 of 7 cycles per issued instruction).
constexpr RadixPlan radix_plan(int logn) {
  switch (logn) {
    case 6: return {6, {1, 1, 1, 1, 1, 1}};
    case 7: return {4, {2, 2, 2, 1}};
    case 8: return {3, {3, 3, 2}};
    case 9: return {3, {3, 3, 3}};
    case 10: return {4, {3, 3, 2, 2}};
    case 11: return {4, {3, 3, 3, 2}};
    case 12: return {4, {3, 3, 3, 3}};
    case 13: return {4, {4, 3, 3, 3}};
    case 14: return {4, {4, 4, 4, 2}};
    case 15: return {4, {4, 4, 4, 3}};
    default: return {4, {4, 4, 4, 4}};
  }
}

// Twiddle table of one size: for every pass but the last, in turn,
// [q < R][j < S] of exp(-2 pi i j q / L), L = R S the length the pass works on (2^logn for
// pass 0, then B, B / R_1, ...), so that a warp's lanes (consecutive j) read consecutive
// entries and a thread's q advance by a constant.
constexpr size_t twiddle_entries(int logn) {
  const RadixPlan p = radix_plan(logn);
  size_t n = 0;
  int l = logn;
  for (int i = 0; i + 1 < p.n; ++i) {
    n += (size_t)1 << l;
    l -= p.r[i];
  }
  return n;
}
constexpr size_t twiddle_offset(int logn) {  // sizes one after the other
  size_t n = 0;
  for (int l = kMinLogN; l < logn; ++l) n += twiddle_entries(l);
  return n;
}
constexpr size_t kTwiddles = twiddle_offset(kMaxLogN + 1);

// Storage order of a spectrum in global memory. The frequency
//   k = k_1 + A (q_1 + R_1 (q_2 + R_2 (...)))
// of a transform is left in sub-row k_1, butterfly b = (q_1, ..., q_{m-1}) (q_1 most
// significant), output q_m of the last pass; it is stored at k_1 B + q_m (B / R_m) + b, so
// that the lanes of a warp (consecutive b) touch consecutive samples. The order is the same for
// both precisions and every row split (Geo::spec0).

}  // namespace mmp
