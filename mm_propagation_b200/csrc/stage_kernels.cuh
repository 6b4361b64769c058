// stage_kernels.cuh — the fused Lawson–RK stage kernels.
//
// The solver keeps the interaction-picture field in the FREQUENCY domain
// (psi_hat = FFT(psi), FP64). The reference keeps psi in the time domain and
// runs FFT -> *E_i -> IFFT on it in every stage
// (src/MultimodePropagation_CPU.cpp:114-119); since the FFT is linear,
// FFT(psi + h sum a_ij N_j) = psi_hat + h sum a_ij N_hat_j, so each stage needs
// one inverse transform per mode to get U and one forward transform per mode
// to turn sigma into N_hat, instead of two of each.
//
// One RK stage i of step n is, with Raman on and h_R a damped sinusoid (every workload),
// three launches; two with Raman off:
//   k_raman_agg    per time tile:   the Raman recurrence's aggregate over the tile for
//                                   every pair field V = U_l conj(U_m)
//   k_contract_sp  per time tile:   the state entering the tile from the aggregates of the tiles
//                                   before it (tile_carry; a response too long for that takes a
//                                   k_raman_carry launch), R through the tile, then
//                                   sigma_p = sum Q U_k [(1-fR) V_lm + R_lm] (all p)
//                  (k_contract_sr for tiles with too many pair fields to hold at once,
//                   k_contract_tc for dense Q on the tensor cores, k_contract for short tiles and
//                   the register-blocked dense form)
//   k_nu           per mode p:      FFT(sigma_p) -> N_hat_i = i sgn(gamma) conj(E_i) *.,
//                                   [last stage: psi_hat += h sum b_j N_hat_j, monitors],
//                                   x_hat = psi_hat + h sum a_{i+1,j} N_hat_j,
//                                   * E_{i+1} -> IFFT -> U for the next stage
// Any other h_R takes k_pair (V -> FFT -> * H_R -> IFFT = R, a row per pair field) instead of
// the first, and the contraction reads R as rows. k_prime makes U for stage 0 when a
// propagate call starts. E_i = exp(i Im L_p(w) z) is never stored: the phase
// Im L_p(w) * (z_n + c_i h) is evaluated in FP64, reduced in FP64 and only then passed
// to sin/cos in T.
#pragma once

#include <type_traits>

#include "fft.cuh"
#include "tc_sm100.cuh"

namespace mmp {

// One stage of the tableau as its k_nu needs it (host: stage_args). Stored N_hat_j entering
// x_hat of the next stage, or at the last stage psi_{n+1} = psi_n + h sum_j b_j N_j
// (src/MultimodePropagation_CPU.cpp:75-85), with their coefficients a or b; N_hat_i itself
// comes from registers (cself).
struct StageArgs {
  int stage;
  int last;  // 1: the final stage
  int nq;
  int jq[kMaxStages];
  double cq[kMaxStages];
  double cself;
  double c_this, c_next;  // z at this stage and the next, in steps beyond z_n
};

struct KParams {
  const SolveDesc* descs;
  const void* tw;    // twiddle table of the kernel's precision and size (radix_plan.h)
  StageArgs st;
};

// Im L_p(alpha) by Horner over the per-mode polynomial (FP64).
__device__ __forceinline__ double im_L(const double* poly, int nb, double alpha) {
  double r = poly[nb - 1];
  for (int j = nb - 2; j >= 0; --j) r = fma(r, alpha, poly[j]);
  return r;
}

// Small integer -> double without the conversion unit: the bits 0x43300000:(j + 2^31) are
// the double 2^52 + 2^31 + j (exact for |j| < 2^31), so one subtraction leaves j.
__device__ __forceinline__ double int_to_double(int j) {
  return __hiloint2double(0x43300000, (int)((unsigned)j ^ 0x80000000u)) - 4503601774854144.0;
}

__device__ __forceinline__ double alpha_of(int k, int nt, double alpha_scale) {
  // src/MultimodePropagation.cpp:167-171: index j <= nt/2 -> j, else j - nt
  const int kk = (k <= (nt >> 1)) ? k : k - nt;
  return alpha_scale * int_to_double(kk);
}

// exp(i theta) with theta reduced in FP64 (Cody–Waite with a two-part constant).
// FP32: reduced by pi/2 to x in [-pi/4, pi/4] and quadrant n mod 4 (n = theta 2/pi rounded
// by adding 1.5 * 2^52, whose ulp is 1: n and its low bits come out of one FMA, with
// no conversion instruction; valid for |theta 2/pi| < 2^51), then the Taylor
// series of sin and cos to x^9 and x^10 (truncation below 2e-9 on that interval),
// evaluated by Horner in x^2 in FP32; the quadrant swaps and negates. Short, branch-free
// code with no large-argument path (the argument is already small). FP64: the same reduction
// (a finite theta beyond its range ends on the unit circle too) and the series to x^17 and x^16
// (truncation below 1e-19 and 2.1e-18).
template <typename T> __device__ __forceinline__ c2<T> expi(double theta) {
  if constexpr (sizeof(T) == 4) {
    constexpr double k2OverPi = 0.63661977236758134308;
    constexpr double kHalfPiHi = 1.57079632679489655800;    // nearest double to pi/2
    constexpr double kHalfPiLo = 6.12323399573676603587e-17;  // pi/2 - kHalfPiHi
    constexpr double kRound = 6755399441055744.0;  // 1.5 * 2^52
    const double t = fma(theta, k2OverPi, kRound);
    const double n = t - kRound;
    const double r = fma(-n, kHalfPiLo, fma(-n, kHalfPiHi, theta));
    const float x = (float)r, x2 = x * x;
    // sin x = x (1 - x^2/3! + x^4/5! - x^6/7! + x^8/9!), cos x = 1 - x^2/2! + ... - x^10/10!
    const float sp =
        x * fmaf(x2, fmaf(x2, fmaf(x2, fmaf(x2, 1.0f / 362880.0f, -1.0f / 5040.0f), 1.0f / 120.0f), -1.0f / 6.0f), 1.0f);
    const float cp = fmaf(
        x2, fmaf(x2, fmaf(x2, fmaf(x2, fmaf(x2, -1.0f / 3628800.0f, 1.0f / 40320.0f), -1.0f / 720.0f), 1.0f / 24.0f),
                 -0.5f),
        1.0f);
    const int q = __double2loint(t) & 3;
    const float c = (q & 1) ? sp : cp, s = (q & 1) ? cp : sp;
    return make_float2((q == 1 || q == 2) ? -c : c, (q >= 2) ? -s : s);
  } else {
    constexpr double k2OverPi = 0.63661977236758134308;
    constexpr double kHalfPiHi = 1.57079632679489655800;
    constexpr double kHalfPiLo = 6.12323399573676603587e-17;
    constexpr double kRound = 6755399441055744.0;
    const double t = fma(theta, k2OverPi, kRound);
    const double n = t - kRound;
    double x = fma(-n, kHalfPiLo, fma(-n, kHalfPiHi, theta));
    x = fabs(x) > 1.0 ? 0.0 : x;  // |theta| > 3.5e15, whose own spacing is 0.5 or more: some point of the circle
    const double x2 = x * x;
    double sp = 1.0 / 355687428096000.0, cp = 1.0 / 20922789888000.0;  // 1/17!, 1/16!
    constexpr double sc[7] = {-1.0 / 1307674368000.0, 1.0 / 6227020800.0, -1.0 / 39916800.0, 1.0 / 362880.0,
                              -1.0 / 5040.0, 1.0 / 120.0, -1.0 / 6.0};
    constexpr double cc[7] = {-1.0 / 87178291200.0, 1.0 / 479001600.0, -1.0 / 3628800.0, 1.0 / 40320.0,
                              -1.0 / 720.0, 1.0 / 24.0, -0.5};
#pragma unroll
    for (int j = 0; j < 7; ++j) {
      sp = fma(sp, x2, sc[j]);
      cp = fma(cp, x2, cc[j]);
    }
    sp = fma(sp * x2, x, x);
    cp = fma(cp, x2, 1.0);
    const int q = __double2loint(t) & 3;
    const double c = (q & 1) ? sp : cp, s = (q & 1) ? cp : sp;
    return make_double2((q == 1 || q == 2) ? -c : c, (q >= 2) ? -s : s);
  }
}

template <typename T> __device__ __forceinline__ c2<T>* as_t2(void* p) { return reinterpret_cast<c2<T>*>(p); }
template <typename T> __device__ __forceinline__ const c2<T>* as_t2(const void* p) { return reinterpret_cast<const c2<T>*>(p); }

// two adjacent complex samples (one 16-byte access in FP32; p 16-byte aligned)
template <typename T>
__device__ __forceinline__ void ld2(const c2<T>* p, c2<T>& a, c2<T>& b) {
  a = p[0];
  b = p[1];
}
template <>
__device__ __forceinline__ void ld2<float>(const float2* p, float2& a, float2& b) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  a = make_float2(v.x, v.y);
  b = make_float2(v.z, v.w);
}
template <typename T>
__device__ __forceinline__ void st2(c2<T>* p, c2<T> a, c2<T> b) {
  p[0] = a;
  p[1] = b;
}
template <>
__device__ __forceinline__ void st2<float>(float2* p, float2 a, float2 b) {
  *reinterpret_cast<float4*>(p) = make_float4(a.x, a.y, b.x, b.y);
}

// The CTA copies its solve descriptor and mode p's dispersion polynomial into shared memory
// instead of every field becoming its own dependent global load. Published by the caller's
// next barrier.
static_assert(sizeof(SolveDesc) % 8 == 0, "descriptor copied in 8-byte words");
// a pointer field of a descriptor in global memory (constant while kernels run)
template <typename P> __device__ __forceinline__ P* ldg_ptr(P* const* f) {
  return reinterpret_cast<P*>(__ldg(reinterpret_cast<const unsigned long long*>(f)));
}
__device__ __forceinline__ void stage_desc(SolveDesc* dst, const SolveDesc* src) {
  constexpr int W = (int)(sizeof(SolveDesc) / 8);
  for (int i = threadIdx.x; i < W; i += blockDim.x)
    reinterpret_cast<unsigned long long*>(dst)[i] = __ldg(reinterpret_cast<const unsigned long long*>(src) + i);
}
__device__ __forceinline__ void stage_poly(double* poly, const SolveDesc* gd, int p) {
  const int nb = __ldg(&gd->n_beta);
  const double* src = ldg_ptr(&gd->poly);
  if ((int)threadIdx.x < nb) poly[threadIdx.x] = __ldg(src + p * nb + threadIdx.x);
}

// Ask the TMA engine to pull [p, p + bytes) into L2 without waiting for it
// (p 16-byte aligned, bytes a multiple of 16). Used to have a row ready in L2 by the
// time a kernel's epilogue reads it.
__device__ __forceinline__ void prefetch_l2(const void* p, unsigned bytes) {
  constexpr unsigned kPiece = 64u * 1024u;
  const char* c = static_cast<const char*>(p);
  for (unsigned off = 0; off < bytes; off += kPiece) {
    const unsigned n = bytes - off < kPiece ? bytes - off : kPiece;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(c + off), "r"(n) : "memory");
  }
}

// Programmatic dependent launch: the kernels of a step are launched to start while the one before
// them still runs (solver.cu, launch). What does not depend on it (descriptors, polynomials,
// terms: written only by copies, which order fully) is staged first; grid_sync_wait returns
// once the earlier kernel is complete and its writes are visible. Every CTA passes it before it
// reads a field or leaves, so that a kernel's completion implies that of all before it.
// grid_release lets the next kernel start; it stands late, before a kernel's last stores, so that
// the next one's waiting CTAs do not take SMs from kernels that could run.
__device__ __forceinline__ void grid_sync_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Ampere-style asynchronous copies global -> shared (both addresses aligned to the size),
// grouped and waited for per thread: the loads are in flight without holding registers.
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <typename G> __device__ __forceinline__ int cluster_rank() {
  if constexpr (G::C == 1) return 0;
  else return (int)cg::this_cluster().block_rank();
}

// A streamed value (used once by this kernel: kept out of L1, which holds the twiddles)
__device__ __forceinline__ float2 ld_stream(const float2* p) { return __ldcg(p); }
__device__ __forceinline__ double2 ld_stream(const double2* p) { return __ldcg(p); }

// Common names of a row kernel: this CTA's sub-rows and the thread's place in its own.
#define MMP_ROW_SETUP()                                              \
  extern __shared__ __align__(128) unsigned char smem_raw[];          \
  V* s = reinterpret_cast<V*>(smem_raw);                              \
  const int rank = cluster_rank<Gm>();                                \
  const int tid = threadIdx.x;                                        \
  const int u = tid % Gm::TPR, lrow = tid / Gm::TPR;                  \
  const int k1 = rank * Gm::RPC + lrow;                               \
  V* sr = s + lrow * Gm::RS;                                          \
  const int i0 = rank * Gm::NTHR + tid;

// Packed two-lane FMA and product (FP32: one instruction; each lane rounds as the scalar one does).
__device__ __forceinline__ float2 pk_fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 pk_mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ double2 pk_fma(double2 a, double2 b, double2 c) {
  return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}
__device__ __forceinline__ double2 pk_mul(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }

// The U rows a slot reads, and its value from their samples (common.cuh: V_q, or the
// real parts of two fields).
template <bool REAL> __device__ __forceinline__ int4 slot_rows(const SolveDesc& d, int s) {
  if constexpr (REAL) return __ldg(d.rpairs + s);
  const int2 lm = __ldg(d.pairs + s);
  return make_int4(lm.x, lm.y, 0, 0);
}
template <bool REAL, typename V> __device__ __forceinline__ V slot_value(V l0, V m0, V l1, V m1) {
  if constexpr (!REAL) return cmulc(l0, m0);
  V r;
  r.x = fma(l0.x, m0.x, l0.y * m0.y);
  r.y = fma(l1.x, m1.x, l1.y * m1.y);
  return r;
}

// ---- k_prime: U for stage 0 from psi_hat --------------------------------------------------
template <typename T, int LOGN, int XC>
__global__ void __launch_bounds__(Geo<T, LOGN, XC>::NTHR, Geo<T, LOGN, XC>::MIN_BLOCKS) k_prime(const KParams kp) {
  using Gm = Geo<T, LOGN, XC>;
  using V = c2<T>;
  MMP_ROW_SETUP();
  __shared__ double poly[kMaxBeta];
  __shared__ SolveDesc sdesc;
  const SolveDesc* gd = kp.descs + blockIdx.y;
  const int p = blockIdx.x / Gm::C;
  if (p >= __ldg(&gd->M)) return;  // uniform over the cluster
  stage_desc(&sdesc, gd);
  stage_poly(poly, gd, p);
  __syncthreads();
  const SolveDesc& d = sdesc;
  const V* tw = static_cast<const V*>(kp.tw);
  const unsigned long long n = __ldcg(d.step);
  const double zs = ((double)n + kp.st.c_this) * d.dz;
  const size_t row = (size_t)p * Gm::N;
  rows_last<Gm>(sr, u, [&](int b, V* x) {
    const double2* ps = d.psi_hat + row + Gm::spec0(k1, b);
    const int k0 = Gm::freq0(k1, b);
    V v[Gm::RM];
#pragma unroll
    for (int r = 0; r < Gm::RM; ++r) v[r] = from_d2<T>(__ldcg(ps + r * Gm::SSTR));
#pragma unroll
    for (int r = 0; r < Gm::RM; ++r) {
      const double th = im_L(poly, d.n_beta, alpha_of(k0 + r * Gm::KSTR, Gm::N, d.alpha_scale)) * zs;
      v[r] = cmul(v[r], expi<T>(th));
    }
    RegDFT<Gm::RM, true>::run(v);
#pragma unroll
    for (int r = 0; r < Gm::RM; ++r) x[Gm::pad(r)] = v[r];
  });
  rows_inv<Gm>(sr, tw, u);
  V v[Gm::E];
  row_last_inv<Gm>(v, s, tw, rank);
  V* U = as_t2<T>(d.U) + row + i0;
  const T inv = (T)d.inv_nt;
#pragma unroll
  for (int r = 0; r < Gm::E; ++r) U[r * Gm::B] = cscale(v[r], inv);
  row_leave<Gm>();
}

// ---- k_pair: R_q = IFFT(FFT(V_q) * H), V_q = U_l conj(U_m) -------------------------------
// One pair field per row (common.cuh: why never two).
template <typename T, int LOGN, int XC>
__global__ void __launch_bounds__(Geo<T, LOGN, XC>::NTHR, Geo<T, LOGN, XC>::MIN_BLOCKS) k_pair(const KParams kp) {
  using Gm = Geo<T, LOGN, XC>;
  using V = c2<T>;
  MMP_ROW_SETUP();
  const SolveDesc* gd = kp.descs + blockIdx.y;
  const int q = blockIdx.x / Gm::C;
  if (q >= __ldg(&gd->P)) {  // uniform over the cluster
    grid_sync_wait();
    return;
  }
  const unsigned long long* step = ldg_ptr(&gd->step);
  const V* U = as_t2<T>(static_cast<const void*>(ldg_ptr(&gd->U))) + i0;
  const V* H = as_t2<T>(static_cast<const void*>(ldg_ptr(&gd->H)));
  V* W = as_t2<T>(ldg_ptr(&gd->W));
  const int4 lm = slot_rows<false>(*gd, q);
  grid_sync_wait();
  if (__ldcg(step) >= __ldg(&gd->step_limit)) return;  // uniform over the cluster
  row_enter<Gm>();
  const V* tw = static_cast<const V*>(kp.tw);
  V v[Gm::E];
  {
    const V* Ul = U + (size_t)lm.x * Gm::N;
    const V* Um = U + (size_t)lm.y * Gm::N;
#pragma unroll
    for (int r = 0; r < Gm::E; ++r) v[r] = cmulc(ld_stream(Ul + r * Gm::B), ld_stream(Um + r * Gm::B));
  }
  row_first<Gm>(v, s, tw, rank);
  rows_fwd<Gm>(sr, tw, u);
  rows_last<Gm>(sr, u, [&](int b, V* x) {
    const V* h = H + Gm::spec0(k1, b);
    V w[Gm::RM];
#pragma unroll
    for (int r = 0; r < Gm::RM; ++r) w[r] = x[Gm::pad(r)];
    RegDFT<Gm::RM, false>::run(w);
#pragma unroll
    for (int r = 0; r < Gm::RM; ++r) w[r] = cmul(w[r], __ldg(h + r * Gm::SSTR));
    RegDFT<Gm::RM, true>::run(w);
#pragma unroll
    for (int r = 0; r < Gm::RM; ++r) x[Gm::pad(r)] = w[r];
  });
  rows_inv<Gm>(sr, tw, u);
  grid_release();
  row_last_inv<Gm>(v, s, tw, rank);
  // R_q = (H_R conv V_q); the Kerr part (1 - fR) V_q is formed by the contraction from
  // the U tile it already holds
  V* R = W + (size_t)q * Gm::N + i0;
#pragma unroll
  for (int r = 0; r < Gm::E; ++r) R[r * Gm::B] = v[r];
  row_leave<Gm>();
}

// ---- k_raman_scan: R_q = h_R (*) V_q as a periodic linear recurrence ----------------------
// Used instead of k_pair when the sampled Raman response is a damped sinusoid,
// h_i = Im(c lambda^i) for every i < NT (the model simulations/main.cpp:67-75 samples;
// the host checks the fit to 1e-10 of max|h|). With V = a + i b (a, b real) and
// w = Delta_t T0 f_R,
//   R[n] = w sum_i h_i V[(n - i) mod NT] = Im(kappa S_a[n]) + i Im(kappa S_b[n]),
//   S[n] = lambda S[n-1] + x[n]  (x = a or b, periodic in n), kappa = w c (1 - lambda^NT):
// the same circular convolution k_pair evaluates by FFT, in O(NT) per row.
// Each thread owns E consecutive samples in sub-chunks of 8. Sub-chunk scans run in T
// from zero; carries between sub-chunks and threads are FP64: a block-wide scan of
// the affine maps s -> A s + B (A = lambda^E) gives every thread the state entering its
// samples, and the periodic start S[-1] = S_lin[NT-1] / (1 - lambda^NT) closes the circle.
struct Affine {  // s -> a s + (ba, bb) for the two scans
  double2 a, ba, bb;
};
__device__ __forceinline__ Affine affine_then(const Affine& first, const Affine& second) {
  Affine r;
  r.a = cmul(first.a, second.a);
  r.ba = cadd(cmul(second.a, first.ba), second.ba);
  r.bb = cadd(cmul(second.a, first.bb), second.bb);
  return r;
}
__device__ __forceinline__ double2 shfl_up_d2(double2 v, int off, unsigned mask) {
  v.x = __shfl_up_sync(mask, v.x, off);
  v.y = __shfl_up_sync(mask, v.y, off);
  return v;
}
__device__ __forceinline__ Affine shfl_up_affine(const Affine& v, int off, unsigned mask) {
  Affine r;
  r.a = shfl_up_d2(v.a, off, mask);
  r.ba = shfl_up_d2(v.ba, off, mask);
  r.bb = shfl_up_d2(v.bb, off, mask);
  return r;
}
// inclusive scan over the lanes of a warp (lanes >= n hold identities)
__device__ __forceinline__ Affine warp_scan_affine(Affine v, int lane) {
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const Affine o = shfl_up_affine(v, off, 0xffffffffu);
    if (lane >= off) v = affine_then(o, v);
  }
  return v;
}

// Block-wide exclusive scan of the threads' maps (in thread order): returns the map of
// all earlier threads; *total receives the composition over the whole block.
__device__ __forceinline__ Affine affine_identity() {
  Affine r;
  r.a = make_double2(1.0, 0.0);
  r.ba = r.bb = make_double2(0.0, 0.0);
  return r;
}
// warp_tot holds 17 entries: per-warp totals, then (after the scan) per-warp exclusive
// prefixes in [0, 16) and the block total in [16].
__device__ __forceinline__ Affine block_scan_affine(const Affine& mine, Affine* warp_tot, Affine* total) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const Affine incl = warp_scan_affine(mine, lane);
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {  // one warp scans the warp totals
    const Affine wt = lane < nwarps ? warp_tot[lane] : affine_identity();
    const Affine wi = warp_scan_affine(wt, lane);
    Affine we = shfl_up_affine(wi, 1, 0xffffffffu);
    if (lane == 0) we = affine_identity();
    __syncwarp();
    if (lane < nwarps) warp_tot[lane] = we;
    if (lane == 31) warp_tot[16] = wi;
  }
  __syncthreads();
  const Affine wpre = warp_tot[warp];
  *total = warp_tot[16];
  Affine lpre = shfl_up_affine(incl, 1, 0xffffffffu);  // earlier lanes of this warp
  if (lane == 0) lpre = affine_identity();
  __syncthreads();  // warp_tot is reused by the next scan
  return affine_then(wpre, lpre);
}

// Rows are processed in segments of `seg` samples (the whole row when it fits the
// 128 KB staging buffer): V = U_l conj(U_m) of a segment is formed in shared memory from
// coalesced loads, every thread scans its E consecutive samples from there, and the
// outputs are written back in place and stored coalesced. With one segment the staged
// V serves both passes; with several, pass 1 records each segment's map and pass 2
// stages every segment again.
template <typename T>
__global__ void __launch_bounds__(512) k_raman_scan(const SolveDesc* __restrict__ descs, int nt, int seg) {
  using V = c2<T>;
  constexpr int kMaxSeg = 16;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  V* sv = reinterpret_cast<V*>(smem_raw);  // padded: element i at pad(i)
  __shared__ Affine warp_tot[17];
  __shared__ Affine seg_map[kMaxSeg];
  const SolveDesc& d = descs[blockIdx.y];
  const int q = blockIdx.x;
  grid_sync_wait();
  if (q >= d.P || __ldcg(d.step) >= d.step_limit) return;  // uniform over the CTA
  const int tid = threadIdx.x;
  const int nthr = blockDim.x;                   // 32..512, a power of two
  const int nseg = nt / seg;                     // <= kMaxSeg
  const int act = min(nthr, seg >> 3);           // threads that own samples
  const int E = seg / act;                       // a multiple of 8
  const int myE = tid < act ? E : 0;
  const int off = min(tid, act - 1) * E;
  const int2 lm = d.pairs[q];
  const V* Ul = as_t2<T>(d.U) + (size_t)lm.x * nt;
  const V* Um = as_t2<T>(d.U) + (size_t)lm.y * nt;
  V* R = as_t2<T>(d.W) + (size_t)q * nt;
  const double2 lam = d.iir_lambda;
  V pw[8];  // lambda^(k+1)
  double2 lam8;
  {
    double2 p = lam;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      pw[k] = from_d2<T>(p);
      lam8 = p;
      p = cmul(p, lam);
    }
  }
  const V lt = from_d2<T>(lam);
  // s <- lambda s + x for a real input x (two dependent FMAs per component)
  auto step = [&](V s, T x) {
    return mk<T>(fma(lt.x, s.x, fma(-lt.y, s.y, x)), fma(lt.x, s.y, lt.y * s.x));
  };
  // stage V of segment g into shared memory (coalesced: two samples per thread per load)
  auto stage = [&](int g) {
    const size_t base = (size_t)g * seg;
#pragma unroll 8
    for (int i2 = tid; i2 < (seg >> 1); i2 += nthr) {
      V ul0, ul1, um0, um1;
      ld2<T>(Ul + base + 2 * i2, ul0, ul1);
      ld2<T>(Um + base + 2 * i2, um0, um1);
      sv[pad(2 * i2)] = cmulc(ul0, um0);
      sv[pad(2 * i2 + 1)] = cmulc(ul1, um1);
    }
    __syncthreads();
  };
  // this thread's map s -> lambda^E s + (S_a, S_b) over its samples of the staged segment
  auto thread_map = [&]() {
    Affine mine;
    mine.a = make_double2(1.0, 0.0);
    mine.ba = make_double2(0.0, 0.0);
    mine.bb = make_double2(0.0, 0.0);
    for (int j = 0; j < myE; j += 8) {
      V la = mk<T>(0, 0), lb = mk<T>(0, 0);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const V x = sv[pad(off + j + k)];
        la = step(la, x.x);
        lb = step(lb, x.y);
      }
      mine.a = cmul(mine.a, lam8);
      mine.ba = cadd(cmul(lam8, mine.ba), to_d2(la));
      mine.bb = cadd(cmul(lam8, mine.bb), to_d2(lb));
    }
    return mine;
  };
  // pass 1: every segment's map (a single segment stays staged for pass 2)
  Affine pre, tot;
  for (int g = 0; g < nseg; ++g) {
    stage(g);
    pre = block_scan_affine(thread_map(), warp_tot, &tot);
    if (tid == 0) seg_map[g] = tot;
    if (nseg > 1) __syncthreads();  // the next segment overwrites sv
  }
  __syncthreads();
  // periodic start: S[-1] = S_lin[NT-1] / (1 - lambda^NT)
  Affine row;
  row.a = make_double2(1.0, 0.0);
  row.ba = row.bb = make_double2(0.0, 0.0);
  for (int g = 0; g < nseg; ++g) row = affine_then(row, seg_map[g]);
  const double2 inv = d.iir_inv_one_minus;
  double2 sa = cmul(row.ba, inv), sb = cmul(row.bb, inv);  // state entering segment 0
  const double2 kap = d.iir_kappa;
  const V kt = from_d2<T>(kap);
  grid_release();
  // pass 2: outputs R = Im(kappa s), s = local + lambda^(k+1) C within each sub-chunk
  for (int g = 0; g < nseg; ++g) {
    if (nseg > 1) {
      stage(g);
      pre = block_scan_affine(thread_map(), warp_tot, &tot);
    }
    double2 Ca = cadd(cmul(pre.a, sa), pre.ba);
    double2 Cb = cadd(cmul(pre.a, sb), pre.bb);
    for (int j = 0; j < myE; j += 8) {
      const V kca = from_d2<T>(cmul(kap, Ca)), kcb = from_d2<T>(cmul(kap, Cb));
      V la = mk<T>(0, 0), lb = mk<T>(0, 0);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        V& cell = sv[pad(off + j + k)];
        const V x = cell;
        la = step(la, x.x);
        lb = step(lb, x.y);
        // Im(kappa local) + Im(lambda^(k+1) kappa C)
        cell = mk<T>(fma(kt.x, la.y, fma(kt.y, la.x, fma(pw[k].x, kca.y, pw[k].y * kca.x))),
                     fma(kt.x, lb.y, fma(kt.y, lb.x, fma(pw[k].x, kcb.y, pw[k].y * kcb.x))));
      }
      Ca = cadd(cmul(lam8, Ca), to_d2(la));
      Cb = cadd(cmul(lam8, Cb), to_d2(lb));
    }
    __syncthreads();
    const size_t base = (size_t)g * seg;
    for (int i2 = tid; i2 < (seg >> 1); i2 += nthr) st2<T>(R + base + 2 * i2, sv[pad(2 * i2)], sv[pad(2 * i2 + 1)]);
    // state entering the next segment
    const double2 na = cadd(cmul(seg_map[g].a, sa), seg_map[g].ba);
    const double2 nb = cadd(cmul(seg_map[g].a, sb), seg_map[g].bb);
    sa = na;
    sb = nb;
    if (nseg > 1) __syncthreads();
  }
}

// ---- k_nu: sigma_p -> N_hat_i, final accumulation, next stage's U ------------------------
// BODY: the stage arithmetic of an intermediate stage that reads n stored N_hat_j terms
// (BODY = n), of a last stage that reads n (BODY = kNuLastBody + n), or of any stage (-1).
// The host launches the instantiation that matches each stage of its tableau (RK4: 0 at
// the intermediate stages, kNuLastBody + 3 at the last), so each kernel carries one body.
//
// What bounds it: instruction issue and shared memory, then the row's global traffic. sigma goes
// from global memory into the first pass's registers, the stage arithmetic runs between the
// forward and the inverse radix step of the last pass (straight in its registers where the
// radix is 4; else chunk by chunk through the thread's own shared positions, so that the code
// stays one short loop), and U leaves from the last pass's registers: two block- or
// cluster-wide barriers a stage. Measured on a B200, a launch, against Stockham passes with
// block barriers between them and one layout per cluster size:
//   192 rows of 16384, FP32, intermediate stage   64-69 -> 49-53 us, 22.6-25.2 -> 16.3-19.0
//                                                 million warp instructions
//   6 rows of 16384, FP32 (one solve)             30-39 -> 12-15 us (6 -> 48 CTAs)
//   6 rows of 8192, FP64, order 8                 35-49 -> 12-15 us (6 -> 48 CTAs)
//   1 row of 2048, FP32                           9.1 -> 5.9 us
//   56 rows of 65536, FP32                        170-217 -> 118-156 us
constexpr int kNuLastBody = 10;
template <typename T, int LOGN, int XC, int BODY>
__global__ void __launch_bounds__(Geo<T, LOGN, XC>::NTHR, Geo<T, LOGN, XC>::MIN_BLOCKS) k_nu(const KParams kp) {
  using Gm = Geo<T, LOGN, XC>;
  using V = c2<T>;
  MMP_ROW_SETUP();
  __shared__ double poly[kMaxBeta];
  __shared__ double red[2][32];
  __shared__ SolveDesc sdesc;
  const SolveDesc* gd = kp.descs + blockIdx.y;
  const int p = blockIdx.x / Gm::C;
  if (p >= __ldg(&gd->M)) {  // also an empty slot (its descriptor is zero); uniform over the cluster
    grid_sync_wait();
    return;
  }
  const unsigned long long* stepp = ldg_ptr(&gd->step);
  const unsigned long long* totalp = ldg_ptr(&gd->total);
  const V* sg = as_t2<T>(static_cast<const void*>(ldg_ptr(&gd->sigma))) + (size_t)p * Gm::N + i0;
  const unsigned long long limit = __ldg(&gd->step_limit);
  const double h = __ldg(&gd->dz);
  stage_desc(&sdesc, gd);
  stage_poly(poly, gd, p);
  grid_sync_wait();
  const unsigned long long n_step = __ldcg(stepp), n_total = __ldcg(totalp);
  V v[Gm::E];
#pragma unroll
  for (int r = 0; r < Gm::E; ++r) v[r] = ld_stream(sg + r * Gm::B);
  // a specialised BODY serves intermediate or last stages only: fixed at compile time, so
  // each instantiation carries only its half of the stage arithmetic
  const bool last = BODY < 0 ? kp.st.last != 0 : (BODY >= kNuLastBody);
  {
    // the row's psi_hat (FP64 at the last stage, in T at the others), 1/C of it per CTA (the
    // part the CTA reads), on its way to L2 while the forward passes run, one piece of at
    // most 32 KB per thread. The N_hat_j are not prefetched: a wave's rows of them do not
    // fit in L2 beside the rest.
    const unsigned esz = last ? (unsigned)sizeof(double2) : (unsigned)sizeof(V);
    const unsigned bytes = Gm::NL * esz;
    const unsigned piece = bytes < 32u * 1024u ? bytes : 32u * 1024u;
    const void* src = last ? static_cast<const void*>(ldg_ptr(&gd->psi_hat)) : static_cast<const void*>(ldg_ptr(&gd->psi_t));
    const char* base = static_cast<const char*>(src) + ((size_t)p * Gm::N + (size_t)rank * Gm::NL) * esz;
    for (unsigned t = tid; t < bytes / piece; t += Gm::NTHR) prefetch_l2(base + (size_t)t * piece, piece);
  }
  if (n_step >= limit) return;  // finished solve; uniform over the cluster
  row_enter<Gm>();
  const V* tw = static_cast<const V*>(kp.tw);
  row_first<Gm>(v, s, tw, rank);  // its barrier publishes the descriptor and the polynomial
  rows_fwd<Gm>(sr, tw, u);
  const SolveDesc& d = sdesc;
  const int i = kp.st.stage;
  const size_t row = (size_t)p * Gm::N;
  const size_t mstride = (size_t)d.M * Gm::N;
  // FP32 stage bodies of one kind read psi_hat's T copy at the intermediate stages; the
  // FP64 ones (psi_t is psi_hat) and the any-stage body read psi_hat
  constexpr bool kReadT = sizeof(T) == 4 && BODY >= 0;
  const double zi = ((double)n_step + kp.st.c_this) * h, znext = ((double)n_step + kp.st.c_next) * h;
  double e_part = 0.0, p_part = 0.0;
  float p_part_f = 0.0f;
  bool finite = true;
  const double cself = kp.st.cself * h;
  // E_{i+1} = E_i when z does not move between the stages (RK4: c_2 = c_3, c_4 = 1)
  const bool same_z = zi == znext;
  const float w0f = (float)d.omega0_T0, asf = (float)d.alpha_scale;
  const bool nb3 = d.n_beta == 3;
  // stored terms: their count at compile time, or (any-stage body) at run time
  constexpr int NQ = BODY < 0 ? -1 : (BODY >= kNuLastBody ? BODY - kNuLastBody : BODY);
  constexpr int NQR = NQ > 0 ? NQ : 1;
  double cq[NQR];
#pragma unroll
  for (int q = 0; q < NQR; ++q) cq[q] = NQ > 0 ? kp.st.cq[q] * h : 0.0;
  // frequencies per chunk: a chunk's loads are all in flight before its arithmetic
  constexpr int CHK0 = NQ <= (sizeof(T) == 8 ? 0 : 2) ? 4 : 2;
  constexpr int CHK = CHK0 < Gm::RM ? CHK0 : Gm::RM;
  rows_last<Gm>(sr, u, [&](int b, V* x) {
    const size_t at = row + Gm::spec0(k1, b);
    const int k0 = Gm::freq0(k1, b);
    double2 ps[CHK];  // last stage (and FP64): psi_hat in FP64
    V pt[CHK];        // other stages: psi_hat in T
    V nj[CHK][NQR];
    auto fetch = [&](int c0) {
#pragma unroll
      for (int c = 0; c < CHK; ++c) {
        const size_t f = at + (c0 + c) * Gm::SSTR;
        if (!kReadT || last) ps[c] = __ldcg(d.psi_hat + f);
        else pt[c] = __ldcg(as_t2<T>(d.psi_t) + f);
        if constexpr (NQ > 0) {
#pragma unroll
          for (int q = 0; q < NQ; ++q) nj[c][q] = __ldcg(as_t2<T>(d.Nh) + (size_t)kp.st.jq[q] * mstride + f);
        }
      }
    };
    // the chunk's values w become the spectrum entering the inverse
    auto chunk = [&](V* w, int c0) {
#pragma unroll
      for (int c = 0; c < CHK; ++c) {
        const int r = c0 + c;
        const size_t f = at + r * Gm::SSTR;
        const int k = k0 + r * Gm::KSTR;
        const double alpha = alpha_of(k, Gm::N, d.alpha_scale);
        const double L = nb3 ? fma(fma(poly[2], alpha, poly[1]), alpha, poly[0]) : im_L(poly, d.n_beta, alpha);
        // N_hat_i = i sgn(gamma) conj(E_i) FFT(sigma)   (src/MultimodePropagation_CPU.cpp:231-237)
        const V ei = expi<T>(L * zi);
        const V xe = cmulc(w[c], ei);
        V nh;
        nh.x = (T)(-d.sgn_gamma) * xe.y;
        nh.y = (T)(d.sgn_gamma) * xe.x;
        as_t2<T>(d.Nh)[(size_t)i * mstride + f] = nh;
        V xt;
        if (last || BODY < 0) {
          // FP32 bodies of the last stage: the increment h sum_j b_j N_j is formed in FP32 from
          // the FP32 N_j (its rounding is that of the N_j themselves); psi_{n+1} = psi_n + inc
          // in FP64. FP64 and the any-stage body accumulate in FP64 throughout.
          double2 y = ps[c];
          if constexpr (sizeof(T) == 4 && BODY >= 0) {
            V inc = mk<T>((T)cself * nh.x, (T)cself * nh.y);
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
              inc.x = fma((T)cq[q], nj[c][q].x, inc.x);
              inc.y = fma((T)cq[q], nj[c][q].y, inc.y);
            }
            y = make_double2(y.x + (double)inc.x, y.y + (double)inc.y);
          } else {
            const double2 nhd = to_d2(nh);
            y.x = fma(cself, nhd.x, y.x);
            y.y = fma(cself, nhd.y, y.y);
            if constexpr (NQ >= 0) {
#pragma unroll
              for (int q = 0; q < NQ; ++q) {
                const double2 nv = to_d2(nj[c][q]);
                y.x = fma(cq[q], nv.x, y.x);
                y.y = fma(cq[q], nv.y, y.y);
              }
            } else {
              for (int q = 0; q < kp.st.nq; ++q) {
                const double2 nv = to_d2(__ldcg(as_t2<T>(d.Nh) + (size_t)kp.st.jq[q] * mstride + f));
                const double cr = kp.st.cq[q] * h;
                y.x = fma(cr, nv.x, y.x);
                y.y = fma(cr, nv.y, y.y);
              }
            }
          }
          xt = from_d2<T>(y);
          if (last) {
            d.psi_hat[f] = y;
            if constexpr (sizeof(T) == 4) as_t2<T>(d.psi_t)[f] = xt;
            const double a2 = y.x * y.x + y.y * y.y;
            finite = finite && isfinite(a2);
            e_part += a2;
            if constexpr (sizeof(T) == 4) {
              // photon monitor in FP32 (per-thread partial sums; FP64 across threads)
              if (w0f != 0.0f) {
                const int kk = (k <= (Gm::N >> 1)) ? k : k - Gm::N;
                const float af = __int_as_float(0x4B400000 + kk) - 12582912.0f;  // kk as float, exact
                p_part_f += __fdividef(xt.x * xt.x + xt.y * xt.y, fmaf(asf, af, w0f));
              }
            } else {
              if (d.omega0_T0 != 0.0) p_part += a2 / (d.omega0_T0 + alpha);
            }
          }
        } else {
          if constexpr (!kReadT) xt = from_d2<T>(ps[c]);
          else xt = pt[c];  // = psi_hat rounded to T
          const T cs = (T)cself;
          xt.x = fma(cs, nh.x, xt.x);
          xt.y = fma(cs, nh.y, xt.y);
          if constexpr (NQ > 0) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
              xt.x = fma((T)cq[q], nj[c][q].x, xt.x);
              xt.y = fma((T)cq[q], nj[c][q].y, xt.y);
            }
          }
        }
        V en;
        if (same_z) en = ei;
        else en = expi<T>(L * znext);
        w[c] = cmul(xt, en);
      }
    };
    V w[Gm::RM];
    fetch(0);
#pragma unroll
    for (int r = 0; r < Gm::RM; ++r) w[r] = x[Gm::pad(r)];
    RegDFT<Gm::RM, false>::run(w);
    if constexpr (CHK == Gm::RM) {
      chunk(w, 0);
    } else {
      // through the thread's own positions in shared memory: a loop with one body, whose
      // registers hold one chunk
#pragma unroll
      for (int r = 0; r < Gm::RM; ++r) x[Gm::pad(r)] = w[r];
#pragma unroll 1
      for (int c0 = 0; c0 < Gm::RM; c0 += CHK) {
        V wc[CHK];
        if (c0 > 0) fetch(c0);
#pragma unroll
        for (int c = 0; c < CHK; ++c) wc[c] = x[Gm::pad(c0) + c];
        chunk(wc, c0);
#pragma unroll
        for (int c = 0; c < CHK; ++c) x[Gm::pad(c0) + c] = wc[c];
      }
#pragma unroll
      for (int r = 0; r < Gm::RM; ++r) w[r] = x[Gm::pad(r)];
    }
    RegDFT<Gm::RM, true>::run(w);
#pragma unroll
    for (int r = 0; r < Gm::RM; ++r) x[Gm::pad(r)] = w[r];
  });
  p_part += (double)p_part_f;
  if (last) {
    // Block reduction of the monitors, then the last CTA of this solve advances the
    // step. Done before the inverse passes, so none of it is live across them; every CTA of
    // the solve has read the step counter, and the next launch's reads follow this launch.
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      e_part += __shfl_xor_sync(0xffffffffu, e_part, o);
      p_part += __shfl_xor_sync(0xffffffffu, p_part, o);
    }
    const int finite_all = __syncthreads_and(finite ? 1 : 0);
    if ((tid & 31) == 0) { red[0][tid >> 5] = e_part; red[1][tid >> 5] = p_part; }
    __syncthreads();
    if (tid == 0) {
      double es = 0.0, ps = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { es += red[0][w]; ps += red[1][w]; }
      if (!finite_all) atomicOr(d.status, kStatusNonFinite);
      if (d.monitors && n_total < d.mon_cap) {
        atomicAdd(&d.energy[n_total], es * d.energy_scale);
        if (d.omega0_T0 != 0.0) atomicAdd(&d.photons[n_total], ps * d.photon_scale);
      }
      __threadfence();
      const unsigned prev = atomicAdd(d.done_ctr, 1u);
      if (prev == (unsigned)(d.M * Gm::C) - 1u) {
        *d.done_ctr = 0u;
        *d.step = n_step + 1;
        *d.total = n_total + 1;
        if (d.drift_tol > 0.0 && d.monitors && n_total < d.mon_cap) {
          // every CTA's energy sum is in (their adds precede their counter increments)
          const double en = __ldcg(&d.energy[n_total]), e0 = *d.drift_ref;
          if (e0 == 0.0) *d.drift_ref = en;
          else if (!(fabs(en - e0) <= d.drift_tol * e0)) atomicOr(d.status, kStatusDrift);
        }
        __threadfence();
      }
    }
  }
  rows_inv<Gm>(sr, tw, u);
  grid_release();
  row_last_inv<Gm>(v, s, tw, rank);
  V* U = as_t2<T>(d.U) + row + i0;
  const T inv = (T)d.inv_nt;
#pragma unroll
  for (int r = 0; r < Gm::E; ++r) U[r * Gm::B] = cscale(v[r], inv);
  row_leave<Gm>();
}

// ---- k_result: phi_p = IFFT(exp(L_p z) psi_hat_p) / conversion_factor -> io (FP64) --------
// In FP64 whatever the solve's precision: psi_hat's order is the same.
template <typename T, int LOGN, int XC>
__global__ void __launch_bounds__(Geo<T, LOGN, XC>::NTHR, Geo<T, LOGN, XC>::MIN_BLOCKS) k_result(const KParams kp) {
  using Gm = Geo<T, LOGN, XC>;
  using V = c2<T>;
  MMP_ROW_SETUP();
  __shared__ double poly[kMaxBeta];
  __shared__ SolveDesc sdesc;
  const SolveDesc* gd = kp.descs + blockIdx.y;
  const int p = blockIdx.x / Gm::C;
  if (p >= __ldg(&gd->M)) return;  // uniform over the cluster
  stage_desc(&sdesc, gd);
  stage_poly(poly, gd, p);
  __syncthreads();
  const SolveDesc& d = sdesc;
  const V* tw = static_cast<const V*>(kp.tw);
  const unsigned long long n = __ldcg(d.step);
  const double z = (double)n * d.dz;
  const size_t row = (size_t)p * Gm::N;
  rows_last<Gm>(sr, u, [&](int b, V* x) {
    const double2* ps = d.psi_hat + row + Gm::spec0(k1, b);
    const int k0 = Gm::freq0(k1, b);
    V w[Gm::RM];
#pragma unroll
    for (int r = 0; r < Gm::RM; ++r) w[r] = from_d2<T>(__ldcg(ps + r * Gm::SSTR));
#pragma unroll
    for (int r = 0; r < Gm::RM; ++r) {
      const double th = im_L(poly, d.n_beta, alpha_of(k0 + r * Gm::KSTR, Gm::N, d.alpha_scale)) * z;
      w[r] = cmul(w[r], expi<T>(th));
    }
    RegDFT<Gm::RM, true>::run(w);
#pragma unroll
    for (int r = 0; r < Gm::RM; ++r) x[Gm::pad(r)] = w[r];
  });
  rows_inv<Gm>(sr, tw, u);
  V v[Gm::E];
  row_last_inv<Gm>(v, s, tw, rank);
  double2* io = d.io + row + i0;
#pragma unroll
  for (int r = 0; r < Gm::E; ++r) {
    const double2 y = to_d2(v[r]);
    io[r * Gm::B] = make_double2(y.x * d.result_scale, y.y * d.result_scale);
  }
  row_leave<Gm>();
}

// ---- k_dft: rows of FP64 samples -> transform in precision T -> rows of FP64 -------------
// Forward (INV=false): out = scale * FFT(in), in a solve's order or (natural) by frequency. Inverse (natural order
// in): out = scale * sum_k in[k] e^{+...}. in may be out: a row is read whole before a
// barrier after which it is written.
struct DftArgs {
  const double2* in;
  double2* out;
  int rows;
  int natural;
  double scale;
  const void* tw;
  // forward, where not null: the spectrum in single precision too, and a solve's counters to
  // clear (step, status, drift reference), so that new fields take one launch
  float2* out_t;
  unsigned long long* restart;
};

template <typename T, int LOGN, int XC, bool INV>
__global__ void __launch_bounds__(Geo<T, LOGN, XC>::NTHR, Geo<T, LOGN, XC>::MIN_BLOCKS) k_dft(const DftArgs a) {
  using Gm = Geo<T, LOGN, XC>;
  using V = c2<T>;
  MMP_ROW_SETUP();
  const int p = blockIdx.x / Gm::C;
  if (p >= a.rows) return;
  const V* tw = static_cast<const V*>(a.tw);
  const size_t row = (size_t)p * Gm::N;
  V v[Gm::E];
  if constexpr (!INV) {
    if (a.restart && blockIdx.x == 0 && threadIdx.x == 0) {
      a.restart[0] = 0;
      *reinterpret_cast<int*>(a.restart + 3) = 0;
      a.restart[4] = 0;
    }
    row_enter<Gm>();
#pragma unroll
    for (int r = 0; r < Gm::E; ++r) v[r] = from_d2<T>(__ldcg(a.in + row + i0 + r * Gm::B));
    row_first<Gm>(v, s, tw, rank);
    rows_fwd<Gm>(sr, tw, u);
    rows_last<Gm>(sr, u, [&](int b, V* x) {
      const int at0 = a.natural ? Gm::freq0(k1, b) : Gm::spec0(k1, b), step = a.natural ? Gm::KSTR : Gm::SSTR;
      V w[Gm::RM];
#pragma unroll
      for (int r = 0; r < Gm::RM; ++r) w[r] = x[Gm::pad(r)];
      RegDFT<Gm::RM, false>::run(w);
#pragma unroll
      for (int r = 0; r < Gm::RM; ++r) {
        const double2 y = to_d2(w[r]), z = make_double2(y.x * a.scale, y.y * a.scale);
        const size_t at = row + at0 + r * step;
        a.out[at] = z;
        if (a.out_t) a.out_t[at] = make_float2((float)z.x, (float)z.y);
      }
    });
    // no peer's shared memory is touched after row_first
  } else {
    rows_last<Gm>(sr, u, [&](int b, V* x) {
      const int k0 = Gm::freq0(k1, b);
      V w[Gm::RM];
#pragma unroll
      for (int r = 0; r < Gm::RM; ++r) w[r] = from_d2<T>(__ldcg(a.in + row + k0 + r * Gm::KSTR));
      RegDFT<Gm::RM, true>::run(w);
#pragma unroll
      for (int r = 0; r < Gm::RM; ++r) x[Gm::pad(r)] = w[r];
    });
    rows_inv<Gm>(sr, tw, u);
    row_last_inv<Gm>(v, s, tw, rank);
#pragma unroll
    for (int r = 0; r < Gm::E; ++r) {
      const double2 y = to_d2(v[r]);
      a.out[row + i0 + r * Gm::B] = make_double2(y.x * a.scale, y.y * a.scale);
    }
    row_leave<Gm>();
  }
}

// ---- bulk-async copies (TMA engine) into shared memory, completing on an mbarrier -------
__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}
// global -> this CTA's shared memory; dst, src 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}
// Wait for phase `parity` of the mbarrier, giving up after `max_iter` polls.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, unsigned max_iter) {
  const unsigned a = smem_addr(bar);
  for (unsigned it = 0; it < max_iter; ++it) {
    unsigned done;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
constexpr unsigned kMaxWaitPolls = 1u << 24;  // far above any copy time; then report, not hang

// ---- the Raman recurrence inside a contraction tile ---------------------------------------
// With h_R a damped sinusoid (see k_raman_scan) the pair fields' convolutions need no
// row pass at all: per tile of TT = 32 c samples (2 <= c <= 8)
//   k_raman_agg    the recurrence's aggregate over the tile from a zero start,
//   k_raman_carry  per pair row, a scan of the tile aggregates (periodic start): the
//                  state entering every tile,
//   k_contract     (mode 2) runs the recurrence through its own tile from that state
//                  and forms W = (1 - f_R) V + R in shared memory; R never leaves the SM.
// Within a tile one warp handles one pair field at a time, lane L owning samples
// [c L, c L + c). The pair field row is written once, coalesced, in a swizzled layout
// (wsw) in which a lane's c samples are also conflict-free 16-byte loads; the lane keeps
// them in registers through the scan and writes W back in place, in the same layout.
template <typename T> struct TileScan {
  using V = c2<T>;
  V lt, kt;
  V rw[8];      // lambda^(c-1-k): weights of the lane's local aggregate
  V lvl[5];     // lambda^(c 2^j): the multipliers of the lane scan's levels
  V lane_pow;   // lambda^(c lane): carries the tile's entering state to this lane
  int c;
  __device__ __forceinline__ void init(const SolveDesc& d, int c_, int lane) {
    c = c_;
    const double2 lam = d.iir_lambda;
    lt = from_d2<T>(lam);
    kt = from_d2<T>(d.iir_kappa);
    double2 p = make_double2(1.0, 0.0);
#pragma unroll
    for (int k = 7; k >= 0; --k) {
      rw[k] = from_d2<T>(p);
      if (k < c) p = cmul(p, lam);
    }
    // p = lambda^c
    double2 lp = make_double2(1.0, 0.0);
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      lvl[j] = from_d2<T>(p);
      if ((lane >> j) & 1) lp = cmul(lp, p);
      p = cmul(p, p);
    }
    lane_pow = from_d2<T>(lp);
  }
  // inclusive scan over the lanes of (la, lb): s_L = lambda^c s_{L-1} + local_L
  __device__ __forceinline__ void lane_scan(V& a, V& b, int lane) const {
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      const int o = 1 << j;
      V pa, pb;
      pa.x = __shfl_up_sync(0xffffffffu, a.x, o);
      pa.y = __shfl_up_sync(0xffffffffu, a.y, o);
      pb.x = __shfl_up_sync(0xffffffffu, b.x, o);
      pb.y = __shfl_up_sync(0xffffffffu, b.y, o);
      if (lane >= o) {
        a = cadd(cmul(lvl[j], pa), a);
        b = cadd(cmul(lvl[j], pb), b);
      }
    }
  }
  __device__ __forceinline__ V step(V s, T x) const {
    return mk<T>(fma(lt.x, s.x, fma(-lt.y, s.y, x)), fma(lt.x, s.y, lt.y * s.x));
  }
};

// Position of the sample pair (2h, 2h + 1) in a pair-field row of the contraction tile:
// 16-byte chunk h ^ ((h >> 3) & mask). With mask = TT/64 - 1 (TT = 128, 256) both a
// warp's 32 consecutive chunks and lane L's chunks [g L, g L + g) (g = TT/64) fall on
// distinct banks per quarter warp; mask 0 is the plain layout.
__device__ __forceinline__ int wsw(int h, int mask) { return h ^ ((h >> 3) & mask); }

// The state entering tile `tile` for idx = 2 s (real part of slot s) or 2 s + 1 (imaginary part).
// look = 0: k_raman_carry has left it in the aggregates' place. Else it is summed here from the
// aggregates of the `look` tiles before (around the period),
//   C = sum_{i=1..look} lambda^(TT (i-1)) A_{tile-i}     [times 1 / (1 - lambda^NT) over a whole row],
// in FP64: what lies further back is below rounding. Measured on a B200 against a launch of
// k_raman_carry per stage (microseconds a step): 6 modes of 16384 98 -> 91, 2 of 4096 in FP64
// 65 -> 59, 1 of 2048 48 -> 44 (RK4, one solve); 3 solves of 10 x 32768 261 -> 257; 8 of the
// 28-mode order-6 solves 6450 -> 6394.
// The aggregates lie [tile][q][2] for that, and [q][tile][2] where k_raman_carry scans them.
template <typename T>
__device__ __forceinline__ c2<T> tile_carry(const SolveDesc& d, int slots, int ntiles, int tile, int idx, int look,
                                            double2 lamT) {
  using V = c2<T>;
  const V* tiles = as_t2<T>(static_cast<const void*>(d.raman_tiles));
  if (look == 0) return __ldcg(tiles + ((size_t)(idx >> 1) * ntiles + tile) * 2 + (idx & 1));
  const size_t P2 = 2 * (size_t)slots;
  tiles += idx;
  double2 c = make_double2(0.0, 0.0);
  for (int i0 = look; i0 > 0; i0 -= 4) {  // the farthest first, four loads in flight
    V a[4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (i0 - e > 0) a[e] = __ldcg(tiles + (size_t)((tile - (i0 - e) + ntiles) & (ntiles - 1)) * P2);
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (i0 - e > 0) c = cadd(cmul(lamT, c), to_d2(a[e]));
  }
  if (look == ntiles) c = cmul(c, d.iir_inv_one_minus);
  return from_d2<T>(c);
}
__device__ __forceinline__ double2 lambda_tile(const SolveDesc& d, int TT) {  // lambda^TT, TT = 64, 128, 256
  return TT == 256 ? d.iir_lam256 : TT == 128 ? d.iir_lam128 : d.iir_lam64;
}
// Tiles a solve looks back: all of a short row's.
__device__ __forceinline__ int tile_look(const SolveDesc& d, int ntiles, int TT, int raman_mode) {
  return raman_mode == 3 ? min((d.iir_len + TT - 1) / TT, ntiles) : 0;
}

// The states entering tile `tile` for every slot into shared memory, [s][2]; published by the
// caller's next barrier.
template <typename T>
__device__ __forceinline__ void stage_tile_carries(c2<T>* sC, const SolveDesc& d, int slots, int ntiles, int tile,
                                                   int look, double2 lamT) {
  for (int i = threadIdx.x; i < 2 * slots; i += blockDim.x) sC[i] = tile_carry<T>(d, slots, ntiles, tile, i, look, lamT);
}

// The recurrence through one pair field of a contraction tile, by one warp (TT = 32 c
// samples, 64 <= TT <= 256): V = U_l conj(U_m) is written coalesced to row (pair positions
// swizzled by wmask), each lane takes its c samples into registers, the lanes' aggregates
// are scanned, every lane runs the recurrence from the state entering it (carry[0..1]: the
// states entering the tile for Re V and Im V) and writes W = (1 - f_R) V + R for its samples
// c lane .. c lane + c - 1 back into row, in place. One slot (REAL: two pair fields).
template <typename T, bool REAL>
__device__ __forceinline__ void tile_pair_recurrence(const TileScan<T>& ts, const c2<T>* sU, int TT, int4 lm,
                                                     c2<T>* row, int wmask, const c2<T>* carry, T kerr, int lane) {
  using V = c2<T>;
  const int H = TT >> 1, c = ts.c, g = c >> 1;
  V x[8];
  // V = U_l conj(U_m), coalesced over the sample pairs, then each lane's own samples
  for (int h = lane; h < H; h += 32) {
    V ul0, ul1, um0, um1, vl0 = {}, vl1 = {}, vm0 = {}, vm1 = {};
    ld2<T>(sU + lm.x * TT + 2 * h, ul0, ul1);
    ld2<T>(sU + lm.y * TT + 2 * h, um0, um1);
    if constexpr (REAL) {
      ld2<T>(sU + lm.z * TT + 2 * h, vl0, vl1);
      ld2<T>(sU + lm.w * TT + 2 * h, vm0, vm1);
    }
    st2<T>(row + 2 * wsw(h, wmask), slot_value<REAL>(ul0, um0, vl0, vm0), slot_value<REAL>(ul1, um1, vl1, vm1));
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (j < g) ld2<T>(row + 2 * wsw(g * lane + j, wmask), x[2 * j], x[2 * j + 1]);
  // this lane's aggregate from a zero start: sum_k lambda^(c-1-k) x_k, x_k = Re or Im V
  V la = mk<T>(0, 0), lb = mk<T>(0, 0);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (k < c) {
      la = mk<T>(fma(ts.rw[k].x, x[k].x, la.x), fma(ts.rw[k].y, x[k].x, la.y));
      lb = mk<T>(fma(ts.rw[k].x, x[k].y, lb.x), fma(ts.rw[k].y, x[k].y, lb.y));
    }
  }
  ts.lane_scan(la, lb, lane);
  // state entering this lane's samples: lambda^(c lane) C_tile + earlier lanes
  V ea, eb;
  ea.x = __shfl_up_sync(0xffffffffu, la.x, 1);
  ea.y = __shfl_up_sync(0xffffffffu, la.y, 1);
  eb.x = __shfl_up_sync(0xffffffffu, lb.x, 1);
  eb.y = __shfl_up_sync(0xffffffffu, lb.y, 1);
  if (lane == 0) ea = eb = mk<T>(0, 0);
  V sa = cadd(cmul(ts.lane_pow, carry[0]), ea);
  V sb = cadd(cmul(ts.lane_pow, carry[1]), eb);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (k < c) {
      sa = ts.step(sa, x[k].x);
      sb = ts.step(sb, x[k].y);
      // R = Im(kappa S), W = (1 - f_R) V + R
      x[k] = mk<T>(fma(kerr, x[k].x, fma(ts.kt.x, sa.y, ts.kt.y * sa.x)),
                   fma(kerr, x[k].y, fma(ts.kt.x, sb.y, ts.kt.y * sb.x)));
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (j < g) st2<T>(row + 2 * wsw(g * lane + j, wmask), x[2 * j], x[2 * j + 1]);
}

// k_raman_agg: the recurrence's aggregate over a tile from a zero start, for every slot, as
// a weighted sum,
//   S_end = sum_t lambda^(TT-1-t) x_t   (x = Re or Im of U_l conj(U_m)),
// so it needs no sequential pass. A warp takes a field at a time: each lane sums its sample pairs
// (2h, 2h + 1), h = lane, lane + 32, ..., with the weights it keeps in registers, and the lanes'
// four sums are added by halving (each exchange hands over half of what a lane holds: 6
// shuffles for the four). What bounds it: the latency of the tile's copy, then issue. Measured
// on a B200, 32 solves of 6 x 16384, against weights read per field and 20 shuffles: 21 -> 18 us.
template <typename T, bool REAL>
__global__ void __launch_bounds__(256, (sizeof(T) == 4 ? 5 : 3)) k_raman_agg(const SolveDesc* __restrict__ descs, int nt, int TT, int by_tile) {
  using V = c2<T>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const SolveDesc& d = descs[blockIdx.y];
  const int tile = blockIdx.x, t0 = tile * TT;
  if (t0 >= nt || d.M == 0 || d.real != REAL) {  // empty slot, other form
    grid_sync_wait();
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int M = d.M, P = slot_count<REAL>(d.P);
  V* sU = reinterpret_cast<V*>(smem_raw);  // [M][TT]
  const V* U = as_t2<T>(d.U) + t0;
  V w0[4], w1[4];  // the weights of the lane's pairs
  {
    const V* pw = static_cast<const V*>(d.raman_pow) + TT - 2;
#pragma unroll
    for (int j = 0; j < 4; ++j)  // lambda^(TT-2-2h) for sample 2h + 1, lambda^(TT-1-2h) for 2h
      if (j < (TT >> 6)) ld2<T>(pw - 2 * (lane + 32 * j), w1[j], w0[j]);
  }
  grid_sync_wait();
  {  // the U tile as 16-byte asynchronous copies, before the step check
    constexpr int PER = 16 / (int)sizeof(V);  // samples a copy
    const int per_row = TT / PER, sh = 31 - __clz(per_row);
    for (int idx = threadIdx.x; idx < M * per_row; idx += blockDim.x) {
      const int r = idx >> sh, c = idx & (per_row - 1);
      cp_async16(sU + (size_t)r * TT + c * PER, U + (size_t)r * nt + c * PER);
    }
    cp_async_commit();
  }
  if (__ldcg(d.step) >= d.step_limit) {  // finished solve: the copies land before the CTA leaves
    cp_async_wait<0>();
    return;
  }
  cp_async_wait<0>();
  __syncthreads();
  grid_release();
  T* out = static_cast<T*>(d.raman_tiles) + (size_t)tile * (by_tile ? 4 * P : 4);
  const size_t sq = by_tile ? 4 : 4 * (size_t)(nt / TT);
  for (int q = warp; q < P; q += nwarps) {
    const int4 lm = slot_rows<REAL>(d, q);
    const V* ul = sU + lm.x * TT + 2 * lane;
    const V* um = sU + lm.y * TT + 2 * lane;
    const V* vl = sU + lm.z * TT + 2 * lane;
    const V* vm = sU + lm.w * TT + 2 * lane;
    V sr = mk<T>(0, 0), si = mk<T>(0, 0);  // Re and Im of the sums for (Re V, Im V)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (j < (TT >> 6)) {
        V ul0, ul1, um0, um1, vl0 = {}, vl1 = {}, vm0 = {}, vm1 = {};
        ld2<T>(ul + 64 * j, ul0, ul1);
        ld2<T>(um + 64 * j, um0, um1);
        if constexpr (REAL) {
          ld2<T>(vl + 64 * j, vl0, vl1);
          ld2<T>(vm + 64 * j, vm0, vm1);
        }
        const V x0 = slot_value<REAL>(ul0, um0, vl0, vm0), x1 = slot_value<REAL>(ul1, um1, vl1, vm1);
        sr = pk_fma(mk<T>(w0[j].x, w0[j].x), x0, pk_fma(mk<T>(w1[j].x, w1[j].x), x1, sr));
        si = pk_fma(mk<T>(w0[j].y, w0[j].y), x0, pk_fma(mk<T>(w1[j].y, w1[j].y), x1, si));
      }
    }
    // lanes 0-15 add up the sums for Re V, lanes 16-31 those for Im V, then real and imaginary
    // parts part at bit 3
    const bool up = (lane & 16) != 0, up2 = (lane & 8) != 0;
    T a = (up ? sr.y : sr.x) + __shfl_xor_sync(0xffffffffu, up ? sr.x : sr.y, 16);
    T b = (up ? si.y : si.x) + __shfl_xor_sync(0xffffffffu, up ? si.x : si.y, 16);
    T v = (up2 ? b : a) + __shfl_xor_sync(0xffffffffu, up2 ? a : b, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((lane & 7) == 0) out[q * sq + (lane >> 3)] = v;
  }
}

// one warp per (pair field, solve): tile aggregates -> states entering the tiles
template <typename T>
__global__ void __launch_bounds__(32) k_raman_carry(const SolveDesc* __restrict__ descs, int nt, int TT) {
  using V = c2<T>;
  const SolveDesc& d = descs[blockIdx.y];
  const int q = blockIdx.x;
  const int lane = threadIdx.x;
  const int ntiles = nt / TT;
  const int per = (ntiles + 31) / 32;  // tiles per lane
  const int first = min(lane * per, ntiles), last = min(first + per, ntiles);
  const double2 lamT = lambda_tile(d, TT);
  grid_sync_wait();
  grid_release();
  if (q >= (d.real ? slot_count<true>(d.P) : d.P) || d.M == 0 || __ldcg(d.step) >= d.step_limit) return;
  V* tiles = as_t2<T>(d.raman_tiles) + (size_t)q * ntiles * 2;
  Affine mine = affine_identity();
  for (int i = first; i < last; ++i) {
    mine.a = cmul(mine.a, lamT);
    mine.ba = cadd(cmul(lamT, mine.ba), to_d2(tiles[2 * i]));
    mine.bb = cadd(cmul(lamT, mine.bb), to_d2(tiles[2 * i + 1]));
  }
  const Affine incl = warp_scan_affine(mine, lane);
  Affine pre = shfl_up_affine(incl, 1, 0xffffffffu);
  if (lane == 0) pre = affine_identity();
  const Affine tot = [&] {
    Affine t;
    t.a = make_double2(__shfl_sync(0xffffffffu, incl.a.x, 31), __shfl_sync(0xffffffffu, incl.a.y, 31));
    t.ba = make_double2(__shfl_sync(0xffffffffu, incl.ba.x, 31), __shfl_sync(0xffffffffu, incl.ba.y, 31));
    t.bb = make_double2(__shfl_sync(0xffffffffu, incl.bb.x, 31), __shfl_sync(0xffffffffu, incl.bb.y, 31));
    return t;
  }();
  const double2 inv = d.iir_inv_one_minus;
  double2 ca = cadd(cmul(pre.a, cmul(tot.ba, inv)), pre.ba);
  double2 cb = cadd(cmul(pre.a, cmul(tot.bb, inv)), pre.bb);
  for (int i = first; i < last; ++i) {
    const double2 ga = to_d2(tiles[2 * i]), gb = to_d2(tiles[2 * i + 1]);
    tiles[2 * i] = from_d2<T>(ca);
    tiles[2 * i + 1] = from_d2<T>(cb);
    ca = cadd(cmul(lamT, ca), ga);
    cb = cadd(cmul(lamT, cb), gb);
  }
}

// ---- k_contract: sigma_p(t) = sum_terms Q U_k(t) W(t) over a tile of t, all p ----------
// The U tile [M][TT] and the R tile [P][TT] (Raman on) arrive in shared memory as
// one bulk-async copy per row segment (TT contiguous samples), issued by the
// threads of the CTA and counted on one mbarrier. Then
//   1. every pair field of the tile is formed once, in place:
//        W_lm = (1 - f_R) U_l conj(U_m) + R_lm      (Raman off: U_l conj(U_m)),
//   2. each thread accumulates sigma_p for two adjacent samples over p's terms,
//        sigma_p += q U_k W_pair   (conj(W_pair) for terms whose (l, m) is (m, l) of the
//        stored pair: R_ml = conj(R_lm) as h_R is real, and the Kerr part likewise).
// A warp covers 64 consecutive t of one p (TT >= 64), so term reads are warp-uniform
// and tile reads are conflict-free; terms are staged in shared memory with the
// coefficient already in T.
template <typename T> struct StagedTerm {
  unsigned short k, pc;
  T q;
};

// 16 consecutive values of T from 16-byte aligned shared memory, by 16-byte loads
template <typename T> __device__ __forceinline__ void lds16(const T* a, T* v);
template <> __device__ __forceinline__ void lds16<float>(const float* a, float* v) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float4 x = reinterpret_cast<const float4*>(a)[j];
    v[4 * j] = x.x; v[4 * j + 1] = x.y; v[4 * j + 2] = x.z; v[4 * j + 3] = x.w;
  }
}
template <> __device__ __forceinline__ void lds16<double>(const double* a, double* v) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const double2 x = reinterpret_cast<const double2*>(a)[j];
    v[2 * j] = x.x; v[2 * j + 1] = x.y;
  }
}

// Resident CTAs per SM the FP32 build is held to (registers): 3 for the term loop, 2 for the
// dense form (its accumulators), none for FP64.
template <typename T, int DENSE> constexpr int contract_min_blocks() {
  return sizeof(T) == 4 ? (DENSE == 0 ? 3 : 2) : 1;
}

// raman_mode: 0 Raman off; 1 the convolutions R arrive as rows (k_pair / k_raman_scan);
// 2 the recurrence runs through the tile here from the carries of k_raman_carry; 3 from carries
// the tile sums itself from the aggregates before it (tile_carry; no k_raman_carry).
// DENSE = 0: the term loop (tiles under 64 samples, or too many terms to stage: k_contract_sp
// takes the rest). DENSE = 1: the contraction in its dense form (SolveDesc::dense_q, M <= 16, TT >= 64):
//   T_pk(t) = sum_q A_re[p][q][k] Re W_q(t) + i sum_q A_im[p][q][k] Im W_q(t),
//   sigma_p(t) = sum_k U_k(t) T_pk(t),
// one warp per (p, 64 samples), each lane two samples with all k in registers: a
// register-blocked matrix product instead of one complex triple product per term.
// mixed: the batch holds solves of both forms; each kernel skips the other's.
template <typename T, int DENSE, bool REAL>
__global__ void __launch_bounds__(256, (contract_min_blocks<T, DENSE>())) k_contract(const SolveDesc* __restrict__ descs, int nt, int TT,
                                                  int stage_terms, int raman_mode, int mixed) {
  using V = c2<T>;
  using ST = StagedTerm<T>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long bar;
  V* sU = reinterpret_cast<V*>(smem_raw);
  const SolveDesc& d = descs[blockIdx.y];
  const int t0 = blockIdx.x * TT;
  if (t0 >= nt || d.M == 0 || d.real != REAL || (mixed && (d.dense_q != nullptr) != (DENSE == 1))) {  // empty slot, other form
    grid_sync_wait();
    return;
  }
  const int M = d.M;
  const int raman = raman_mode;
  static_assert(DENSE == 1 || !REAL, "the term loop reads complex pair fields");
  const int P = slot_count<REAL>(d.P);        // slots formed in this tile
  const int Pl = raman == 1 ? P : 0;          // pair rows loaded (Raman convolutions)
  const V* U = as_t2<T>(d.U);
  const V* R = as_t2<T>(d.W);
  const unsigned row_bytes = (unsigned)(TT * sizeof(V));
  const T kerr = (T)d.one_minus_fR;
  V* sW = sU + (size_t)M * TT;
  const int n_terms = d.term_off[M];
  // pair-field rows: swizzled (wsw) when the recurrence runs here, else plain
  const int wmask = raman >= 2 ? max(TT >> 6, 1) - 1 : 0;
  // raman_mode 2, 3: the states entering this tile per pair field (Re V, Im V), staged while
  // the tile lands
  V* sC = sW + (size_t)P * TT;
  const int ntiles = nt / TT, look = tile_look(d, ntiles, TT, raman);
  const double2 lamT = look ? lambda_tile(d, TT) : make_double2(0.0, 0.0);
  // dense form: per warp, two chunks of kDenseChunk coefficient rows (cp.async double buffer)
  T* sA = reinterpret_cast<T*>(sC + (raman >= 2 ? 2 * (size_t)P : 0));
  const size_t dense_elems = DENSE ? (size_t)(blockDim.x >> 5) * 2 * kDenseChunk * 2 * kDenseMaxModes : 0;
  ST* st = reinterpret_cast<ST*>(sA + dense_elems);
  // the terms are staged while the kernel before this one still runs
  if (DENSE == 0 && stage_terms) {
    for (int j = threadIdx.x; j < n_terms; j += blockDim.x) {
      const Term tm = d.terms[j];
      ST s;
      s.k = tm.k;
      s.pc = tm.pc;
      s.q = (T)tm.q;
      st[j] = s;
    }
  }
  if (threadIdx.x == 0) mbar_init(&bar, 1);
  grid_sync_wait();
  if (__ldcg(d.step) >= d.step_limit) return;  // finished solve (nothing is in flight yet)
  if (threadIdx.x == 0) mbar_arrive_expect_tx(&bar, (unsigned)(M + Pl) * row_bytes);
  __syncthreads();
  for (int r = threadIdx.x; r < M + Pl; r += blockDim.x) {
    const V* src = (r < M) ? U + (size_t)r * nt + t0 : R + (size_t)(r - M) * nt + t0;
    bulk_g2s(sU + (size_t)r * TT, src, row_bytes, &bar);
  }
  if (raman >= 2) stage_tile_carries<T>(sC, d, P, ntiles, blockIdx.x, look, lamT);
  // every thread polls with a bound; the barrier makes the outcome CTA-uniform and
  // also publishes the staged terms
  const bool landed = mbar_wait(&bar, 0, d.tile_wait_polls);
  if (!__syncthreads_and(landed ? 1 : 0)) {
    if (threadIdx.x == 0) atomicOr(d.status, kStatusTimeout);
    // give the copies a second bounded chance to land before the CTA leaves
    mbar_wait(&bar, 0, kMaxWaitPolls);
    return;
  }
  const int H = TT >> 1;  // sample pairs per row
  // 1. pair fields
  if (raman < 2) {  // two samples per thread
    for (int idx = threadIdx.x; idx < P * H; idx += blockDim.x) {
      const int q = idx / H, tt = 2 * (idx - q * H);
      const int4 lm = slot_rows<REAL>(d, q);
      V ul0, ul1, um0, um1, vl0 = {}, vl1 = {}, vm0 = {}, vm1 = {};
      ld2<T>(sU + lm.x * TT + tt, ul0, ul1);
      ld2<T>(sU + lm.y * TT + tt, um0, um1);
      if constexpr (REAL) {
        ld2<T>(sU + lm.z * TT + tt, vl0, vl1);
        ld2<T>(sU + lm.w * TT + tt, vm0, vm1);
      }
      V w0 = slot_value<REAL>(ul0, um0, vl0, vm0), w1 = slot_value<REAL>(ul1, um1, vl1, vm1);
      if (raman) {
        V r0, r1;
        ld2<T>(sW + q * TT + tt, r0, r1);
        w0 = mk<T>(fma(kerr, w0.x, r0.x), fma(kerr, w0.y, r0.y));
        w1 = mk<T>(fma(kerr, w1.x, r1.x), fma(kerr, w1.y, r1.y));
      }
      st2<T>(sW + q * TT + tt, w0, w1);
    }
  } else {  // one warp per pair field: the recurrence through the tile, then W in place
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    TileScan<T> ts;
    ts.init(d, TT >> 5, lane);
    for (int q = warp; q < P; q += nwarps)
      tile_pair_recurrence<T, REAL>(ts, sU, TT, slot_rows<REAL>(d, q), sW + (size_t)q * TT, wmask, sC + 2 * q, kerr, lane);
  }
  __syncthreads();
  grid_release();
  // 2. contraction
  V* sigma = as_t2<T>(d.sigma);
  if constexpr (DENSE == 1) {
    constexpr int K = kDenseMaxModes;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    constexpr int ROW = 2 * K;                       // values per coefficient row (p, q)
    constexpr int CH = kDenseChunk;                  // rows per staged chunk
    constexpr int PIECES = CH * ROW * (int)sizeof(T) / 16;  // 16-byte copies per chunk
    const T* A = static_cast<const T*>(d.dense_q);
    T* sAw = sA + (size_t)warp * 2 * CH * ROW;       // this warp's two chunk buffers
    const int chunks = TT >> 6;
    const int nchunk = (P + CH - 1) / CH;
    for (int item = warp; item < M * chunks; item += nwarps) {
      const int p = item / chunks, tt = ((item - p * chunks) << 6) + 2 * lane;
      const int tw = 2 * wsw(tt >> 1, wmask);
      T re0[K], re1[K], im0[K], im1[K];
#pragma unroll
      for (int k = 0; k < K; ++k) re0[k] = re1[k] = im0[k] = im1[k] = 0;
      const T* Ap = A + (size_t)p * P * ROW;
      // rows q0 .. q0 + CH - 1 (clamped to P) into buffer buf, as one cp.async group
      auto stage_rows = [&](int buf, int q0) {
        const int rows = min(CH, P - q0);
        const int pieces = rows * ROW * (int)sizeof(T) / 16;
        const char* src = reinterpret_cast<const char*>(Ap + (size_t)q0 * ROW);
        char* dst = reinterpret_cast<char*>(sAw + (size_t)buf * CH * ROW);
        for (int i = lane; i < pieces && i < PIECES; i += 32) cp_async16(dst + 16 * i, src + 16 * i);
        cp_async_commit();
      };
      __syncwarp();  // the previous item's reads of both buffers are done
      stage_rows(0, 0);
      for (int c = 0; c < nchunk; ++c) {
        if (c + 1 < nchunk) {
          stage_rows((c + 1) & 1, (c + 1) * CH);
          cp_async_wait<1>();
        } else {
          cp_async_wait<0>();
        }
        __syncwarp();  // every lane's copies of chunk c have landed
        const T* rowp = sAw + (size_t)(c & 1) * CH * ROW;
        const int q0 = c * CH, rows = min(CH, P - q0);
#pragma unroll 2
        for (int r = 0; r < rows; ++r) {
          V w0, w1;
          ld2<T>(sW + (q0 + r) * TT + tw, w0, w1);
          T ar[K], ai[K];  // the same addresses on every lane: broadcasts, 16 bytes per load
          lds16<T>(rowp + r * ROW, ar);
          lds16<T>(rowp + r * ROW + K, ai);
#pragma unroll
          for (int k = 0; k < K; ++k) {
            re0[k] = fma(ar[k], w0.x, re0[k]);
            re1[k] = fma(ar[k], w1.x, re1[k]);
            if constexpr (REAL) {  // the slot's second field
              re0[k] = fma(ai[k], w0.y, re0[k]);
              re1[k] = fma(ai[k], w1.y, re1[k]);
            } else {
              im0[k] = fma(ai[k], w0.y, im0[k]);
              im1[k] = fma(ai[k], w1.y, im1[k]);
            }
          }
        }
        __syncwarp();  // reads of buffer c & 1 done before chunk c + 2 is staged into it
      }
      T sx0 = 0, sy0 = 0, sx1 = 0, sy1 = 0;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (k < M) {
          V u0, u1;
          ld2<T>(sU + k * TT + tt, u0, u1);
          if constexpr (REAL) {
            sx0 = fma(u0.x, re0[k], sx0);
            sy0 = fma(u0.y, re0[k], sy0);
            sx1 = fma(u1.x, re1[k], sx1);
            sy1 = fma(u1.y, re1[k], sy1);
          } else {
            sx0 = fma(u0.x, re0[k], fma(-u0.y, im0[k], sx0));
            sy0 = fma(u0.x, im0[k], fma(u0.y, re0[k], sy0));
            sx1 = fma(u1.x, re1[k], fma(-u1.y, im1[k], sx1));
            sy1 = fma(u1.x, im1[k], fma(u1.y, re1[k], sy1));
          }
        }
      }
      st2<T>(sigma + (size_t)p * nt + t0 + tt, mk<T>(sx0, sy0), mk<T>(sx1, sy1));
    }
    return;
  }
  for (int idx = threadIdx.x; idx < M * H; idx += blockDim.x) {
    const int p = idx / H, tt = 2 * (idx - p * H);
    const int tw = 2 * wsw(tt >> 1, wmask);
    T ax0 = 0, ay0 = 0, ax1 = 0, ay1 = 0;
    const int j1 = d.term_off[p + 1];
    for (int j = d.term_off[p]; j < j1; ++j) {
      unsigned short k, pc;
      T qv;
      if (stage_terms) {
        const ST s = st[j];
        k = s.k; pc = s.pc; qv = s.q;
      } else {
        const Term tm = d.terms[j];
        k = tm.k; pc = tm.pc; qv = (T)tm.q;
      }
      V u0, u1, w0, w1;
      ld2<T>(sU + k * TT + tt, u0, u1);
      ld2<T>(sW + (pc & 0x7fff) * TT + tw, w0, w1);
      if (pc & 0x8000) {
        w0.y = -w0.y;
        w1.y = -w1.y;
      }
      const V a0 = cmul(u0, w0), a1 = cmul(u1, w1);
      ax0 = fma(qv, a0.x, ax0);
      ay0 = fma(qv, a0.y, ay0);
      ax1 = fma(qv, a1.x, ax1);
      ay1 = fma(qv, a1.y, ay1);
    }
    st2<T>(sigma + (size_t)p * nt + t0 + tt, mk<T>(ax0, ay0), mk<T>(ax1, ay1));
  }
}

// ---- k_contract_pc: the term loop with the Raman recurrence in the tiles, for tiles with
// too many pair fields to hold at once (tall tiles). Only `pc` pair fields live in shared
// memory at a time: per chunk the warps run the recurrence for the chunk's fields, then
// every thread advances each of its (p, two samples) items through the terms of p whose
// pair field lies in the chunk, accumulating in registers. The terms of each p are sorted
// by pair field, so one cursor per item walks them chunk by chunk. At most kPcItems items
// per thread (M * TT / 2 <= kPcItems * blockDim.x), every term staged in shared memory.
constexpr int kPcItems = 4;
template <typename T>
__global__ void __launch_bounds__(256, (sizeof(T) == 4 ? 3 : 2)) k_contract_pc(const SolveDesc* __restrict__ descs,
                                                                              int nt, int TT, int pc, int raman_mode) {
  using V = c2<T>;
  using ST = StagedTerm<T>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long bar;
  V* sU = reinterpret_cast<V*>(smem_raw);  // [M][TT]
  const SolveDesc& d = descs[blockIdx.y];
  const int t0 = blockIdx.x * TT;
  if (t0 >= nt || d.M == 0) {  // empty slot
    grid_sync_wait();
    return;
  }
  const int M = d.M, P = d.P;
  const unsigned row_bytes = (unsigned)(TT * sizeof(V));
  V* sW = sU + (size_t)M * TT;                             // [pc][TT], pair positions swizzled
  ST* st = reinterpret_cast<ST*>(sW + (size_t)pc * TT);   // every term, sorted by (p, pair field)
  const int n_terms = d.term_off[M];
  V* sC = reinterpret_cast<V*>(st + n_terms);               // states entering the tile, [P][2]
  for (int j = threadIdx.x; j < n_terms; j += blockDim.x) {
    const Term tm = d.terms[j];
    ST x;
    x.k = tm.k;
    x.pc = tm.pc;
    x.q = (T)tm.q;
    st[j] = x;
  }
  if (threadIdx.x == 0) mbar_init(&bar, 1);
  grid_sync_wait();
  if (__ldcg(d.step) >= d.step_limit) return;  // finished solve (nothing is in flight yet)
  if (threadIdx.x == 0) mbar_arrive_expect_tx(&bar, (unsigned)M * row_bytes);
  __syncthreads();
  for (int r = threadIdx.x; r < M; r += blockDim.x)
    bulk_g2s(sU + (size_t)r * TT, as_t2<T>(d.U) + (size_t)r * nt + t0, row_bytes, &bar);
  {
    const int look = tile_look(d, nt / TT, TT, raman_mode);
    stage_tile_carries<T>(sC, d, P, nt / TT, blockIdx.x, look, lambda_tile(d, TT));
  }
  const bool landed = mbar_wait(&bar, 0, d.tile_wait_polls);
  if (!__syncthreads_and(landed ? 1 : 0)) {
    if (threadIdx.x == 0) atomicOr(d.status, kStatusTimeout);
    mbar_wait(&bar, 0, kMaxWaitPolls);
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int H = TT >> 1, nitems = M * H;
  const int wmask = max(TT >> 6, 1) - 1;
  const T kerr = (T)d.one_minus_fR;
  TileScan<T> ts;
  ts.init(d, TT >> 5, lane);
  T acc[kPcItems][4];
  int cur[kPcItems], end[kPcItems];
#pragma unroll
  for (int i = 0; i < kPcItems; ++i) {
    const int idx = threadIdx.x + i * blockDim.x;
    const int p = idx < nitems ? idx / H : 0;
    cur[i] = idx < nitems ? d.term_off[p] : 0;
    end[i] = idx < nitems ? d.term_off[p + 1] : 0;
    acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0;
  }
  for (int c0 = 0; c0 < P; c0 += pc) {
    const int c1 = min(P, c0 + pc);
    for (int q = c0 + warp; q < c1; q += nwarps)
      tile_pair_recurrence<T, false>(ts, sU, TT, slot_rows<false>(d, q), sW + (size_t)(q - c0) * TT, wmask, sC + 2 * q, kerr, lane);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kPcItems; ++i) {
      const int idx = threadIdx.x + i * blockDim.x;
      if (idx >= nitems) continue;
      const int p = idx / H, tt = 2 * (idx - p * H);
      const int tw = 2 * wsw(tt >> 1, wmask);
      int j = cur[i];
      for (; j < end[i]; ++j) {
        const ST x = st[j];
        const int q = x.pc & 0x7fff;
        if (q >= c1) break;
        V u0, u1, w0, w1;
        ld2<T>(sU + x.k * TT + tt, u0, u1);
        ld2<T>(sW + (q - c0) * TT + tw, w0, w1);
        if (x.pc & 0x8000) {
          w0.y = -w0.y;
          w1.y = -w1.y;
        }
        const V a0 = cmul(u0, w0), a1 = cmul(u1, w1);
        acc[i][0] = fma(x.q, a0.x, acc[i][0]);
        acc[i][1] = fma(x.q, a0.y, acc[i][1]);
        acc[i][2] = fma(x.q, a1.x, acc[i][2]);
        acc[i][3] = fma(x.q, a1.y, acc[i][3]);
      }
      cur[i] = j;
    }
    __syncthreads();  // the chunk's fields are read before the next chunk overwrites them
  }
  grid_release();
  V* sigma = as_t2<T>(d.sigma);
#pragma unroll
  for (int i = 0; i < kPcItems; ++i) {
    const int idx = threadIdx.x + i * blockDim.x;
    if (idx >= nitems) continue;
    const int p = idx / H, tt = 2 * (idx - p * H);
    st2<T>(sigma + (size_t)p * nt + t0 + tt, mk<T>(acc[i][0], acc[i][1]), mk<T>(acc[i][2], acc[i][3]));
  }
}

// ---- k_contract_sr: the term loop with the Raman recurrence run serially per pair field --
// For tall tiles (more pair fields than k_contract holds in a tile). A CTA owns TB
// consecutive samples of one solve and walks them in sub-blocks of kSrSub = 16 samples
// (SrLayout: two at a time in the FP32 REAL form):
//   staging  U of the next sub-block is loaded from global memory while this one is
//            worked on; in shared memory each sample pair (t, t + 1) of a
//            row is stored as (Re t, Re t+1, Im t, Im t+1);
//   phase A  each thread owns one or two pair fields q = (l, m) for the whole tile and runs
//            the Raman recurrence S = lambda S + x (x = Re V and Im V, V = U_l conj(U_m))
//            sample after sample from the state entering the tile; the state stays in registers from one sub-block to the next, and
//            W_q = (1 - f_R) V + Im(kappa S) for the sub-block goes to shared memory
//            (Raman off: W_q = V). REAL form: a slot's two fields are the two lanes, and
//            only their Re W is formed;
//   phase B  sigma_p(t) = sum over p's merged terms of U_k (a Re W_q + i b Im W_q)
//            (SolveDesc::sr_coef), eight lanes per group, each with one sample pair (FP32
//            REAL: two); a plan
//            made on the host (SolveDesc::sr_plan) gives each group a mode, or half of a
//            mode with many terms (the two halves sit in one warp and are added by a
//            shuffle), so the longest group's term loop is about half as long as the
//            heaviest mode's; groups of similar length share a warp.
// Shared memory bounds it: per term a lane reads W_q (16 bytes) and the term's record, and U_k
// when k changes; per sub-block a slot reads two rows of U (REAL: four). Measured on a B200 at
// 28 x 65536, 150 slots, 1060 merged terms, 8 solves, a launch: 519 us in the general form; REAL
// form, which halves the phase-A chains and the FMAs of a term, 420 us; with four samples a
// lane (half the W loads and records a sample; one U buffer keeps three CTAs an SM) 378 us, the
// shared-memory pipe busy 75% of the time, issue 49%.
// Compared with the warp-per-field scan, a sample costs one step of each recurrence and no
// scan levels. FP32 solves use the packed two-lane FMA (fma.rn.f32x2): phase A packs the
// two recurrences (Re V and Im V share lambda), phase B the two samples of a pair; each
// lane rounds exactly as the scalar FMA does. No asynchronous copies and no waits besides
// __syncthreads.
constexpr int kSrSub = 16;
constexpr int kSrThreads = 256;
constexpr int kSrPairsPerThread = 2;  // pair fields per thread: P <= 512
constexpr int kSrMaxModes = 64;       // staging: M * kSrSub / 2 <= 2 kSrThreads

// A sample pair (t, t + 1) of one row: re = (Re t, Re t+1), im = (Im t, Im t+1).
template <typename T> struct SrPair {
  c2<T> re, im;
};
template <typename T> __device__ __forceinline__ SrPair<T> ld_pair(const SrPair<T>* p) {
  if constexpr (sizeof(T) == 4) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    SrPair<T> r;
    r.re = make_float2(v.x, v.y);
    r.im = make_float2(v.z, v.w);
    return r;
  } else {
    return *p;
  }
}
template <typename T> __device__ __forceinline__ void st_pair(SrPair<T>* p, c2<T> re, c2<T> im) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(re.x, re.y, im.x, im.y);
  } else {
    p->re = re;
    p->im = im;
  }
}
constexpr int kSrGroups = (kSrThreads / 32) * 4;  // groups of eight lanes in phase B

// One merged term as k_contract_sr keeps it in shared memory: the coefficients (a, b) and
// q | k << 16 in one record of 2 complex values (16 bytes in FP32, 32 in FP64), so that a
// term costs one shared-memory access (two in FP64).
template <typename T> struct SrRec {
  c2<T> ab;
  unsigned kq;
  unsigned pad[sizeof(T) == 4 ? 1 : 3];
};
static_assert(sizeof(SrRec<float>) == 16 && sizeof(SrRec<double>) == 32, "SrRec layout");
template <typename T> __device__ __forceinline__ void ld_rec(const SrRec<T>* r, c2<T>& ab, unsigned& kq) {
  if constexpr (sizeof(T) == 4) {
    const float4 v = *reinterpret_cast<const float4*>(r);
    ab = make_float2(v.x, v.y);
    kq = __float_as_uint(v.z);
  } else {
    ab = r->ab;
    kq = r->kq;
  }
}

template <typename V> __device__ __forceinline__ V shfl_down_c(V v, int d) {
  v.x = __shfl_down_sync(0xffffffffu, v.x, d);
  v.y = __shfl_down_sync(0xffffffffu, v.y, d);
  return v;
}

// Shared-memory layout of k_contract_sr. General form and FP64: sub-blocks of
// kSrSub samples, U double-buffered, a lane of phase B takes one sample pair. FP32 REAL form:
// two sub-blocks at a time; a lane takes four samples, so that a term costs it 16 bytes of W and
// an 8-byte record.
template <typename T, bool REAL> struct SrLayout {
  static constexpr bool WIDE = REAL && sizeof(T) == 4;
  static constexpr int S = WIDE ? 2 * kSrSub : kSrSub;  // samples at a time
  static constexpr int J = S / 2;                       // sample pairs
  static constexpr int NI = (kSrMaxModes * J + kSrThreads - 1) / kSrThreads;  // staged pairs a thread
  static constexpr int BUF = WIDE ? 1 : 2;
  // Row strides: consecutive rows start 16 bytes apart mod 128, so that a quarter warp's rows
  // fall on different banks. U in sample pairs, a field's Re W (REAL) in pairs of reals.
  static constexpr int RS = J + 1;
  static constexpr int WS = WIDE ? J + 2 : J + 1;
  static constexpr int SLOT_BYTES = REAL ? 2 * WS * (int)sizeof(c2<T>) : RS * (int)sizeof(SrPair<T>);
  // where pair j of a U row lies: WIDE has a lane's two pairs 8 positions apart, so that eight
  // lanes read 128 consecutive bytes
  static __host__ __device__ constexpr int pos(int j) { return WIDE ? (j >> 1) + (j & 1) * (J / 2) : j; }
  struct Narrow {
    float ab;
    unsigned kq;
  };
  using Rec = std::conditional_t<WIDE, Narrow, SrRec<T>>;
  static __device__ __forceinline__ auto coef(c2<T> ab) {
    if constexpr (WIDE) return ab.x;
    else return ab;
  }
  static size_t bytes(size_t M, size_t slots, size_t groups, size_t terms) {
    const size_t n = BUF * M * RS * sizeof(SrPair<T>) + slots * SLOT_BYTES + groups * sizeof(int4) + terms * sizeof(Rec);
    return (n + 15) & ~(size_t)15;
  }
};
static_assert(sizeof(SrLayout<float, true>::Rec) == 8, "one term in 8 bytes");

// raman_mode: 0 Raman off, 2 the recurrence from the tile carries of k_raman_carry (tiles of TB), 3 from
// carries summed here (tile_carry)
template <typename T, bool REAL>
__global__ void __launch_bounds__(kSrThreads, (sizeof(T) == 4 ? 3 : 1))
    k_contract_sr(const SolveDesc* __restrict__ descs, int nt, int TB, int raman_mode) {
  using V = c2<T>;
  using SP = SrPair<T>;
  using CF = c2<T>;  // merged coefficient (a, b)
  using L = SrLayout<T, REAL>;
  constexpr bool WIDE = L::WIDE;
  constexpr int J = L::J, RS = L::RS, NI = L::NI;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const SolveDesc& d = descs[blockIdx.y];
  const int t0 = blockIdx.x * TB;
  if (t0 >= nt || d.M == 0 || d.real != REAL) {  // empty slot, other form
    grid_sync_wait();
    return;
  }
  const int M = d.M, P = slot_count<REAL>(d.P), nterm = d.sr_terms, rounds = d.sr_rounds;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // shared memory: U [BUF][M][RS], W [P][RS] (REAL: two planes [P][WS] of sample pairs, the slots'
  // first and second fields, so that a quarter warp's rows stay on different banks), group
  // plan [rounds kSrGroups], merged terms [nterm] (coefficients and row positions)
  SP* sU = reinterpret_cast<SP*>(smem_raw);
  SP* sW = sU + (size_t)L::BUF * M * RS;
  V* sW0 = reinterpret_cast<V*>(sW);
  V* sW1 = sW0 + (size_t)P * L::WS;
  int4* sPlan = reinterpret_cast<int4*>(reinterpret_cast<unsigned char*>(sW) + (size_t)P * L::SLOT_BYTES);
  using Rec = typename L::Rec;
  Rec* sRec = reinterpret_cast<Rec*>(sPlan + rounds * kSrGroups);
  {
    const CF* gCf = static_cast<const CF*>(d.sr_coef);
    for (int i = tid; i < nterm; i += kSrThreads) {
      Rec r = {};
      r.ab = L::coef(gCf[i]);
      r.kq = d.sr_kq[i];
      if constexpr (REAL) {  // the pair field's plane and row as one position
        const unsigned q = r.kq & 0xffffu;
        r.kq = (r.kq >> 16) * (WIDE ? RS << 16 : 1 << 16) | ((q & 1u) * P + (q >> 1)) * L::WS;
      }
      sRec[i] = r;
    }
    for (int i = tid; i < rounds * kSrGroups; i += kSrThreads) sPlan[i] = d.sr_plan[i];
  }
  const double2 lamT = raman_mode == 3 ? lambda_tile(d, TB) : make_double2(0.0, 0.0);
  grid_sync_wait();
  if (__ldcg(d.step) >= d.step_limit) return;  // finished solve (nothing is in flight yet)
  // U staging: sample pair j of row r is item r J + j; a thread carries at most NI
  const V* U = as_t2<T>(d.U);
  const int nu = M * J;
  V pre[NI][2];
  auto fetch = [&](int sub) {
    const int ts = t0 + sub * L::S;
#pragma unroll
    for (int r = 0; r < NI; ++r) {
      const int idx = tid + r * kSrThreads;
      if (idx < nu) {
        const int row = idx / J, j = idx - row * J;
        ld2<T>(U + (size_t)row * nt + ts + 2 * j, pre[r][0], pre[r][1]);
      }
    }
  };
  auto park = [&](int buf) {
#pragma unroll
    for (int r = 0; r < NI; ++r) {
      const int idx = tid + r * kSrThreads;
      if (idx < nu) {
        const int row = idx / J, j = idx - row * J;
        st_pair<T>(sU + ((size_t)buf * M + row) * RS + L::pos(j), mk<T>(pre[r][0].x, pre[r][1].x),
                   mk<T>(pre[r][0].y, pre[r][1].y));
      }
    }
  };
  // phase A: this thread's pair fields and their recurrence states, packed as
  // sr = (Re S_a, Re S_b), si = (Im S_a, Im S_b) (S_a for Re V, S_b for Im V)
  int4 lm[kSrPairsPerThread];
  V sr[kSrPairsPerThread], si[kSrPairsPerThread];
  const int ntiles = nt / TB, look = tile_look(d, ntiles, TB, raman_mode);
#pragma unroll
  for (int i = 0; i < kSrPairsPerThread; ++i) {
    const int q = tid + i * kSrThreads;
    lm[i] = make_int4(0, 0, 0, 0);
    sr[i] = si[i] = mk<T>(0, 0);
    if (q < P) {
      lm[i] = slot_rows<REAL>(d, q);
      if (raman_mode >= 2) {
        const V ca = tile_carry<T>(d, P, ntiles, blockIdx.x, 2 * q, look, lamT);
        const V cb = tile_carry<T>(d, P, ntiles, blockIdx.x, 2 * q + 1, look, lamT);
        sr[i] = mk<T>(ca.x, cb.x);
        si[i] = mk<T>(ca.y, cb.y);
      }
    }
  }
  const T lr = (T)d.iir_lambda.x, li = (T)d.iir_lambda.y;
  const V lr2 = mk<T>(lr, lr), li2 = mk<T>(li, li), nli2 = mk<T>(-li, -li);
  const V kr2 = mk<T>((T)d.iir_kappa.x, (T)d.iir_kappa.x), ki2 = mk<T>((T)d.iir_kappa.y, (T)d.iir_kappa.y);
  const T kerr = (T)d.one_minus_fR;
  const V kerr2 = mk<T>(kerr, kerr);
  V* sigma = as_t2<T>(d.sigma);
  const int nsub = TB / L::S;
  fetch(0);
  park(0);
  __syncthreads();  // U of sub-block 0, the terms
  for (int sub = 0; sub < nsub; ++sub) {
    const int buf = WIDE ? 0 : sub & 1;
    if (sub + 1 == nsub) grid_release();
    else if (!WIDE) fetch(sub + 1);  // lands while this sub-block is worked on
    const SP* uc = sU + (size_t)buf * M * RS;
    // phase A
#pragma unroll
    for (int i = 0; i < kSrPairsPerThread; ++i) {
      const int q = tid + i * kSrThreads;
      if (q < P) {
        const SP* ul = uc + lm[i].x * RS;
        const SP* um = uc + lm[i].y * RS;
        const SP* vl = uc + lm[i].z * RS;
        const SP* vm = uc + lm[i].w * RS;
        SP* wq = sW + (size_t)q * RS;
        V Sr = sr[i], Si = si[i];
        // pair j of the slot: W of its two samples, by fields (REAL) or by parts
        auto pair_w = [&](int j, V (&w)[2]) {
          const SP a = ld_pair<T>(ul + j), b = ld_pair<T>(um + j);
          V v0 = {}, v1 = {};  // REAL: Re V of the two fields, both samples
          if constexpr (REAL) {
            const SP a1 = ld_pair<T>(vl + j), b1 = ld_pair<T>(vm + j);
            v0 = pk_fma(a.re, b.re, pk_mul(a.im, b.im));
            v1 = pk_fma(a1.re, b1.re, pk_mul(a1.im, b1.im));
          }
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            V x;  // V = U_l conj(U_m): (Re V, Im V), or the slot's two Re V
            if constexpr (REAL) {
              x = e ? mk<T>(v0.y, v1.y) : mk<T>(v0.x, v1.x);
            } else {
              const V ue = e ? mk<T>(a.re.y, a.im.y) : mk<T>(a.re.x, a.im.x);
              const V me = e ? mk<T>(b.re.y, b.im.y) : mk<T>(b.re.x, b.im.x);
              x = cmulc(ue, me);
            }
            if (raman_mode >= 2) {
              // S <- lambda S + x for both recurrences, then W = (1 - f_R) V + Im(kappa S)
              const V t = pk_mul(li2, Sr);
              Sr = pk_fma(lr2, Sr, pk_fma(nli2, Si, x));
              Si = pk_fma(lr2, Si, t);
              w[e] = pk_fma(kerr2, x, pk_fma(kr2, Si, pk_mul(ki2, Sr)));
            } else {
              w[e] = x;
            }
          }
        };
        if constexpr (WIDE) {
          float4* w0 = reinterpret_cast<float4*>(sW0 + (size_t)q * L::WS);
          float4* w1 = reinterpret_cast<float4*>(sW1 + (size_t)q * L::WS);
#pragma unroll 4
          for (int h = 0; h < J / 2; ++h) {  // pairs 2h, 2h + 1
            V w[2], y[2];
            pair_w(L::pos(2 * h), w);
            pair_w(L::pos(2 * h + 1), y);
            w0[h] = make_float4(w[0].x, w[1].x, y[0].x, y[1].x);
            w1[h] = make_float4(w[0].y, w[1].y, y[0].y, y[1].y);
          }
        } else {
#pragma unroll
          for (int j = 0; j < J; ++j) {
            V w[2];
            pair_w(j, w);
            if constexpr (REAL) {
              sW0[(size_t)q * L::WS + j] = mk<T>(w[0].x, w[1].x);
              sW1[(size_t)q * L::WS + j] = mk<T>(w[0].y, w[1].y);
            } else {
              st_pair<T>(wq + j, mk<T>(w[0].x, w[1].x), mk<T>(w[0].y, w[1].y));
            }
          }
        }
        sr[i] = Sr;
        si[i] = Si;
      }
    }
    __syncthreads();  // W of this sub-block is complete
    if (WIDE && sub + 1 < nsub) fetch(sub + 1);  // lands during phase B
    // phase B
    {
      const int j = lane & 7;
      const int ts = t0 + sub * L::S;
      for (int r = 0; r < rounds; ++r) {
        const int4 pl = sPlan[r * kSrGroups + warp * 4 + (lane >> 3)];  // p, first term, end, role
        if constexpr (WIDE) {
          // sigma = U X summed over the terms, X = a Re W: Re and Im of the lane's pairs 2j, 2j + 1
          V ra = mk<T>(0, 0), rb = ra, ia = ra, ib = ra;
          SP u = {}, v = {};
          int kprev = -1;
#pragma unroll 2
          for (int n = pl.y; n < pl.z; ++n) {
            const Rec c = sRec[n];
            const int k = (int)(c.kq >> 16);
            if (k != kprev) {  // a mode's terms are sorted by k
              u = ld_pair<T>(uc + k + j);
              v = ld_pair<T>(uc + k + j + 8);
              kprev = k;
            }
            const float4 w = *reinterpret_cast<const float4*>(sW0 + (c.kq & 0xffffu) + 2 * j);
            const V c2 = mk<T>(c.ab, c.ab);
            const V xa = pk_mul(c2, mk<T>(w.x, w.y)), xb = pk_mul(c2, mk<T>(w.z, w.w));
            ra = pk_fma(u.re, xa, ra);
            ia = pk_fma(u.im, xa, ia);
            rb = pk_fma(v.re, xb, rb);
            ib = pk_fma(v.im, xb, ib);
          }
          // the upper half of a split mode (the next group, 8 lanes up) adds into the lower half
          const V ra2 = shfl_down_c(ra, 8), ia2 = shfl_down_c(ia, 8);
          const V rb2 = shfl_down_c(rb, 8), ib2 = shfl_down_c(ib, 8);
          if (pl.w == 1) {
            ra = cadd(ra, ra2);
            ia = cadd(ia, ia2);
            rb = cadd(rb, rb2);
            ib = cadd(ib, ib2);
          }
          if (pl.w <= 1) {
            V* out = sigma + (size_t)pl.x * nt + ts + 4 * j;
            st2<T>(out, mk<T>(ra.x, ia.x), mk<T>(ra.y, ia.y));
            st2<T>(out + 2, mk<T>(rb.x, ib.x), mk<T>(rb.y, ib.y));
          }
        } else {
          // sigma = U X summed over the terms: Re = a1 - a2, Im = a3 + a4 with a1 = sum Re U Re X,
          // a2 = sum Im U Im X, a3 = sum Re U Im X, a4 = sum Im U Re X (packed over the pair)
          V a1 = mk<T>(0, 0), a2 = a1, a3 = a1, a4 = a1;
          // a mode's terms are sorted by k: U_k is read again only when k changes
          SP u = {};
          int kprev = -1;
#pragma unroll 2
          for (int n = pl.y; n < pl.z; ++n) {
            CF c;
            unsigned kq;
            ld_rec<T>(sRec + n, c, kq);
            const int k = (int)(kq >> 16);
            if (k != kprev) {
              u = ld_pair<T>(uc + k * RS + j);
              kprev = k;
            }
            if constexpr (REAL) {
              const V xr = pk_mul(mk<T>(c.x, c.x), sW0[(kq & 0xffffu) + j]);  // X = a Re W
              a1 = pk_fma(u.re, xr, a1);
              a4 = pk_fma(u.im, xr, a4);
            } else {
              const SP w = ld_pair<T>(sW + (kq & 0xffffu) * RS + j);
              const V xr = pk_mul(mk<T>(c.x, c.x), w.re), xi = pk_mul(mk<T>(c.y, c.y), w.im);  // X
              a1 = pk_fma(u.re, xr, a1);
              a2 = pk_fma(u.im, xi, a2);
              a3 = pk_fma(u.re, xi, a3);
              a4 = pk_fma(u.im, xr, a4);
            }
          }
          // the upper half of a split mode (the next group, 8 lanes up) adds into the lower half
          const V b1 = shfl_down_c(a1, 8), b4 = shfl_down_c(a4, 8);
          V b2 = {}, b3 = {};
          if constexpr (!REAL) {
            b2 = shfl_down_c(a2, 8);
            b3 = shfl_down_c(a3, 8);
          }
          if (pl.w == 1) {
            a1 = cadd(a1, b1);
            a2 = cadd(a2, b2);
            a3 = cadd(a3, b3);
            a4 = cadd(a4, b4);
          }
          if (pl.w <= 1)
            st2<T>(sigma + (size_t)pl.x * nt + ts + 2 * j, mk<T>(a1.x - a2.x, a3.x + a4.x), mk<T>(a1.y - a2.y, a3.y + a4.y));
        }
      }
    }
    if constexpr (WIDE) __syncthreads();  // the one U buffer is free
    // else buffer buf ^ 1 was last read in the previous sub-block, which ended at a barrier
    if (sub + 1 < nsub) park(WIDE ? 0 : buf ^ 1);
    __syncthreads();  // W is free again; the next U is in place
  }
}

// ---- k_raman_agg_sr: the tile aggregates for k_contract_sr's tiles ------------------------
// One thread per pair field: the aggregate of the recurrence over the tile from a zero
// start, S_end = sum_t lambda^(TB-1-t) x_t (x = Re V, Im V, V = U_l conj(U_m)), run as
// S <- lambda S + x sample after sample (the arithmetic of k_contract_sr's phase A without
// the output), U arriving in sub-blocks of kSrSub samples through the same double buffer.
// The contraction's tiles (tile_carry), or k_raman_carry, make the states entering the tiles of them.
// Shared-memory reads of U bound it (l1tex 88% busy): 8 solves of 28 x 65536 with 150 slots, 105 us a
// launch; skipping the second row where a slot's two fields share a mode made it 134.
template <typename T, bool REAL>
__global__ void __launch_bounds__(kSrThreads, (sizeof(T) == 4 ? 4 : 2))
    k_raman_agg_sr(const SolveDesc* __restrict__ descs, int nt, int TB, int by_tile) {
  using V = c2<T>;
  using SP = SrPair<T>;
  constexpr int J = kSrSub / 2;
  constexpr int RS = J + 1;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const SolveDesc& d = descs[blockIdx.y];
  const int t0 = blockIdx.x * TB;
  grid_sync_wait();
  if (t0 >= nt || d.M == 0 || d.real != REAL) return;  // empty slot, other form
  if (__ldcg(d.step) >= d.step_limit) return;  // finished solve
  const int M = d.M, P = slot_count<REAL>(d.P), tid = threadIdx.x;
  SP* sU = reinterpret_cast<SP*>(smem_raw);  // [2][M][RS]
  const V* U = as_t2<T>(d.U);
  const int nu = M * J;
  V pre[2][2];
  auto fetch = [&](int sub) {
    const int ts = t0 + sub * kSrSub;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int idx = tid + r * kSrThreads;
      if (idx < nu) {
        const int row = idx / J, j = idx - row * J;
        ld2<T>(U + (size_t)row * nt + ts + 2 * j, pre[r][0], pre[r][1]);
      }
    }
  };
  auto park = [&](int buf) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int idx = tid + r * kSrThreads;
      if (idx < nu) {
        const int row = idx / J, j = idx - row * J;
        st_pair<T>(sU + ((size_t)buf * M + row) * RS + j, mk<T>(pre[r][0].x, pre[r][1].x),
                   mk<T>(pre[r][0].y, pre[r][1].y));
      }
    }
  };
  int4 lm[kSrPairsPerThread];
  V sr[kSrPairsPerThread], si[kSrPairsPerThread];
#pragma unroll
  for (int i = 0; i < kSrPairsPerThread; ++i) {
    const int q = tid + i * kSrThreads;
    lm[i] = make_int4(0, 0, 0, 0);
    sr[i] = si[i] = mk<T>(0, 0);
    if (q < P) lm[i] = slot_rows<REAL>(d, q);
  }
  const T lr = (T)d.iir_lambda.x, li = (T)d.iir_lambda.y;
  const V lr2 = mk<T>(lr, lr), li2 = mk<T>(li, li), nli2 = mk<T>(-li, -li);
  const int nsub = TB / kSrSub;
  fetch(0);
  park(0);
  __syncthreads();
  for (int sub = 0; sub < nsub; ++sub) {
    const int buf = sub & 1;
    if (sub + 1 < nsub) fetch(sub + 1);
    else grid_release();
    const SP* uc = sU + (size_t)buf * M * RS;
#pragma unroll
    for (int i = 0; i < kSrPairsPerThread; ++i) {
      if (tid + i * kSrThreads < P) {
        const SP* ul = uc + lm[i].x * RS;
        const SP* um = uc + lm[i].y * RS;
        const SP* vl = uc + lm[i].z * RS;
        const SP* vm = uc + lm[i].w * RS;
        V Sr = sr[i], Si = si[i];
#pragma unroll
        for (int j = 0; j < J; ++j) {
          const SP a = ld_pair<T>(ul + j), b = ld_pair<T>(um + j);
          V v0 = {}, v1 = {};
          if constexpr (REAL) {
            const SP a1 = ld_pair<T>(vl + j), b1 = ld_pair<T>(vm + j);
            v0 = pk_fma(a.re, b.re, pk_mul(a.im, b.im));
            v1 = pk_fma(a1.re, b1.re, pk_mul(a1.im, b1.im));
          }
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            V x;
            if constexpr (REAL) x = e ? mk<T>(v0.y, v1.y) : mk<T>(v0.x, v1.x);
            else
              x = cmulc(e ? mk<T>(a.re.y, a.im.y) : mk<T>(a.re.x, a.im.x),
                        e ? mk<T>(b.re.y, b.im.y) : mk<T>(b.re.x, b.im.x));
            const V t = pk_mul(li2, Sr);
            Sr = pk_fma(lr2, Sr, pk_fma(nli2, Si, x));
            Si = pk_fma(lr2, Si, t);
          }
        }
        sr[i] = Sr;
        si[i] = Si;
      }
    }
    // buffer buf ^ 1 was last read in the previous sub-block, which ended at this barrier
    if (sub + 1 < nsub) park(buf ^ 1);
    __syncthreads();
  }
  V* out = as_t2<T>(d.raman_tiles) + (size_t)blockIdx.x * (by_tile ? 2 * P : 2);
  const size_t sq = by_tile ? 2 : 2 * (size_t)(nt / TB);
#pragma unroll
  for (int i = 0; i < kSrPairsPerThread; ++i) {
    const int q = tid + i * kSrThreads;
    if (q < P) {
      st2<T>(out + q * sq, mk<T>(sr[i].x, si[i].x), mk<T>(sr[i].y, si[i].y));  // Re V, Im V recurrences
    }
  }
}

// ---- k_contract_sp: the sparse contraction of tiles of 64 to 256 samples -------------------
// All pair fields of the tile at once in shared memory, as k_contract, with the arithmetic of
// k_contract_sr: packed two-lane FMAs (FP32) and merged terms. Samples lie in pairs
// (Re t, Re t+1, Im t, Im t+1), pair h of a row at wsw(h), so that a warp's 32 consecutive
// pairs and lane L's own g = TT/64 pairs g L .. g L + g - 1 are both conflict-free.
//   1. the U tile lands (bulk copies, bounded wait) and is put in that form, each warp its own
//      32 pairs in place;
//   2. one warp per pair field: each lane forms V of its c = TT/32 samples, runs the recurrence
//      through them from zero, the lanes' ends are scanned, and the lane runs it again from the
//      state entering it, now with W = (1 - f_R) V + Im(kappa S) as output. The recurrences of
//      Re V and Im V are the two lanes of one packed chain. (Raman off, or R from rows: W
//      pointwise.)
//   3. one warp per (p, 32 pairs): sigma = sum over p's merged terms of U_k (a Re W + i b Im W),
//      terms as one record (a, b, positions of row k and row q), U_k read when k changes.
// What bounds it: the latency of the tile and of the states entering it (long_scoreboard stalls
// first, 3.7 of 7 cycles an issued instruction, 28 warps an SM), then issue (53% of cycles). Measured on a
// B200 against the scalar term loop over unmerged terms (k_contract<T, 0>), a launch: 32 solves
// of 6 x 16384 (16 pair fields) 56 -> 44 us, 38.2 -> 27.8 million warp instructions; 128 of
// 2 x 4096 29 -> 24 us; a step of one 6 x 8192 FP64 solve 112 -> 96 us. REAL form (8 slots for
// the 16 pair fields): 45 -> 41 us.
template <typename T> struct LaneScan {
  using V = c2<T>;
  V lr2, li2, nli2, kr2, ki2;  // lambda and kappa, each component in both lanes
  V lvl[5];                    // lambda^(c 2^j), zero for the lanes a level does not reach
  V lane_pow;                  // lambda^(c lane)
  int c;
  __device__ __forceinline__ void init(const SolveDesc& d, int c_, int lane) {
    c = c_;
    const T lr = (T)d.iir_lambda.x, li = (T)d.iir_lambda.y;
    lr2 = mk<T>(lr, lr);
    li2 = mk<T>(li, li);
    nli2 = mk<T>(-li, -li);
    kr2 = mk<T>((T)d.iir_kappa.x, (T)d.iir_kappa.x);
    ki2 = mk<T>((T)d.iir_kappa.y, (T)d.iir_kappa.y);
    const V* pw = static_cast<const V*>(d.raman_pow);  // lambda^j, j < 256, from FP64
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      const V l = __ldg(pw + (c << j));
      lvl[j] = lane >= (1 << j) ? l : mk<T>(0, 0);
    }
    lane_pow = __ldg(pw + c * lane);
  }
  // S <- lambda S + x, S = (re, im), lanes Re V and Im V
  __device__ __forceinline__ void step(V& re, V& im, V x) const {
    const V t = pk_mul(li2, re);
    re = pk_fma(lr2, re, pk_fma(nli2, im, x));
    im = pk_fma(lr2, im, t);
  }
  // (re, im): the lane's end from a zero start -> the state entering the lane, from the ends
  // of the lanes before it (inclusive scan S_L = lambda^c S_{L-1} + end_L, handed up by one) and
  // the state entering the tile, carry = (Re V's, Im V's)
  __device__ __forceinline__ void enter(V& re, V& im, int lane, const V* carry) const {
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      const int o = 1 << j;
      V pr, pi;
      pr.x = __shfl_up_sync(0xffffffffu, re.x, o);
      pr.y = __shfl_up_sync(0xffffffffu, re.y, o);
      pi.x = __shfl_up_sync(0xffffffffu, im.x, o);
      pi.y = __shfl_up_sync(0xffffffffu, im.y, o);
      const V l = lvl[j];
      re = mk<T>(fma(l.x, pr.x, fma(-l.y, pi.x, re.x)), fma(l.x, pr.y, fma(-l.y, pi.y, re.y)));
      im = mk<T>(fma(l.x, pi.x, fma(l.y, pr.x, im.x)), fma(l.x, pi.y, fma(l.y, pr.y, im.y)));
    }
    V er, ei;
    er.x = __shfl_up_sync(0xffffffffu, re.x, 1);
    er.y = __shfl_up_sync(0xffffffffu, re.y, 1);
    ei.x = __shfl_up_sync(0xffffffffu, im.x, 1);
    ei.y = __shfl_up_sync(0xffffffffu, im.y, 1);
    if (lane == 0) er = ei = mk<T>(0, 0);
    V ca, cb;
    ld2<T>(carry, ca, cb);
    const V l = lane_pow;
    re = mk<T>(fma(l.x, ca.x, fma(-l.y, ca.y, er.x)), fma(l.x, cb.x, fma(-l.y, cb.y, er.y)));
    im = mk<T>(fma(l.x, ca.y, fma(l.y, ca.x, ei.x)), fma(l.x, cb.y, fma(l.y, cb.x, ei.y)));
  }
};

// REAL form: rows of W are real, one per pair field (TT values of T): pair h at rs(h), which spreads
// a lane's own 16-byte chunks (four samples in FP32, two in FP64) over the banks.
template <typename T> __device__ __forceinline__ int rs(int h, int wmask) {
  return sizeof(T) == 8 ? wsw(h, wmask) : h ^ (wmask == 3 ? ((h >> 4) & 1) << 1 : 0);
}

template <typename T, bool REAL>
__global__ void __launch_bounds__(256, (sizeof(T) == 4 ? 4 : 2))
    k_contract_sp(const SolveDesc* __restrict__ descs, int nt, int TT, int raman_mode, int mixed) {
  using V = c2<T>;
  using SP = SrPair<T>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long bar;
  const SolveDesc& d = descs[blockIdx.y];
  const int t0 = blockIdx.x * TT;
  if (t0 >= nt || d.M == 0 || d.real != REAL || (mixed && d.dense_q != nullptr)) {  // empty slot, other form
    grid_sync_wait();
    return;
  }
  const int M = d.M, P = slot_count<REAL>(d.P), nterm = d.sr_terms;
  const int H = TT >> 1, wmask = (TT >> 6) - 1;  // pairs per row
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  SP* sU = reinterpret_cast<SP*>(smem_raw);      // [M][H]
  SP* sW = sU + (size_t)M * H;                   // [P][H] (REAL: [2 P][H] real pairs)
  V* sR = reinterpret_cast<V*>(sW);
  SrRec<T>* sRec = reinterpret_cast<SrRec<T>*>(sW + (size_t)P * H);
  V* sC = reinterpret_cast<V*>(sRec + nterm);    // states entering the tile, [P][2]
  // staged while the kernel before this one still runs: the terms, with k and q as row positions
  {
    const V* cf = static_cast<const V*>(d.sr_coef);
    for (int i = tid; i < nterm; i += blockDim.x) {
      const unsigned kq = d.sr_kq[i];
      SrRec<T> r = {};
      r.ab = cf[i];
      r.kq = (kq & 0xffffu) * H | ((kq >> 16) * H) << 16;  // a row of W is H pairs in both forms
      sRec[i] = r;
    }
  }
  const int ntiles = nt / TT, look = tile_look(d, ntiles, TT, raman_mode);
  const double2 lamT = look ? lambda_tile(d, TT) : make_double2(0.0, 0.0);
  const T kerr = (T)d.one_minus_fR;
  LaneScan<T> ts;
  if (raman_mode >= 2) ts.init(d, TT >> 5, lane);
  if (tid == 0) mbar_init(&bar, 1);
  const int Pl = !REAL && raman_mode == 1 ? P : 0;  // rows of R loaded (never in the REAL form)
  const unsigned row_bytes = (unsigned)(TT * sizeof(V));
  if (tid == 0) mbar_arrive_expect_tx(&bar, (unsigned)(M + Pl) * row_bytes);
  __syncthreads();
  grid_sync_wait();
  for (int r = tid; r < M; r += blockDim.x)
    bulk_g2s(sU + (size_t)r * H, as_t2<T>(d.U) + (size_t)r * nt + t0, row_bytes, &bar);
  for (int r = tid; r < Pl; r += blockDim.x)
    bulk_g2s(sW + (size_t)r * H, as_t2<T>(d.W) + (size_t)r * nt + t0, row_bytes, &bar);
  if (__ldcg(d.step) >= d.step_limit) {  // finished solve: the copies land before the CTA leaves
    mbar_wait(&bar, 0, kMaxWaitPolls);
    return;
  }
  if (raman_mode >= 2) stage_tile_carries<T>(sC, d, P, ntiles, blockIdx.x, look, lamT);
  const bool landed = mbar_wait(&bar, 0, d.tile_wait_polls);
  if (!__syncthreads_and(landed ? 1 : 0)) {
    if (tid == 0) atomicOr(d.status, kStatusTimeout);
    // give the copies a second bounded chance to land before the CTA leaves
    mbar_wait(&bar, 0, kMaxWaitPolls);
    return;
  }
  // 1. U in pairs of real and imaginary parts (rows of H = 32, 64 or 128 pairs: a warp stays in one)
  for (int i = tid; i < M * H; i += blockDim.x) {
    const int h = i & (H - 1);
    SP* row = sU + (i - h);
    V u0, u1;
    ld2<T>(reinterpret_cast<const V*>(row + h), u0, u1);
    __syncwarp();
    st_pair<T>(row + wsw(h, wmask), mk<T>(u0.x, u1.x), mk<T>(u0.y, u1.y));
  }
  __syncthreads();
  // V of one pair of samples
  auto pair_product = [](const SP& a, const SP& b, V& vre, V& vim) {
    vre = pk_fma(a.re, b.re, pk_mul(a.im, b.im));
    vim = pk_fma(a.im, b.re, pk_mul(mk<T>(-a.re.x, -a.re.y), b.im));
  };
  auto real_product = [](const SP& a, const SP& b) { return pk_fma(a.re, b.re, pk_mul(a.im, b.im)); };
  // 2. pair fields
  if (raman_mode >= 2) {
    const int g = ts.c >> 1;
    for (int q = warp; q < P; q += nwarps) {
      const int4 lm = slot_rows<REAL>(d, q);
      const SP* ul = sU + lm.x * H;
      const SP* um = sU + lm.y * H;
      SP* wq = sW + (size_t)q * H;
      V x[8];  // (Re V, Im V) of the lane's samples, or the slot's two Re V
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j < g) {
          const int at = wsw(g * lane + j, wmask);
          V vre, vim;
          if constexpr (REAL) {
            vre = real_product(ld_pair<T>(ul + at), ld_pair<T>(um + at));
            vim = real_product(ld_pair<T>(sU + lm.z * H + at), ld_pair<T>(sU + lm.w * H + at));
          } else {
            pair_product(ld_pair<T>(ul + at), ld_pair<T>(um + at), vre, vim);
          }
          x[2 * j] = mk<T>(vre.x, vim.x);
          x[2 * j + 1] = mk<T>(vre.y, vim.y);
        }
      }
      V sr = x[0], si = mk<T>(0, 0);  // the lane's end from a zero start
#pragma unroll
      for (int k = 1; k < 8; ++k)
        if (k < ts.c) ts.step(sr, si, x[k]);
      ts.enter(sr, si, lane, sC + 2 * q);  // the state entering the lane
      const V kerr2 = mk<T>(kerr, kerr);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (k < ts.c) {
          ts.step(sr, si, x[k]);
          x[k] = pk_fma(kerr2, x[k], pk_fma(ts.kr2, si, pk_mul(ts.ki2, sr)));
        }
      }
      if constexpr (REAL) {
        V* w0 = sR + (size_t)(2 * q) * H;
        V* w1 = w0 + H;
        if (sizeof(T) == 4 && g > 1) {  // four samples of a field per 16 bytes
#pragma unroll
          for (int j = 0; j < 4; j += 2) {
            if (j < g) {
              const int at = rs<T>(g * lane + j, wmask);
              st2<T>(w0 + at, mk<T>(x[2 * j].x, x[2 * j + 1].x), mk<T>(x[2 * j + 2].x, x[2 * j + 3].x));
              st2<T>(w1 + at, mk<T>(x[2 * j].y, x[2 * j + 1].y), mk<T>(x[2 * j + 2].y, x[2 * j + 3].y));
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (j < g) {
              const int at = rs<T>(g * lane + j, wmask);
              w0[at] = mk<T>(x[2 * j].x, x[2 * j + 1].x);
              w1[at] = mk<T>(x[2 * j].y, x[2 * j + 1].y);
            }
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j < g)
            st_pair<T>(wq + wsw(g * lane + j, wmask), mk<T>(x[2 * j].x, x[2 * j + 1].x),
                       mk<T>(x[2 * j].y, x[2 * j + 1].y));
      }
    }
  } else {
    for (int i = tid; i < P * H; i += blockDim.x) {
      const int h = i & (H - 1), at = wsw(h, wmask);
      const int4 lm = slot_rows<REAL>(d, i / H);
      V vre, vim;
      if constexpr (REAL) {
        vre = real_product(ld_pair<T>(sU + lm.x * H + at), ld_pair<T>(sU + lm.y * H + at));
        vim = real_product(ld_pair<T>(sU + lm.z * H + at), ld_pair<T>(sU + lm.w * H + at));
        V* w0 = sR + 2 * (size_t)(i - h);
        w0[rs<T>(h, wmask)] = vre;
        w0[H + rs<T>(h, wmask)] = vim;
        continue;
      }
      SP* row = sW + (i - h);
      pair_product(ld_pair<T>(sU + lm.x * H + at), ld_pair<T>(sU + lm.y * H + at), vre, vim);
      if (raman_mode == 1) {  // W = (1 - f_R) V + R, R in place as it landed
        V r0, r1;
        ld2<T>(reinterpret_cast<const V*>(row + h), r0, r1);
        vre = pk_fma(mk<T>(kerr, kerr), vre, mk<T>(r0.x, r1.x));
        vim = pk_fma(mk<T>(kerr, kerr), vim, mk<T>(r0.y, r1.y));
        __syncwarp();
      }
      st_pair<T>(row + at, vre, vim);
    }
  }
  __syncthreads();
  grid_release();
  // 3. contraction
  V* sigma = as_t2<T>(d.sigma);
  for (int item = warp; item < M * (H >> 5); item += nwarps) {
    const int p = item / (H >> 5), h = (item - p * (H >> 5)) * 32 + lane, at = wsw(h, wmask);
    const SP* uc = sU + at;
    const SP* wc = sW + at;
    const V* rc = sR + rs<T>(h, wmask);
    const int n1 = __ldg(d.sr_off + p + 1);
    V a1 = mk<T>(0, 0), a2 = a1, a3 = a1, a4 = a1;
    SP u = {};
    unsigned kprev = ~0u;
#pragma unroll 2
    for (int n = __ldg(d.sr_off + p); n < n1; ++n) {
      V c;
      unsigned kq;
      ld_rec<T>(sRec + n, c, kq);
      if ((kq >> 16) != kprev) {
        kprev = kq >> 16;
        u = ld_pair<T>(uc + kprev);
      }
      if constexpr (REAL) {
        const V xr = pk_mul(mk<T>(c.x, c.x), rc[kq & 0xffffu]);  // a Re W
        a1 = pk_fma(u.re, xr, a1);
        a4 = pk_fma(u.im, xr, a4);
      } else {
        const SP w = ld_pair<T>(wc + (kq & 0xffffu));
        const V xr = pk_mul(mk<T>(c.x, c.x), w.re), xi = pk_mul(mk<T>(c.y, c.y), w.im);  // a Re W, b Im W
        a1 = pk_fma(u.re, xr, a1);
        a2 = pk_fma(u.im, xi, a2);
        a3 = pk_fma(u.re, xi, a3);
        a4 = pk_fma(u.im, xr, a4);
      }
    }
    st2<T>(sigma + (size_t)p * nt + t0 + 2 * h, mk<T>(a1.x - a2.x, a3.x + a4.x), mk<T>(a1.y - a2.y, a3.y + a4.y));
  }
}

// ---- k_contract_tc: the dense contraction on the tensor cores (FP32 solves, M <= 16) -----
// Per tile of kTcTile = 128 samples the dense form is two real matrix products over the
// pair fields q,
//   T_re[t][(p, k)] = sum_q Re W_q(t) A_re[p][q][k],   T_im[t][(p, k)] = sum_q Im W_q(t) A_im[p][q][k],
// followed by sigma_p(t) = sum_k U_k(t) (T_re + i T_im) (the k_contract<T, 1> arithmetic).
// The products are tcgen05 TF32 MMAs: M = 128 samples (TMEM lane = sample), N = 16 M
// columns (p, k) per product (Re in TMEM columns [0, N), Im in [256, 256 + N)), K = the pair
// fields in chunks of kTcChunk = 8. Both operands are split x = hi + lo into TF32 parts
// and every product is formed as hi hi + hi lo + lo hi with FP32 accumulation: relative
// error about 2^-21 (plain TF32 would leave 2^-11).
// Warps 0-15 build the pair fields, one field of every other chunk each: V of the lane's 4 consecutive
// samples, the Raman recurrence through them (raman_mode 2 or 3; the packed chain and lane scan of
// k_contract_sp), and W split into TF32 hi and lo straight into the A operands (stage c % 4) in the
// MN-major TF32 layout (samples contiguous: 4 samples of a field are one 16-byte chunk per
// matrix). Warp 16 drives: it copies the chunk's split coefficients (SolveDesc::dense_tc,
// K-major) up to four ahead, and when the fields and the coefficients are in, issues the chunk's
// 6 MMAs and commits them to the mbarrier that frees the stage. No barrier of the whole CTA stands
// between the chunks: builders run up to four chunks ahead of the tensor core. Every wait is
// bounded; when one gives up, a flag ends the others' waits, the CTA reports kStatusTimeout, waits
// once more for what is in flight and frees its TMEM.
// What bounds it: shared-memory bandwidth (a chunk's MMAs read 70 KB, its operands are written
// with 46 KB: 15.6 thousand of a CTA's 31 thousand cycles), then the CTA's start and end (7
// thousand). Measured on a B200, 16 solves of 15 x 8192, a launch, against two 16-field buffers
// between barriers of the whole CTA and scalar recurrences: 183 -> 141 us, 64 -> 44 million warp
// instructions (24 builder warps instead of 16: 143). REAL form (one product over all fields, half the
// recurrences, operands and MMAs; two CTAs an SM): 76 us.
constexpr int kTcBuilders = 2;  // chunks built at a time, a warp per slot
template <bool REAL> constexpr int tc_threads() { return 32 * (slot_count<REAL>(kTcChunk) * kTcBuilders + 1); }

// mbar_wait that also gives up once *stop is set (by another warp whose wait ran out). The answer is
// a thread's own: two lanes may see the barrier complete and *stop set in either order.
__device__ __forceinline__ bool mbar_wait_or(unsigned long long* bar, unsigned parity, volatile int* stop, unsigned polls) {
  for (unsigned it = 0; it < polls; it += 64) {
    if (mbar_wait(bar, parity, 64)) return true;
    if (*stop) return false;
  }
  *stop = 1;
  return false;
}
// ... for a whole warp: one answer for its lanes, which meet again at full-mask shuffles
__device__ __forceinline__ bool mbar_wait_or_warp(unsigned long long* bar, unsigned parity, volatile int* stop, unsigned polls) {
  return __all_sync(0xffffffffu, mbar_wait_or(bar, parity, stop, polls));
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

template <typename T, bool REAL>
__global__ void __launch_bounds__(tc_threads<REAL>(), REAL ? 2 : 1) k_contract_tc(const SolveDesc* __restrict__ descs, int nt, int raman_mode) {
  static_assert(sizeof(T) == 4, "TF32 operands come from FP32 solves");
  using V = float2;
  constexpr int TT = kTcTile, KC = kTcChunk, NS = kTcStages;
  constexpr int SC = slot_count<REAL>(KC);      // slots per chunk
  constexpr int BW = kTcBuilders * SC;          // builder warps
  constexpr int PARTS = REAL ? 1 : 2;           // products: Re, Im
  constexpr int MATS = 2 * PARTS;               // operand matrices: hi and lo of each
  constexpr uint32_t COLS = 256 * PARTS;        // TMEM columns
  // A operand (MN-major TF32 layout): 32-sample atoms 512 bytes apart, 4-field groups 2048
  static_assert(TT == 128 && KC == 8, "one MMA covers the tile's 128 samples and a chunk");
  constexpr uint32_t A_LBO = 512, A_SBO = 2048;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long bar_u, bar_a[NS], bar_b[NS], bar_m[NS];
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_stop;
  const SolveDesc& d = descs[blockIdx.y];
  const int t0 = blockIdx.x * TT;
  if (t0 >= nt || d.M == 0 || d.real != REAL) {  // empty slot, other form
    grid_sync_wait();
    return;
  }
  const int M = d.M, P = d.P, PS = slot_count<REAL>(P), N = 16 * M;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  V* sU = reinterpret_cast<V*>(smem_raw);                        // [M][TT]
  // [NS][MATS][KC * TT] MN-major operands, on the next 1024-byte boundary (the swizzle pattern's
  // alignment; the launch reserves the slack)
  unsigned char* after_u = reinterpret_cast<unsigned char*>(sU + (size_t)M * TT);
  float* sA = reinterpret_cast<float*>(after_u + ((1024u - (tc::smem_u32(after_u) & 1023u)) & 1023u));
  float* sB = sA + NS * MATS * KC * TT;                          // [NS][MATS][KC/4][N][4]
  V* sC = reinterpret_cast<V*>(sB + NS * MATS * KC * N);          // states entering the tile, [PS][2]
  const int nch = (P + KC - 1) / KC;
  const unsigned bbytes = (unsigned)(MATS * KC * N * sizeof(float));
  const unsigned polls = d.stage_wait_polls;
  LaneScan<float> ts;
  if (raman_mode >= 2) ts.init(d, TT >> 5, lane);
  if (tid == 0) {
    s_stop = 0;
    mbar_init(&bar_u, 1);
    for (int i = 0; i < NS; ++i) {
      mbar_init(&bar_a[i], SC);
      mbar_init(&bar_b[i], 1);
      mbar_init(&bar_m[i], 1);
    }
    mbar_arrive_expect_tx(&bar_u, (unsigned)(M * TT * sizeof(V)));
  }
  __syncthreads();
  int b_issued = 0, committed = 0;  // driver: chunks whose copy was issued, whose MMAs were committed
  const bool driver = warp == BW && lane == 0;
  auto copy_b = [&](int c) {
    mbar_arrive_expect_tx(&bar_b[c % NS], bbytes);
    bulk_g2s(sB + (size_t)(c % NS) * MATS * KC * N, d.dense_tc + (size_t)c * MATS * KC * N, bbytes, &bar_b[c % NS]);
    b_issued = c + 1;
  };
  auto drain_b = [&]() {  // the coefficient copies in flight have landed
    for (int c = b_issued > NS ? b_issued - NS : 0; c < b_issued; ++c)
      mbar_wait(&bar_b[c % NS], (c / NS) & 1, kMaxWaitPolls);
  };
  if (driver)  // the first chunks' coefficients, while the kernel before this one still runs
    for (int c = 0; c < NS && c < nch; ++c) copy_b(c);
  grid_sync_wait();
  if (tid < M) bulk_g2s(sU + (size_t)tid * TT, as_t2<float>(d.U) + (size_t)tid * nt + t0, TT * sizeof(V), &bar_u);
  if (__ldcg(d.step) >= d.step_limit) {  // finished solve: the copies land before the CTA leaves
    mbar_wait(&bar_u, 0, kMaxWaitPolls);
    if (driver) drain_b();
    return;
  }
  if (raman_mode >= 2)
    stage_tile_carries<float>(sC, d, PS, nt / TT, blockIdx.x, tile_look(d, nt / TT, TT, raman_mode), lambda_tile(d, TT));
  if (warp == BW) {
    tc::alloc(&s_tmem, COLS);
    tc::relinquish();
  }
  tc::fence_before_sync();
  bool ok = __syncthreads_and(mbar_wait(&bar_u, 0, d.tile_wait_polls) ? 1 : 0);
  const bool u_landed = ok;
  tc::fence_after_sync();
  const uint32_t tmem = s_tmem;
  if (ok && warp < BW) {
    const float kerr = (float)d.one_minus_fR;
    const int f = warp % SC;  // this warp's slot of every other chunk
    for (int c = warp / SC; c < nch; c += kTcBuilders) {
      const int buf = c % NS, q = c * SC + f;
      // chunk c - NS's MMAs read this buffer pair
      if (c >= NS && !mbar_wait_or_warp(&bar_m[buf], ((c / NS) - 1) & 1, &s_stop, polls)) break;
      // lane L's samples 4L .. 4L + 3 of a field: one 16-byte chunk of each operand matrix; the
      // slot's second component goes to the Im matrices, or (REAL) is the next field
      float* a0 = sA + (size_t)buf * MATS * KC * TT + tc::mn_tf32_offset(4 * lane, REAL ? 2 * f : f, A_LBO, A_SBO) / 4;
      float* a1 = REAL ? sA + (size_t)buf * MATS * KC * TT + tc::mn_tf32_offset(4 * lane, 2 * f + 1, A_LBO, A_SBO) / 4
                       : a0 + 2 * KC * TT;
      V x[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      if (q < PS) {  // past the last slot: zeros
        const int4 lm = slot_rows<REAL>(d, q);
        V a[4], b[4], a2[4] = {}, b2[4] = {};
        const V* ul = sU + lm.x * TT + 4 * lane;
        const V* um = sU + lm.y * TT + 4 * lane;
        ld2<float>(ul, a[0], a[1]);
        ld2<float>(ul + 2, a[2], a[3]);
        ld2<float>(um, b[0], b[1]);
        ld2<float>(um + 2, b[2], b[3]);
        if constexpr (REAL) {
          const V* vl = sU + lm.z * TT + 4 * lane;
          const V* vm = sU + lm.w * TT + 4 * lane;
          ld2<float>(vl, a2[0], a2[1]);
          ld2<float>(vl + 2, a2[2], a2[3]);
          ld2<float>(vm, b2[0], b2[1]);
          ld2<float>(vm + 2, b2[2], b2[3]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = slot_value<REAL>(a[e], b[e], a2[e], b2[e]);
        if (raman_mode >= 2) {
          V sr = x[0], si = make_float2(0.f, 0.f);
#pragma unroll
          for (int e = 1; e < 4; ++e) ts.step(sr, si, x[e]);
          ts.enter(sr, si, lane, sC + 2 * q);
          const V kerr2 = make_float2(kerr, kerr);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            ts.step(sr, si, x[e]);
            x[e] = pk_fma(kerr2, x[e], pk_fma(ts.kr2, si, pk_mul(ts.ki2, sr)));
          }
        }
      }
      float rh[4], rl[4], ih[4], il[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        rh[e] = tc::tf32_hi(x[e].x);
        rl[e] = x[e].x - rh[e];
        ih[e] = tc::tf32_hi(x[e].y);
        il[e] = x[e].y - ih[e];
      }
      *reinterpret_cast<float4*>(a0) = make_float4(rh[0], rh[1], rh[2], rh[3]);
      *reinterpret_cast<float4*>(a0 + KC * TT) = make_float4(rl[0], rl[1], rl[2], rl[3]);
      *reinterpret_cast<float4*>(a1) = make_float4(ih[0], ih[1], ih[2], ih[3]);
      *reinterpret_cast<float4*>(a1 + KC * TT) = make_float4(il[0], il[1], il[2], il[3]);
      tc::fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_a[buf]);
    }
  } else if (ok && driver) {
    const uint32_t idesc = tc::idesc_tf32(TT, N, true);
    for (int c = 0; c < nch; ++c) {
      const int buf = c % NS;
      const unsigned par = (c / NS) & 1;
      if (!mbar_wait_or(&bar_b[buf], par, &s_stop, polls) || !mbar_wait_or(&bar_a[buf], par, &s_stop, polls)) break;
      tc::fence_after_sync();
      const float* A = sA + (size_t)buf * MATS * KC * TT;
      const float* B = sB + (size_t)buf * MATS * KC * N;
      // Re: (A Re hi, B Re hi), (Re hi, Re lo), (Re lo, Re hi); Im likewise
      constexpr int ta[3] = {0, 0, 1}, tb[3] = {0, 1, 0};
#pragma unroll
      for (int part = 0; part < PARTS; ++part)
#pragma unroll
        for (int term = 0; term < 3; ++term)
        {
          const float* a = A + (size_t)(2 * part + ta[term]) * KC * TT;
          const float* b = B + (size_t)(2 * part + tb[term]) * KC * N;
          tc::mma_tf32(tmem + 256u * part, tc::desc_mn_tf32(a, A_LBO, A_SBO), tc::desc_kmajor(b, N * 16, 128),
                       idesc, (c > 0 || term > 0) ? 1u : 0u);
        }
      tc::commit(&bar_m[buf]);
      committed = c + 1;
      if (c >= 1 && c - 1 + NS < nch) {  // once chunk c - 1 is done, its coefficients may be replaced
        if (!mbar_wait_or(&bar_m[(c - 1) % NS], ((c - 1) / NS) & 1, &s_stop, polls)) break;
        copy_b(c - 1 + NS);
      }
    }
    // the last chunk's MMAs complete after all earlier ones (in-order issue, one thread)
    if (committed == nch && nch > 0) mbar_wait_or(&bar_m[(nch - 1) % NS], ((nch - 1) / NS) & 1, &s_stop, polls);
  }
  grid_release();
  ok = __syncthreads_and(ok && !s_stop ? 1 : 0);
  tc::fence_after_sync();
  if (ok) {
    // sigma_p(t) = sum_k U_k(t) (T_re + i T_im): warp w reads TMEM lanes 32 (w % 4) .. + 31
    if (warp < BW) {
      const int quad = warp & 3, t = quad * 32 + lane;
      const uint32_t tl = tmem + ((uint32_t)(quad * 32) << 16);
      V* sigma = as_t2<float>(d.sigma);
      for (int p = warp >> 2; p < M; p += BW >> 2) {
        float re[16], im[16];
        tc::ld16(tl + 16u * p, re);
        if constexpr (!REAL) tc::ld16(tl + 256u + 16u * p, im);
        float sx = 0.f, sy = 0.f;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          if (k < M) {
            const V u = sU[k * TT + t];
            if constexpr (REAL) {
              sx = fmaf(u.x, re[k], sx);
              sy = fmaf(u.y, re[k], sy);
            } else {
              sx = fmaf(u.x, re[k], fmaf(-u.y, im[k], sx));
              sy = fmaf(u.x, im[k], fmaf(u.y, re[k], sy));
            }
          }
        }
        sigma[(size_t)p * nt + t0 + t] = make_float2(sx, sy);
      }
    }
  } else {
    if (tid == 0) atomicOr(d.status, kStatusTimeout);
    // nothing may still be writing this CTA's shared memory or TMEM when it leaves: the
    // tile and coefficient copies in flight, the MMAs in flight (each waited for once more)
    if (!u_landed) mbar_wait(&bar_u, 0, kMaxWaitPolls);
    if (driver) {
      drain_b();
      if (committed > 0) mbar_wait(&bar_m[(committed - 1) % NS], ((committed - 1) / NS) & 1, kMaxWaitPolls);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == BW) tc::dealloc(tmem, COLS);
}

// FP64 rows -> T rows (used for the Raman spectrum)
template <typename T>
__global__ void k_to_t2(const double2* __restrict__ in, c2<T>* __restrict__ out, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = from_d2<T>(in[i]);
}

}  // namespace mmp
