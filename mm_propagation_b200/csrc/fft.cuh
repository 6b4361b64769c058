// fft.cuh — the transform of one row of N = 2^LOGN complex samples (precision T) by one CTA or
// by a thread-block cluster of C CTAs, built for sm_100a.
//
// N = A B, both powers of two. Forward (decimation in frequency):
//   first pass   thread i < B takes the A samples x[i + B r] straight from global memory (a
//                warp's loads are consecutive), a radix-A butterfly in registers, the twiddles
//                w_N^{i k_1}, and hands output k_1 to sub-row k_1 in shared memory;
//   row passes   sub-row k_1 (B samples y_{k_1}) is transformed in place by B / A threads (rows of up
//                to 8192 samples: one warp or less): radices R_1, ..., R_m, each pass reading
//                and writing the same positions, so that one synchronisation of those
//                threads separates two passes;
//   last pass    leaves X[k_1 + A k_2] in registers, where the caller works on it.
// The inverse runs the same steps backwards with conjugate twiddles, from registers to
// registers: x[i + B r] ends in the thread that stores it. A spectrum is never put in natural
// order: it is stored in the order of the last pass (radix_plan.h).
//
// With C > 1 the CTA of rank c takes i in [c B/C, (c+1) B/C) in the first pass and keeps the
// sub-rows [c A/C, (c+1) A/C): the first pass's outputs go to their owners through
// distributed shared memory, and the inverse's last step reads them back. Every sample sees the same
// operations in the same order whatever C is, so the bits of a transform do not depend on how
// many CTAs share the row, and C may follow the number of rows at hand.
// (What it measured: see k_nu.)
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"
#include "radix_plan.h"

namespace mmp {
namespace cg = cooperative_groups;

// cos(2*pi*k/32) for any integer k, exact to double rounding.
__host__ __device__ constexpr double cos32(int k) {
  k = ((k % 32) + 32) % 32;
  if (k > 16) k = 32 - k;            // cos is even around 0 (mod 32)
  const bool neg = k > 8;
  if (neg) k = 16 - k;               // cos(pi - x) = -cos(x)
  constexpr double t[9] = {1.0,
                           0.98078528040323044912618223613424,
                           0.92387953251128675612818318939679,
                           0.83146961230254523707878837761791,
                           0.70710678118654752440084436210485,
                           0.55557023301960222474283081394853,
                           0.38268343236508977172845998403040,
                           0.19509032201612826784828486847702,
                           0.0};
  return neg ? -t[k] : t[k];
}

// Multiply v by w_R^e = exp(sgn * 2*pi*i*e / R), sgn = -1 forward, +1 inverse.
// Exact special cases for multiples of pi/4.
template <int R, int E_, bool INV, typename V>
__device__ __forceinline__ V twiddle_const(V v) {
  constexpr int e = ((E_ % R) + R) % R;
  if constexpr (e == 0) {
    return v;
  } else if constexpr ((4 * e) % R == 0) {
    constexpr int quarter = (4 * e) / R;  // 1, 2, 3 quarter turns
    if constexpr (quarter == 2) {
      v.x = -v.x; v.y = -v.y; return v;
    } else {
      // forward: quarter 1 -> -i, quarter 3 -> +i ; inverse: mirrored
      constexpr bool plus_i = (quarter == 1) == INV;
      return crot<plus_i>(v);
    }
  } else {
    using S = decltype(v.x);
    constexpr int k32 = e * (32 / R);
    constexpr double cr = cos32(k32);
    constexpr double si = cos32(k32 - 8);  // sin(2 pi k/32)
    const S c = (S)cr;
    const S s = INV ? (S)si : (S)(-si);
    V r;
    r.x = v.x * c - v.y * s;
    r.y = v.x * s + v.y * c;
    return r;
  }
}

// Complex sums as one packed two-lane operation in FP32 (add.rn.f32x2, and fma.rn.f32x2 by
// -1, which rounds as the subtraction does); the rotated pair of a radix-4 butterfly crosses
// the lanes and stays scalar.
__device__ __forceinline__ float2 pk_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 pk_sub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
__device__ __forceinline__ double2 pk_add(double2 a, double2 b) { return cadd(a, b); }
__device__ __forceinline__ double2 pk_sub(double2 a, double2 b) { return csub(a, b); }

// In-register DFT of size R (power of two <= 32), natural order in and out.
template <int R, bool INV> struct RegDFT;

template <bool INV> struct RegDFT<1, INV> {
  template <typename V> __device__ __forceinline__ static void run(V*) {}
};
template <bool INV> struct RegDFT<2, INV> {
  template <typename V> __device__ __forceinline__ static void run(V* v) {
    const V a = v[0], b = v[1];
    v[0] = pk_add(a, b);
    v[1] = pk_sub(a, b);
  }
};
template <bool INV> struct RegDFT<4, INV> {
  template <typename V> __device__ __forceinline__ static void run(V* v) {
    const V a = v[0], b = v[1], c = v[2], d = v[3];
    const V apc = pk_add(a, c), amc = pk_sub(a, c), bpd = pk_add(b, d);
    const V rot = crot<INV>(pk_sub(b, d));  // forward: -i (b-d); inverse: +i (b-d)
    v[0] = pk_add(apc, bpd);
    v[1] = cadd(amc, rot);
    v[2] = pk_sub(apc, bpd);
    v[3] = csub(amc, rot);
  }
};
// R = A * B with A = 4 (or 2 for R = 8 ... kept at 4 where possible):
// t = a + A*b, k = B*ka + kb:  X[B ka + kb] = sum_a w_A^{a ka} w_R^{a kb} sum_b x[a + A b] w_B^{b kb}
template <int R, bool INV> struct RegDFT {
  static constexpr int A = (R % 4 == 0 && R > 4) ? 4 : 2;
  static constexpr int B = R / A;
  template <typename V> __device__ __forceinline__ static void run(V* v) {
    V y[R];
#pragma unroll
    for (int a = 0; a < A; ++a) {
      V col[B];
#pragma unroll
      for (int b = 0; b < B; ++b) col[b] = v[a + A * b];
      RegDFT<B, INV>::run(col);
#pragma unroll
      for (int kb = 0; kb < B; ++kb) y[a * B + kb] = col[kb];
    }
    apply_tw<0, 0>(y);
#pragma unroll
    for (int kb = 0; kb < B; ++kb) {
      V row[A];
#pragma unroll
      for (int a = 0; a < A; ++a) row[a] = y[a * B + kb];
      RegDFT<A, INV>::run(row);
#pragma unroll
      for (int ka = 0; ka < A; ++ka) v[B * ka + kb] = row[ka];
    }
  }
  // compile-time walk over (a, kb) applying w_R^{a*kb}
  template <int a, int kb, typename V> __device__ __forceinline__ static void apply_tw(V* y) {
    if constexpr (a < A) {
      if constexpr (kb < B) {
        y[a * B + kb] = twiddle_const<R, a * kb, INV>(y[a * B + kb]);
        apply_tw<a, kb + 1>(y);
      } else {
        apply_tw<a + 1, 0>(y);
      }
    }
  }
};

// Geometry of one row transform; the minimal cluster keeps at most 128 KB of a row per CTA,
// XC widens it 2^XC times.
template <typename T, int LOGN_, int XC_ = 0> struct Geo {
  using Real = T;
  static constexpr bool FP64 = sizeof(T) == 8;
  static constexpr int LOGN = LOGN_;
  static constexpr int N = 1 << LOGN;
  static constexpr int LOGSZ = FP64 ? 4 : 3;
  static constexpr int LOGC = ((LOGN + LOGSZ > 17) ? (LOGN + LOGSZ - 17) : 0) + XC_;
  static constexpr int C = 1 << LOGC;
  static constexpr int NL = N / C;
  static constexpr RadixPlan PLAN = radix_plan(LOGN);
  static constexpr int NP = PLAN.n;          // passes
  static constexpr int LOGA = PLAN.r[0], A = 1 << LOGA;
  static constexpr int E = A;                // samples per thread
  static constexpr int LOGB = LOGN - LOGA, B = 1 << LOGB;
  static constexpr int LOGRM = PLAN.r[NP - 1], RM = 1 << LOGRM;  // last pass
  static constexpr int NBF = E / RM;         // its butterflies per thread
  static constexpr int RPC = A / C;          // sub-rows per CTA
  static constexpr int TPR = B / E;          // threads per sub-row
  static constexpr int NTHR = RPC * TPR;     // = B / C
  // length (log2) of the blocks row pass p works on
  __host__ __device__ static constexpr int loglen(int p) {
    int l = LOGB;
    for (int i = 1; i < p; ++i) l -= PLAN.r[i];
    return l;
  }
  // Shared positions are padded by one sample per bank row (16 samples in FP32, 8 in FP64), so
  // that a pass reading and writing at any power-of-two stride spreads over the banks; rows
  // served by less than a bank row of threads start TPR banks apart.
  static constexpr int SLOTS = FP64 ? 8 : 16;
  __host__ __device__ static constexpr int pad(int x) { return x + x / SLOTS; }
  static constexpr int RS0 = pad(B);
  static constexpr int RS = TPR < SLOTS ? RS0 + ((TPR - RS0) % SLOTS + SLOTS) % SLOTS : RS0;
  static constexpr int SMEM_BYTES = RPC * RS * (int)sizeof(c2<T>);
  // 64 registers a thread in FP32 (1024 threads on an SM), 128 in FP64
  static constexpr int REG_BLOCKS = (FP64 ? 512 : 1024) / NTHR;
  static constexpr int MEM_BLOCKS = 222 * 1024 / (SMEM_BYTES + 2048);
  static constexpr int MIN_BLOCKS = REG_BLOCKS < MEM_BLOCKS ? (REG_BLOCKS < 16 ? REG_BLOCKS : 16) : MEM_BLOCKS;
  static constexpr int SYNC_ROWS = RPC > 15 ? 2 : 1;  // sub-rows that share a named barrier
  static_assert(RPC >= 1 && TPR >= 1 && NTHR >= 32 && REG_BLOCKS >= 1, "block size");
  static_assert(MEM_BLOCKS >= 1, "the row fits");

  // The last pass's butterfly b (q_1, ..., q_{m-1}, q_1 most significant): the frequencies
  // it produces are freq0(k1, b) + r KSTR, stored at spec0(k1, b) + r SSTR, r < RM.
  static constexpr int KSTR = N / RM;
  static constexpr int SSTR = B / RM;
  template <int P = 1, int POS = 0, int LOW = LOGB - LOGRM> __device__ __forceinline__ static int digits(int b) {
    if constexpr (P < NP - 1) {  // digits of b from the top
      constexpr int R = PLAN.r[P];
      return (((b >> (LOW - R)) & ((1 << R) - 1)) << POS) + digits<P + 1, POS + R, LOW - R>(b);
    } else {
      return 0;
    }
  }
  __device__ __forceinline__ static int freq0(int k1, int b) { return k1 + (digits(b) << LOGA); }
  __device__ __forceinline__ static int spec0(int k1, int b) { return (k1 << LOGB) + b; }
};

template <bool CONJ, typename V> __device__ __forceinline__ V twiddle(V v, V w) {
  return CONJ ? cmulc(v, w) : cmul(v, w);
}

// Cluster-wide barrier in two halves (every thread of every CTA arrives, then waits).
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// A row kernel on a cluster announces that it runs, before any peer writes to its shared memory
// (row_first waits for that), and leaves only when no peer reads it any more (row_leave).
template <typename Gm> __device__ __forceinline__ void row_enter() {
  if constexpr (Gm::C > 1) cluster_arrive();
}
template <typename Gm> __device__ __forceinline__ void row_leave() {
  if constexpr (Gm::C > 1) cluster_wait();
}

// Threads of one sub-row: between two of its passes.
template <typename Gm> __device__ __forceinline__ void row_sync() {
  if constexpr (Gm::TPR <= 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)threadIdx.x / (Gm::TPR * Gm::SYNC_ROWS)), "n"(Gm::TPR * Gm::SYNC_ROWS) : "memory");
}

// First pass, forward: v[r] = x[i + B r], i = rank NTHR + tid, into the sub-rows. Ends at a
// barrier of all the row's threads (which also publishes whatever else the CTA has staged).
template <typename Gm>
__device__ __forceinline__ void row_first(c2<typename Gm::Real>* v, c2<typename Gm::Real>* s,
                                          const c2<typename Gm::Real>* __restrict__ tw, int rank) {
  using V = c2<typename Gm::Real>;
  const int i = rank * Gm::NTHR + (int)threadIdx.x;
  const V* w = tw + i;
  RegDFT<Gm::A, false>::run(v);
#pragma unroll
  for (int k = 1; k < Gm::A; ++k) v[k] = twiddle<false>(v[k], __ldg(w + k * Gm::B));
  if constexpr (Gm::C == 1) {
    V* d = s + Gm::pad(i);
#pragma unroll
    for (int k = 0; k < Gm::A; ++k) d[k * Gm::RS] = v[k];
    __syncthreads();
  } else {
    cg::cluster_group cl = cg::this_cluster();
    cluster_wait();  // every CTA of the cluster runs
#pragma unroll
    for (int c = 0; c < Gm::C; ++c) {
      V* d = cl.map_shared_rank(s, c) + Gm::pad(i);
#pragma unroll
      for (int k = 0; k < Gm::RPC; ++k) d[k * Gm::RS] = v[c * Gm::RPC + k];
    }
    cluster_arrive();
    cluster_wait();
  }
}

// Row pass P (1 <= P < NP - 1) over this thread's share of its sub-row sr (u-th of TPR).
template <typename Gm, int P, bool INV>
__device__ __forceinline__ void row_pass(c2<typename Gm::Real>* sr,
                                         const c2<typename Gm::Real>* __restrict__ tw, int u) {
  using V = c2<typename Gm::Real>;
  constexpr int LOGR = Gm::PLAN.r[P], R = 1 << LOGR;
  constexpr int LOGL = Gm::loglen(P), LOGS = LOGL - LOGR, S = 1 << LOGS;
#pragma unroll
  for (int bf = 0; bf < Gm::E / R; ++bf) {
    const int b = u + Gm::TPR * bf;
    const int j = b & (S - 1);
    V* d = sr + Gm::pad(((b >> LOGS) << LOGL) + j);
    const V* w = tw + j;
    V v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = d[Gm::pad(r * S)];
    if constexpr (INV) {
#pragma unroll
      for (int q = 1; q < R; ++q) v[q] = twiddle<true>(v[q], __ldg(w + q * S));
    }
    RegDFT<R, INV>::run(v);
    if constexpr (!INV) {
#pragma unroll
      for (int q = 1; q < R; ++q) v[q] = twiddle<false>(v[q], __ldg(w + q * S));
    }
#pragma unroll
    for (int r = 0; r < R; ++r) d[Gm::pad(r * S)] = v[r];
  }
}

// All row passes but the last, forward, each followed by its synchronisation; tw points at
// the row's whole table. OFF: the pass's offset in it.
template <typename Gm, int P = 1, int OFF = Gm::N>
__device__ __forceinline__ void rows_fwd(c2<typename Gm::Real>* sr,
                                         const c2<typename Gm::Real>* __restrict__ tw, int u) {
  if constexpr (P < Gm::NP - 1) {
    row_pass<Gm, P, false>(sr, tw + OFF, u);
    row_sync<Gm>();
    rows_fwd<Gm, P + 1, OFF + (1 << Gm::loglen(P))>(sr, tw, u);
  }
}
// ... inverse, in the opposite order, each preceded by its synchronisation.
template <typename Gm, int P = 1, int OFF = Gm::N>
__device__ __forceinline__ void rows_inv(c2<typename Gm::Real>* sr,
                                         const c2<typename Gm::Real>* __restrict__ tw, int u) {
  if constexpr (P < Gm::NP - 1) {
    rows_inv<Gm, P + 1, OFF + (1 << Gm::loglen(P))>(sr, tw, u);
    row_sync<Gm>();
    row_pass<Gm, P, true>(sr, tw + OFF, u);
  }
}

// The last pass's butterflies of this thread: f(butterfly b, its RM values in shared memory,
// value r at pad(r)).
// f runs the forward or inverse radix-RM step (or both) on them.
template <typename Gm, typename F>
__device__ __forceinline__ void rows_last(c2<typename Gm::Real>* sr, int u, F&& f) {
#pragma unroll 1
  for (int bf = 0; bf < Gm::NBF; ++bf) {
    const int b = u + Gm::TPR * bf;
    f(b, sr + Gm::pad(b * Gm::RM));
  }
}

// Last step, inverse: v[r] = x[i + B r] (unnormalised), i = rank NTHR + tid. Starts with the
// barrier after the row passes; the CTA's shared memory must stay until row_leave.
template <typename Gm>
__device__ __forceinline__ void row_last_inv(c2<typename Gm::Real>* v, c2<typename Gm::Real>* s,
                                             const c2<typename Gm::Real>* __restrict__ tw, int rank) {
  using V = c2<typename Gm::Real>;
  const int i = rank * Gm::NTHR + (int)threadIdx.x;
  const V* w = tw + i;
  if constexpr (Gm::C == 1) {
    __syncthreads();
    const V* d = s + Gm::pad(i);
#pragma unroll
    for (int k = 0; k < Gm::A; ++k) v[k] = d[k * Gm::RS];
  } else {
    cg::cluster_group cl = cg::this_cluster();
    cluster_arrive();
    cluster_wait();
#pragma unroll
    for (int c = 0; c < Gm::C; ++c) {
      const V* d = cl.map_shared_rank(s, c) + Gm::pad(i);
#pragma unroll
      for (int k = 0; k < Gm::RPC; ++k) v[c * Gm::RPC + k] = d[k * Gm::RS];
    }
  }
#pragma unroll
  for (int k = 1; k < Gm::A; ++k) v[k] = twiddle<true>(v[k], __ldg(w + k * Gm::B));
  if constexpr (Gm::C > 1) cluster_arrive();  // this thread has read its peers
  RegDFT<Gm::A, true>::run(v);
}

}  // namespace mmp
