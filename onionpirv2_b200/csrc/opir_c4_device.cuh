// Device arithmetic and the register-resident NTT-4096 for the
// CONFIG_N4096_K2_MP parameter set (includes/database_constants.h:111-125):
// N = 4096, two RNS limbs q0 = 2^60 - 2^14 + 1 and q1 = 2^60 - 2^16 - 2^15 + 1
// (the reference's generate_ntt_friendly_primes({60, 60}, 4096)), every
// polynomial as [limb 0 (N)][limb 1 (N)] u64. Included by opir_c4_kernels.cu only
// (it defines constant-memory arrays).
//
// NTT: 512 threads hold 8 coefficients each; the 12 butterfly stages run as
// four radix-8 passes (3 stages each) with three exchanges through a shared
// plane padded by one word per 8 (p -> p + p/8). Thread t holds, per pass,
//   A: t + 512 k            B: 512 (t >> 6) + (t & 63) + 64 k
//   C: 64 (t >> 3) + (t & 7) + 8 k                D: 8 t + k
// and a pass with twiddle base b and group g uses w[b + g] (stage 1),
// w[2b + 2g (+1)] (stage 2), w[4b + 4g + 0..3] (stage 3): A (1, 0),
// B (8, t >> 6), C (64, t >> 3), D (512, t). Merged Cooley-Tukey forward with
// bit-reversed output and Gentleman-Sande inverse scaled by N^-1, the HEXL
// convention of the reference (utils.cpp:26-56). Butterflies fold modulo
// q = 2^60 - c (opir_fold60.cuh): forward values grow by about q a stage from
// [q, 2q) and stay below 2^64, inverse passes begin and end folded.
#pragma once

#include <cstdint>

#include "opir_c4_kernels.h"
#include "opir_fold60.cuh"

namespace opir4 {

constexpr int kThreads = 512;
constexpr int kPad = kN + kN / 8;           // u64 words per padded plane

template <int L>
struct Limb {
  static constexpr uint64_t q = L ? kQ1 : kQ0;
};

// opir60::twiddle() of the twiddles with index < 64: [limb][index]
static __constant__ ulonglong2 c4_fwt[2][64];
static __constant__ ulonglong2 c4_iwt[2][64];
// N^-1 and iw[1] N^-1 per limb
static __constant__ ulonglong2 c4_ninv[2], c4_w1ninv[2];

__device__ __forceinline__ int pad(int p) { return p + (p >> 3); }
__device__ __forceinline__ int posA(int t, int k) { return t + 512 * k; }
__device__ __forceinline__ int posB(int t, int k) { return ((t >> 6) << 9) + (t & 63) + 64 * k; }
__device__ __forceinline__ int posC(int t, int k) { return ((t >> 3) << 6) + (t & 7) + 8 * k; }
__device__ __forceinline__ int posD(int t, int k) { return 8 * t + k; }

template <uint64_t Q>
__device__ __forceinline__ uint64_t add_mod(uint64_t a, uint64_t b) {
  const uint64_t s = a + b;
  return min(s, s - Q);
}
template <uint64_t Q>
__device__ __forceinline__ uint64_t sub_mod(uint64_t a, uint64_t b) {
  const uint64_t d = a - b + Q;
  return min(d, d - Q);
}
template <uint64_t Q>
__device__ __forceinline__ uint64_t neg_mod(uint64_t a) {
  return a ? Q - a : 0;
}

// ----------------------------------------------------------------- NTT
// twiddles of a pass: base b, group g; constant memory when every index < 64
template <int L, bool FWD>
__device__ __forceinline__ void tw_const(ulonglong2 (&w)[7], int b, int g) {
  const ulonglong2 *T = FWD ? c4_fwt[L] : c4_iwt[L];
  w[0] = T[b + g];
  w[1] = T[2 * b + 2 * g];
  w[2] = T[2 * b + 2 * g + 1];
#pragma unroll
  for (int i = 0; i < 4; ++i) w[3 + i] = T[4 * b + 4 * g + i];
}
__device__ __forceinline__ void tw_global(ulonglong2 (&w)[7], const ulonglong2 *T, int b, int g) {
  w[0] = __ldg(T + b + g);
  w[1] = __ldg(T + 2 * b + 2 * g);
  w[2] = __ldg(T + 2 * b + 2 * g + 1);
#pragma unroll
  for (int i = 0; i < 4; ++i) w[3 + i] = __ldg(T + 4 * b + 4 * g + i);
}

template <int P>
__device__ __forceinline__ int posP(int t, int k) {
  return P == 0 ? posA(t, k) : P == 1 ? posB(t, k) : P == 2 ? posC(t, k) : posD(t, k);
}
template <int P>
__device__ __forceinline__ void st_plane(uint64_t *pl, const uint64_t (&v)[8], int t) {
#pragma unroll
  for (int k = 0; k < 8; ++k) pl[pad(posP<P>(t, k))] = v[k];
}
template <int P>
__device__ __forceinline__ void ld_plane(const uint64_t *pl, uint64_t (&v)[8], int t) {
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = pl[pad(posP<P>(t, k))];
}

// forward pass A (A-order in registers) on canonical inputs, or, Shifted, on
// inputs between 192 c and 2q
template <int L, bool Shifted = false>
__device__ __forceinline__ void fA(uint64_t (&v)[8]) {
  ulonglong2 w[7];
  tw_const<L, true>(w, 1, 0);
  opir60::fpass8<Limb<L>::q, !Shifted>(v, w);
}
// Forward passes B and C over np planes stored in A-order (after fA), up to
// a __syncthreads; ends synchronised. Then: ld_plane<3> + fD.
template <int L>
__device__ __forceinline__ void fwd_mid(uint64_t *sm, int np, const Tables &T) {
  constexpr uint64_t Q = Limb<L>::q;
  const int t = threadIdx.x;
  {
    ulonglong2 w[7];
    tw_const<L, true>(w, 8, t >> 6);
#pragma unroll
    for (int i = 0; i < np; ++i) {
      uint64_t v[8];
      ld_plane<1>(sm + i * kPad, v, t);
      opir60::fpass8<Q, false>(v, w);
      st_plane<1>(sm + i * kPad, v, t);
    }
  }
  __syncthreads();
  {
    ulonglong2 w[7];
    tw_global(w, T.fwt[L], 64, t >> 3);
#pragma unroll
    for (int i = 0; i < np; ++i) {
      uint64_t v[8];
      ld_plane<2>(sm + i * kPad, v, t);
      opir60::fpass8<Q, false>(v, w);
      st_plane<2>(sm + i * kPad, v, t);
    }
  }
  __syncthreads();
}
// forward pass D (stages 10-12, D-order values), output any 64 bits
template <int L>
__device__ __forceinline__ void fD(uint64_t (&v)[8], const ulonglong2 (&w)[7]) {
  opir60::fpass8<Limb<L>::q, false>(v, w);
}
template <int L>
__device__ __forceinline__ void fload_d(ulonglong2 (&w)[7], const Tables &T) {
  tw_global(w, T.fwt[L], 512, threadIdx.x);
}

// inverse: pass D first (D-order, inputs folded)
template <int L>
__device__ __forceinline__ void iload_d(ulonglong2 (&w)[7], const Tables &T) {
  tw_global(w, T.iwt[L], 512, threadIdx.x);
}
template <int L>
__device__ __forceinline__ void iD(uint64_t (&v)[8], const ulonglong2 (&w)[7]) {
  opir60::ipass8<Limb<L>::q>(v, w);
}
// Inverse passes C and B over np planes stored in D-order after iD, up to a
// __syncthreads; ends synchronised. Then: ld_plane<0> + iA.
template <int L>
__device__ __forceinline__ void inv_mid(uint64_t *sm, int np, const Tables &T) {
  constexpr uint64_t Q = Limb<L>::q;
  const int t = threadIdx.x;
  {
    ulonglong2 w[7];
    tw_global(w, T.iwt[L], 64, t >> 3);
#pragma unroll
    for (int i = 0; i < np; ++i) {
      uint64_t v[8];
      ld_plane<2>(sm + i * kPad, v, t);
      opir60::ipass8<Q>(v, w);
      st_plane<2>(sm + i * kPad, v, t);
    }
  }
  __syncthreads();
  {
    ulonglong2 w[7];
    tw_const<L, false>(w, 8, t >> 6);
#pragma unroll
    for (int i = 0; i < np; ++i) {
      uint64_t v[8];
      ld_plane<1>(sm + i * kPad, v, t);
      opir60::ipass8<Q>(v, w);
      st_plane<1>(sm + i * kPad, v, t);
    }
  }
  __syncthreads();
}
// last inverse pass (A-order): stages with twiddles 4..7 and 2, 3, then the
// distance-2048 stage with N^-1 folded in; output canonical
template <int L>
__device__ __forceinline__ void iA(uint64_t (&v)[8]) {
  opir60::ilast8<Limb<L>::q>(v, c4_iwt[L], c4_ninv[L], c4_w1ninv[L]);
}

// ------------------------------------------------------ RNS <-> integer
// Garner compose of canonical limbs into [0, q0 q1) (gsw.cpp:22-53); q0inv =
// q0^-1 mod q1 (opir60::twiddle), q0 s = 2^60 s - c0 s
__device__ __forceinline__ unsigned __int128 compose(uint64_t r0, uint64_t r1, ulonglong2 q0inv) {
  uint64_t s = opir60::mul<kQ1>(r1 - r0 + 2 * kQ1, q0inv);  // r0 < q0 < 2 q1
  s = min(s, s - kQ1);
  using u128 = unsigned __int128;
  return (static_cast<u128>(s) << 60) + r0 - static_cast<u128>(s) * opir60::Fold<kQ0>::c;
}

}  // namespace opir4
