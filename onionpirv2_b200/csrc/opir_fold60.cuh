// Arithmetic modulo the 60-bit NTT primes q = 2^60 - c, c < 2^17
// (CONFIG_N2048_K1: c = 2^14 - 1; CONFIG_N4096_K2_MP: c = 2^14 - 1 and
// 2^16 + 2^15 - 1). 2^60 = c (mod q), so a 64-bit word folds to
// (x mod 2^60) + (x / 2^60) c < 2^60 + 15 c, and products need no quotient.
//
// A twiddle w is kept as w and w' = w 2^32 mod q, each in two limbs of 30
// bits: a w = a0 w + a1 w' for the halves a0, a1 of any 64-bit a, so with
//   A0 = a0 w_0 + a1 w'_0 < 2^63,    A1 = a0 w_1 + a1 w'_1 < 2^63
// a w = A0 + 2^30 lo(A1) + 2^62 hi(A1) = A0 + 2^30 lo(A1) + 4 c hi(A1) (mod q)
// below 2^63 + 2^62 + 2^50, folded once. Six 32 x 32 -> 64 multiply-adds and
// one 32-bit multiply, against six and four (one of them carrying) for
// Shoup's two high and low products; and the result is below q + 16 c
// instead of 2q, so the twelve stages of a forward transform need no
// correction at all. On register operands over every SM
// (opir_measure_butterfly_rate): 1,157 G butterflies/s, Shoup's lazy butterfly
// with its corrections 1,007.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace opir60 {

constexpr uint64_t kLow60 = (1ull << 60) - 1;
constexpr uint32_t kLow30 = (1u << 30) - 1;

template <uint64_t Q>
struct Fold {
  static constexpr uint32_t c = static_cast<uint32_t>((1ull << 60) - Q);
  static_assert(Q < (1ull << 60) && (1ull << 60) - Q < (1ull << 17), "q = 2^60 - c, c < 2^17");
};

// w and w 2^32 mod q in limbs of 30 bits (host side of the tables)
inline ulonglong2 twiddle(uint64_t w, uint64_t q) {
  const uint64_t w2 = static_cast<uint64_t>((static_cast<unsigned __int128>(w) << 32) % q);
  return make_ulonglong2((w & kLow30) | ((w >> 30) << 32), (w2 & kLow30) | ((w2 >> 30) << 32));
}

// The 64-bit additions are spelled in halves: left to itself the compiler
// forms them with multiply-adds on the pipe that the products keep busy
// (0.82 of the rate in the probe that chose between them).
__device__ __forceinline__ uint64_t add64(uint64_t a, uint64_t b) {
  uint32_t l, h;
  asm("add.cc.u32 %0, %2, %4;\n\taddc.u32 %1, %3, %5;"
      : "=r"(l), "=r"(h)
      : "r"(static_cast<uint32_t>(a)), "r"(static_cast<uint32_t>(a >> 32)),
        "r"(static_cast<uint32_t>(b)), "r"(static_cast<uint32_t>(b >> 32)));
  return (static_cast<uint64_t>(h) << 32) | l;
}
__device__ __forceinline__ uint64_t mul32(uint32_t a, uint32_t b) {
  uint64_t r;
  asm("mul.wide.u32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint64_t mad32(uint32_t a, uint32_t b, uint64_t c) {
  uint64_t r;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}

// any x -> the same residue below 2^60 + 15 c (below q + 16 c)
template <uint64_t Q>
__device__ __forceinline__ uint64_t fold(uint64_t x) {
  const uint32_t top = static_cast<uint32_t>(x >> 60);
  return add64(x & kLow60, static_cast<uint64_t>(top * Fold<Q>::c));
}
// any x -> [0, q)
template <uint64_t Q>
__device__ __forceinline__ uint64_t canon(uint64_t x) {
  const uint64_t r = fold<Q>(x);
  return min(r, r - Q);
}
// A0 + 2^30 A1 (mod q) for A0 + 2^62 + 2^50 < 2^64, below q + 16 c
template <uint64_t Q>
__device__ __forceinline__ uint64_t join(uint64_t A0, uint64_t A1) {
  const uint32_t l = static_cast<uint32_t>(A1), h = static_cast<uint32_t>(A1 >> 32);
  const uint64_t r = mad32(h, 4 * Fold<Q>::c, A0);
  return fold<Q>(add64(r, (static_cast<uint64_t>(l >> 2) << 32) | (l << 30)));
}
// a w for any a, w as twiddle() keeps it; below q + 16 c
template <uint64_t Q>
__device__ __forceinline__ uint64_t mul(uint64_t a, ulonglong2 w) {
  const uint32_t a0 = static_cast<uint32_t>(a), a1 = static_cast<uint32_t>(a >> 32);
  const uint64_t A1 = mad32(a1, static_cast<uint32_t>(w.y >> 32), mul32(a0, static_cast<uint32_t>(w.x >> 32)));
  const uint64_t A0 = mad32(a1, static_cast<uint32_t>(w.y), mul32(a0, static_cast<uint32_t>(w.x)));
  return join<Q>(A0, A1);
}

// Key products, summed without reduction: with v = v0 + 2^30 v1 and a row word
// w = w0 + 2^30 w1 < q,
//   lo += v0 w0,   hi += v1 w1,   mix += (v0 + v1)(w0 + w1)
// (Karatsuba; mix only counts mod 2^64) take up to five products and a folded
// sum: lo, hi < 5 2^60 + 2^61, mix - lo - hi < 5 2^61. Three multiply-adds a
// product and one join per sum, against Shoup's high and two low 64-bit
// products and a second stored word per row word.
// v folded, in limbs v0 | v1 << 32 (v1 <= 2^30)
template <uint64_t Q>
__device__ __forceinline__ uint64_t limbs(uint64_t v) {
  const uint64_t x = fold<Q>(v);
  return (x & kLow30) | ((x >> 30) << 32);
}
__device__ __forceinline__ void mac(uint64_t &lo, uint64_t &hi, uint64_t &mix, uint64_t v, uint64_t w) {
  const uint32_t v0 = static_cast<uint32_t>(v), v1 = static_cast<uint32_t>(v >> 32);
  const uint32_t w0 = static_cast<uint32_t>(w) & kLow30, w1 = static_cast<uint32_t>(w >> 30);
  lo = mad32(v0, w0, lo);
  hi = mad32(v1, w1, hi);
  mix = mad32(v0 + v1, w0 + w1, mix);
}
// lo + 2^30 (mix - lo - hi) + 2^60 hi (mod q), below q + 16 c: 2^60 hi = c hi
// with c hi = c (hi mod 2^32) + 2^32 y, y = c (hi >> 32) < 2^49, and 2^32 y =
// c (y >> 28) + 2^32 (y mod 2^28). Sum for join(): below 5 2^60 + 2^61 + 2^50.
template <uint64_t Q>
__device__ __forceinline__ uint64_t mac_join(uint64_t lo, uint64_t hi, uint64_t mix) {
  constexpr uint32_t c = Fold<Q>::c;
  const uint64_t y = mul32(static_cast<uint32_t>(hi >> 32), c);
  uint64_t r = mad32(static_cast<uint32_t>(hi), c, lo);
  r = mad32(static_cast<uint32_t>(y >> 28), c, r);
  r += (y & 0xFFFFFFFull) << 32;
  return join<Q>(r, mix - lo - hi);
}

// Forward butterfly (x, y) -> (x + w y, x - w y + q). With inputs in
// [q, 2q) (First adds that q to canonical ones) twelve stages stay between
// q - 12 16 c > 0 and 14 q + 192 c < 2^64.
template <uint64_t Q, bool First = false>
__device__ __forceinline__ void fbf(uint64_t &X, uint64_t &Y, ulonglong2 w) {
  const uint64_t x = X, t = mul<Q>(Y, w);
  X = First ? x + t + Q : x + t;
  Y = First ? x - t + 2 * Q : x - t + Q;
}
// Three forward stages on 8 values; First: canonical inputs.
template <uint64_t Q, bool First>
__device__ __forceinline__ void fpass8(uint64_t (&v)[8], const ulonglong2 (&w)[7]) {
  fbf<Q, First>(v[0], v[4], w[0]); fbf<Q, First>(v[1], v[5], w[0]);
  fbf<Q, First>(v[2], v[6], w[0]); fbf<Q, First>(v[3], v[7], w[0]);
  fbf<Q>(v[0], v[2], w[1]); fbf<Q>(v[1], v[3], w[1]);
  fbf<Q>(v[4], v[6], w[2]); fbf<Q>(v[5], v[7], w[2]);
  fbf<Q>(v[0], v[1], w[3]); fbf<Q>(v[2], v[3], w[4]);
  fbf<Q>(v[4], v[5], w[5]); fbf<Q>(v[6], v[7], w[6]);
}

// Inverse butterfly (x, y) -> (x + y, (x - y) w) with y <= M q; the sum is
// left unfolded.
template <uint64_t Q, int M>
__device__ __forceinline__ void ibf(uint64_t &X, uint64_t &Y, ulonglong2 w) {
  const uint64_t x = X, y = Y;
  X = x + y;
  Y = mul<Q>(x - y + M * Q, w);
}
// Two inverse stages on four folded values: u0 < 4 (q + 16 c), u1 < 2 (..).
template <uint64_t Q>
__device__ __forceinline__ void ipass4(uint64_t &u0, uint64_t &u1, uint64_t &u2, uint64_t &u3,
                                       ulonglong2 wa, ulonglong2 wb, ulonglong2 wc) {
  ibf<Q, 2>(u0, u1, wa);
  ibf<Q, 2>(u2, u3, wb);
  ibf<Q, 3>(u0, u2, wc);
  ibf<Q, 2>(u1, u3, wc);
}
// Three inverse stages on 8 folded values, folded again: sums reach
// 8 (q + 16 c) < 2^64, only v[0..3] grow past q + 16 c.
template <uint64_t Q>
__device__ __forceinline__ void ipass8(uint64_t (&v)[8], const ulonglong2 (&w)[7]) {
  ipass4<Q>(v[0], v[1], v[2], v[3], w[3], w[4], w[1]);
  ipass4<Q>(v[4], v[5], v[6], v[7], w[5], w[6], w[2]);
  ibf<Q, 5>(v[0], v[4], w[0]);
  ibf<Q, 3>(v[1], v[5], w[0]);
  ibf<Q, 2>(v[2], v[6], w[0]);
  ibf<Q, 2>(v[3], v[7], w[0]);
#pragma unroll
  for (int k = 0; k < 4; ++k) v[k] = fold<Q>(v[k]);
}
// The last three inverse stages, N^-1 folded into the third (a = N^-1,
// b = iw[1] N^-1); canonical.
template <uint64_t Q>
__device__ __forceinline__ void ilast8(uint64_t (&v)[8], const ulonglong2 *iw, ulonglong2 a,
                                       ulonglong2 b) {
  ipass4<Q>(v[0], v[1], v[2], v[3], iw[4], iw[5], iw[2]);
  ipass4<Q>(v[4], v[5], v[6], v[7], iw[6], iw[7], iw[3]);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint64_t X = v[k], Y = v[k + 4];
    const uint64_t ra = mul<Q>(X + Y, a), rb = mul<Q>(X - Y + 5 * Q, b);
    v[k] = min(ra, ra - Q);
    v[k + 4] = min(rb, rb - Q);
  }
}

}  // namespace opir60
