// Client-side batch operations: query packing (PirClient::fast_generate_query,
// src/client.cpp:107-225), response decryption (PirClient::decrypt_mod_q,
// src/client.cpp:364-410) for many queries or responses of one client, and
// its session keys (create_session_keys, src/client.cpp:40-45).
//
// Both are dominated by one negacyclic product x * s with the client's ternary
// secret s. The reference multiplies in the NTT domain mod the target modulus;
// here s is held as two index lists, P (coefficients equal to 1) and M (equal
// to -1), and the product is the exact integer sum
//     (x*s)_i = sum_{j in P} xe[N+i-j] - sum_{j in M} xe[N+i-j]
// over the sign-extended copy xe[N+m] = x[m], xe[m] = -x[m] (m < N) staged in
// shared memory; only the epilogue reduces, so the result equals the NTT
// product mod the same modulus exactly. x is split into parts of at most 31
// bits so each shared word is an int32 and each partial sum fits an int64.
// Three forms of the product. Batches of kTcMinResponses or more, packing and
// decryption, run it as one GEMM on the tensor cores: the client's N x N matrix
// of signed shifts of s by the byte planes of x, an exact integer that the same
// kernel reduces and finishes (k_client_secret_gemm). Below that, and with
// OPIR_CLIENT_TC=0, the index-list form (list_product: one shared load per
// nonzero secret coefficient, output and part) for any batch, and for
// decryption batches that fill the GPU the window form (window_product:
// register windows reused across secret coefficients one block apart, int32
// partial sums), one CTA of kBlock threads per (item, output slice).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <new>
#include <stdexcept>
#include <string>
#include <type_traits>
#include <utility>
#include <vector>

#include "../../include/onionpir_b200.h"
#include "opir_client.h"
#include "opir_host.h"
#include "opir_kernels.h"
#include "opir_params.h"
#include "opir_scan_tc.h"
#include "opir_tc.cuh"

namespace {

using opir::ck;
using opir::DevBuf;
using opir::DeviceGuard;

constexpr int kBlock = 256;
constexpr uint32_t kNoPos = 0xFFFFFFFFu;

// One plaintext-constant addition of a query: c0[limb k][pos] += val[k].
struct ConstEntry {
  uint32_t pos;
  uint32_t pad;
  uint64_t val[2];
};

// xe for one polynomial in NP parts of PB bits, part p at ext + p 2n.
template <int NP, int PB>
__device__ __forceinline__ void stage_ext(const uint64_t *__restrict__ x, uint64_t mod, uint32_t n,
                                          int32_t *ext) {
  constexpr uint64_t kMask = (1ull << PB) - 1;
  for (uint32_t m = threadIdx.x; m < n; m += blockDim.x) {
    const uint64_t v = x[m] % mod;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const int32_t part = static_cast<int32_t>(p + 1 < NP ? (v >> (PB * p)) & kMask : v >> (PB * p));
      ext[2 * n * p + n + m] = part;
      ext[2 * n * p + m] = -part;
    }
  }
}

// Index-list product: acc[p][r] = part p of (x*s)_i for i = i0 + kBlock r,
// one shared load per nonzero secret coefficient, output and part.
template <int NP, int R>
__device__ __forceinline__ void list_product(const int32_t *ext, const uint16_t *sl,
                                             uint32_t npos, uint32_t nneg, uint32_t n,
                                             uint32_t i0, int64_t (&acc)[NP][R]) {
#pragma unroll
  for (int p = 0; p < NP; ++p)
#pragma unroll
    for (int r = 0; r < R; ++r) acc[p][r] = 0;
  const int32_t *e0 = ext + n + i0;
#pragma unroll 4
  for (uint32_t u = 0; u < npos; ++u) {
    const int j = sl[u];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int p = 0; p < NP; ++p) acc[p][r] += e0[2 * n * p + kBlock * r - j];
  }
#pragma unroll 4
  for (uint32_t u = npos; u < npos + nneg; ++u) {
    const int j = sl[u];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int p = 0; p < NP; ++p) acc[p][r] -= e0[2 * n * p + kBlock * r - j];
  }
}

// Window product for n = kBlock J: with j = jl + kBlock jh, the term of output
// i_r = i0 + kBlock r is xe[n + i0 - jl + kBlock (r - jh)], so for one jl the
// thread loads the R + J - 1 window values once into registers and applies
// all J secret coefficients s[jl + kBlock jh] (packed 2 bits each in cs[jl]:
// 1 = +1, 2 = -1, 0 = 0; the same word for every thread, so the branches are
// uniform) to all R outputs. Partial sums run in int32 for F = 2^(31 - PB -
// log2 J) values of jl (each adds at most J terms below 2^PB per output) and
// are then folded into the int64 totals.
template <int NP, int PB, int R, int J>
__device__ __forceinline__ void window_product(const int32_t *ext, const uint32_t *cs, uint32_t n,
                                               uint32_t i0, int64_t (&acc)[NP][R]) {
  constexpr int W = R + J - 1;
  constexpr int kLogJ = J == 16 ? 4 : J == 8 ? 3 : J == 4 ? 2 : J == 2 ? 1 : 0;
  constexpr int F = 1 << (31 - PB - kLogJ);
  static_assert(31 - PB - kLogJ >= 0, "partial sums must fit an int32");
  static_assert((1 << kLogJ) == J, "J is a power of two up to 16");
  int32_t a32[NP][R];
#pragma unroll
  for (int p = 0; p < NP; ++p)
#pragma unroll
    for (int r = 0; r < R; ++r) acc[p][r] = 0, a32[p][r] = 0;
  const int32_t *base = ext + n + i0 - kBlock * (J - 1);
  for (int jl0 = 0; jl0 < kBlock; jl0 += F) {
    const int jend = jl0 + F < kBlock ? jl0 + F : kBlock;
#pragma unroll 1
    for (int jl = jl0; jl < jend; ++jl) {
      const uint32_t c = cs[jl];
      if (c == 0) continue;
      int32_t w[NP][W];
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int d = 0; d < W; ++d) w[p][d] = base[2 * n * p - jl + kBlock * d];
#pragma unroll
      for (int jh = 0; jh < J; ++jh) {
        const uint32_t cc = (c >> (2 * jh)) & 3u;
        if (cc == 1u) {
#pragma unroll
          for (int p = 0; p < NP; ++p)
#pragma unroll
            for (int r = 0; r < R; ++r) a32[p][r] += w[p][r - jh + J - 1];
        } else if (cc == 2u) {
#pragma unroll
          for (int p = 0; p < NP; ++p)
#pragma unroll
            for (int r = 0; r < R; ++r) a32[p][r] -= w[p][r - jh + J - 1];
        }
      }
    }
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
      for (int r = 0; r < R; ++r) acc[p][r] += a32[p][r], a32[p][r] = 0;
  }
}

// sum_p acc[p] 2^(PB p) mod m, canonical.
template <int NP, int PB, int R>
__device__ __forceinline__ uint64_t reduce_parts(const int64_t (&acc)[NP][R], int r, uint64_t m) {
  __int128 v = acc[NP - 1][r];
#pragma unroll
  for (int p = NP - 2; p >= 0; --p) v = v * (static_cast<__int128>(1) << PB) + acc[p][r];
  __int128 x = v % static_cast<__int128>(m);
  if (x < 0) x += m;
  return static_cast<uint64_t>(x);
}

// Constants of the decryption epilogue. When sq t < 2^63 every product fits
// 64 bits and the divisions use Barrett reciprocals mu = floor(2^64 / d):
// mulhi(x, mu) is floor(x / d) or one less (x mu / 2^64 lies in (x/d - 1,
// x/d]), so one correction makes it exact; otherwise (wide) 128-bit division.
struct DecConst {
  uint64_t sq, t, mu_sq, mu_t;
  double inv_sq, inv_t;  // 1/sq, 1/t (wide form)
  uint32_t wide;
  uint32_t narrow;       // sq < 2^24, every dividend below 2^38, both above 2^6:
  uint32_t m_sq, m_t;    // floor(2^38 / d) for 32-bit divisions (div_narrow)
};

// floor(x / d) for x < 2^104 whose quotient is below 2^52: the double
// estimate x (1/d) carries a relative error of a few 2^-53, so it is off by
// at most a small integer, which the exact remainder x - q d corrects
// (long division by an estimated reciprocal with integer correction).
__device__ __forceinline__ uint64_t div_est(unsigned __int128 x, uint64_t d, double inv_d) {
  const double xd = static_cast<double>(static_cast<uint64_t>(x >> 64)) * 18446744073709551616.0 +
                    static_cast<double>(static_cast<uint64_t>(x));
  double qd = xd * inv_d;
  uint64_t q = qd <= 0.0 ? 0 : static_cast<uint64_t>(qd);
  __int128 r = static_cast<__int128>(x) - static_cast<__int128>(static_cast<unsigned __int128>(q) * d);
  for (int it = 0; it < 4 && r < 0; ++it) { --q; r += d; }
  for (int it = 0; it < 4 && r >= static_cast<__int128>(d); ++it) { ++q; r -= d; }
  return q;
}

// (lo + 2^32 hi) mod q, canonical, for |lo|, |hi| below their construction's
// bounds: with the multiple of q (hb 2^32 + lb) added both parts are
// nonnegative, V = hi' 2^32 + lo', and x = floor(V / 2^(32 + sh)) < 2^32.
// m = floor(2^(64 + sh) / q): x m / 2^32 is below V / q by less than
// 1 (m's fraction) + 2^(32 + sh) / q < 2, its floor by less than 3, so the
// quotient estimate from one 32-bit high product leaves a remainder below 3q,
// for which 64-bit words suffice.
struct BigMod {
  uint64_t q, hb, lb;
  uint32_t m, sh;
  __device__ __forceinline__ uint64_t operator()(int64_t lo, int64_t hi) const {
    const uint64_t l = static_cast<uint64_t>(lo) + lb, h = static_cast<uint64_t>(hi) + hb;
    const uint32_t x = static_cast<uint32_t>((h + (l >> 32)) >> sh);
    uint64_t r = l + (h << 32) - __umulhi(x, m) * q;
    r = min(r, r - 2 * q);
    return min(r, r - q);
  }
};
// floor(x / d) for x < 2^38, 2^6 < d: m = floor(2^38 / d) and x / 64 give an
// estimate at most 2 low (x / 64's fraction, m's, the floor), corrected.
__device__ __forceinline__ uint32_t div_narrow(uint64_t x, uint32_t d, uint32_t m) {
  const uint32_t q = __umulhi(static_cast<uint32_t>(x >> 6), m);
  const uint32_t r = static_cast<uint32_t>(x) - q * d;  // below 3 d
  return q + (r >= d) + (r >= 2 * d);
}

__device__ __forceinline__ uint64_t div_barrett(uint64_t x, uint64_t d, uint64_t mu) {
  uint64_t q = __umul64hi(x, mu);
  if (x - q * d >= d) ++q;
  return q;
}

// decrypt_mod_q of one coefficient from prod = (c1 s mod sq): pt =
// round((c0 + prod mod sq) t / sq) mod t; *worst tracks the max noise
// |phase - round(sq m / t)| the reference reports as its noise budget
// (client.cpp:389-407).
__device__ __forceinline__ uint64_t decrypt_coeff(uint64_t prod, uint64_t c0, const DecConst &dc,
                                                  uint64_t &worst) {
  const uint64_t sq = dc.sq, t = dc.t;
  uint64_t m, approx, phase;
  if (!dc.wide) {
    phase = prod + (c0 - div_barrett(c0, sq, dc.mu_sq) * sq);
    if (phase >= sq) phase -= sq;
    m = div_barrett(phase * t + (sq >> 1), sq, dc.mu_sq);
    if (m >= t) m -= t;
    approx = div_barrett(sq * m + (t >> 1), t, dc.mu_t);
    if (approx >= sq) approx -= sq;
  } else {
    phase = prod + c0 % sq;
    if (phase >= sq) phase -= sq;
    m = div_est(static_cast<unsigned __int128>(phase) * t + (sq >> 1), sq, dc.inv_sq);
    if (m >= t) m -= t;
    approx = div_est(static_cast<unsigned __int128>(sq) * m + (t >> 1), t, dc.inv_t);
    if (approx >= sq) approx -= sq;
  }
  const uint64_t pos = phase >= approx ? phase - approx : sq - approx + phase;
  const uint64_t nabs = pos > (sq >> 1) ? sq - pos : pos;
  worst = nabs > worst ? nabs : worst;
  return m;
}

// The same for the narrow moduli, with 32-bit divisions; prod < sq.
__device__ __forceinline__ uint32_t decrypt_narrow(uint32_t prod, uint64_t c0, const DecConst &dc,
                                                   uint32_t &worst) {
  const uint32_t sq = static_cast<uint32_t>(dc.sq), t = static_cast<uint32_t>(dc.t);
  if (c0 >= sq) c0 -= div_barrett(c0, sq, dc.mu_sq) * sq;
  uint32_t phase = prod + static_cast<uint32_t>(c0);
  phase = min(phase, phase - sq);
  uint32_t m = div_narrow(static_cast<uint64_t>(phase) * t + (sq >> 1), sq, dc.m_sq);
  m = m >= t ? m - t : m;
  uint32_t approx = div_narrow(static_cast<uint64_t>(sq) * m + (t >> 1), t, dc.m_t);
  approx = approx >= sq ? approx - sq : approx;
  const uint32_t pos = phase >= approx ? phase - approx : sq - approx + phase;
  worst = max(worst, pos > (sq >> 1) ? sq - pos : pos);
  return m;
}

__device__ __forceinline__ void publish_noise(uint64_t worst, unsigned long long *max_noise) {
  if (!max_noise) return;
  for (int o = 16; o > 0; o >>= 1) {
    const uint64_t w = __shfl_xor_sync(0xFFFFFFFFu, worst, o);
    worst = w > worst ? w : worst;
  }
  if ((threadIdx.x & 31) == 0)
    atomicMax(max_noise + blockIdx.x, static_cast<unsigned long long>(worst));
}

// c0 of one coefficient: -(prod + e) mod q (prod = a s mod q, e any int64).
__device__ __forceinline__ uint64_t pack_coeff(uint64_t prod, int64_t ei, uint64_t q) {
  // |e| is a few units in practice: the 64-bit remainders only for larger ones
  const uint64_t u = static_cast<uint64_t>(ei >= 0 ? ei : -(ei + 1));
  const uint64_t um = u < q ? u : u % q;
  const uint64_t em = ei >= 0 ? um : q - um - 1;
  uint64_t v = prod + em;
  if (v >= q) v -= q;
  return v ? q - v : 0;
}

// The query's plaintext constants that fall in this CTA's output slice
// [o0, o0 + span), after every thread's c0 store (caller synchronises).
__device__ __forceinline__ void add_constants(const ConstEntry *ce, uint32_t nconst, uint32_t limb,
                                              uint32_t o0, uint32_t span, uint64_t q,
                                              uint64_t *c0) {
  for (uint32_t u = threadIdx.x; u < nconst; u += blockDim.x) {
    const uint32_t pos = ce[u].pos;
    if (pos == kNoPos || pos < o0 || pos >= o0 + span) continue;
    const uint64_t v = c0[pos] + ce[u].val[limb];
    c0[pos] = v >= q ? v - q : v;
  }
}

// decrypt_mod_q for response blockIdx.x, output slice blockIdx.y: index-list
// product (any batch) with 31-bit parts.
template <int NP, int R>
__global__ void __launch_bounds__(kBlock) k_client_decrypt(
    const uint64_t *__restrict__ resp, const uint16_t *__restrict__ sidx, uint32_t npos,
    uint32_t nneg, uint32_t n, DecConst dc, uint64_t *__restrict__ pt,
    unsigned long long *__restrict__ max_noise) {
  const uint64_t sq = dc.sq;
  extern __shared__ __align__(16) int32_t smem[];
  int32_t *ext = smem;
  uint16_t *sl = reinterpret_cast<uint16_t *>(smem + NP * 2 * n);
  const uint64_t b = blockIdx.x;
  const uint64_t *c0 = resp + b * 2 * n, *c1 = c0 + n;
  stage_ext<NP, 31>(c1, sq, n, ext);
  for (uint32_t u = threadIdx.x; u < npos + nneg; u += blockDim.x) sl[u] = sidx[u];
  __syncthreads();
  const uint32_t i0 = blockIdx.y * (n / gridDim.y) + threadIdx.x;
  int64_t acc[NP][R];
  list_product<NP, R>(ext, sl, npos, nneg, n, i0, acc);
  uint64_t worst = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t i = i0 + kBlock * r;
    pt[b * n + i] = decrypt_coeff(reduce_parts<NP, 31, R>(acc, r, sq), c0[i], dc, worst);
  }
  publish_noise(worst, max_noise);
}

// The same with the window product (n = kBlock J, PB-bit parts).
template <int NP, int PB, int R, int J>
__global__ void __launch_bounds__(kBlock) k_client_decrypt_w(
    const uint64_t *__restrict__ resp, const uint32_t *__restrict__ code, uint32_t n, DecConst dc,
    uint64_t *__restrict__ pt, unsigned long long *__restrict__ max_noise) {
  const uint64_t sq = dc.sq;
  extern __shared__ __align__(16) int32_t smem[];
  int32_t *ext = smem;
  uint32_t *cs = reinterpret_cast<uint32_t *>(smem + NP * 2 * n);
  const uint64_t b = blockIdx.x;
  const uint64_t *c0 = resp + b * 2 * n, *c1 = c0 + n;
  stage_ext<NP, PB>(c1, sq, n, ext);
  for (uint32_t u = threadIdx.x; u < kBlock; u += blockDim.x) cs[u] = code[u];
  __syncthreads();
  const uint32_t i0 = blockIdx.y * (n / gridDim.y) + threadIdx.x;
  int64_t acc[NP][R];
  window_product<NP, PB, R, J>(ext, cs, n, i0, acc);
  uint64_t worst = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t i = i0 + kBlock * r;
    pt[b * n + i] = decrypt_coeff(reduce_parts<NP, PB, R>(acc, r, sq), c0[i], dc, worst);
  }
  publish_noise(worst, max_noise);
}

// fast_generate_query for item = (query, limb) = blockIdx.x, output slice
// blockIdx.y: c0 = -(a s + e) mod q_k plus the query's plaintext constants,
// c1 = a as given. a and the output are limb-major per query: a [K n], out
// [c0 (K n)][c1 (K n)]. Index-list product with 31-bit parts.
template <int R>
__global__ void __launch_bounds__(kBlock) k_client_pack(
    const uint64_t *__restrict__ a, const int64_t *__restrict__ e,
    const ConstEntry *__restrict__ consts, uint32_t nconst, const uint16_t *__restrict__ sidx,
    uint32_t npos, uint32_t nneg, uint32_t n, uint32_t limbs, uint64_t q0, uint64_t q1,
    uint64_t *__restrict__ out) {
  extern __shared__ __align__(16) int32_t smem[];
  int32_t *ext = smem;
  uint16_t *sl = reinterpret_cast<uint16_t *>(smem + 2 * 2 * n);
  const uint64_t query = blockIdx.x / limbs;
  const uint32_t limb = blockIdx.x % limbs;
  const uint64_t q = limb ? q1 : q0;
  const uint64_t kn = static_cast<uint64_t>(limbs) * n;
  const uint64_t *x = a + query * kn + static_cast<uint64_t>(limb) * n;
  stage_ext<2, 31>(x, q, n, ext);
  for (uint32_t u = threadIdx.x; u < npos + nneg; u += blockDim.x) sl[u] = sidx[u];
  __syncthreads();
  const uint32_t span = n / gridDim.y, o0 = blockIdx.y * span;
  const uint32_t i0 = o0 + threadIdx.x;
  int64_t acc[2][R];
  list_product<2, R>(ext, sl, npos, nneg, n, i0, acc);
  uint64_t *c0 = out + query * 2 * kn + static_cast<uint64_t>(limb) * n;
  uint64_t *c1 = c0 + kn;
  const int64_t *eq = e + query * n;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t i = i0 + kBlock * r;
    c0[i] = pack_coeff(reduce_parts<2, 31, R>(acc, r, q), eq[i], q);
    c1[i] = x[i];
  }
  __syncthreads();
  add_constants(consts + query * nconst, nconst, limb, o0, span, q, c0);
}

// One ciphertext row of the client's session keys (create_session_keys,
// client.cpp:40-45), before the NTT: c0 = -(a s) + esign e + [half = 0] msg,
// c1 = a + [half = 1] msg, msg = scale_k * m for a ternary polynomial m (s for
// the RGSW rows, sigma_k(s) for the BV rows).
struct KeyRow {
  const uint64_t *a;  // K n, coefficient form, limb k below q_k
  const int64_t *e;   // n
  uint64_t *out;      // [c0 (K n)][c1 (K n)]
  uint32_t msg;       // ternary message polynomial: 0 = s, 1 + i = sigma_{N/2^i + 1}(s)
  uint32_t half;      // message in c0 (0) or c1 (1)
  int32_t esign;      // +1: BV row (b = msg - a s + e), -1: encryption of zero
  uint32_t pad;
  uint64_t scale[2];  // message scale per limb, below q_k
};

__device__ __forceinline__ uint64_t signed_mod(int64_t v, uint64_t q) {
  return v >= 0 ? static_cast<uint64_t>(v) % q : (q - static_cast<uint64_t>(-(v + 1)) % q - 1);
}

// Coefficient-form key rows, item = (row, limb) = blockIdx.x, output slice
// blockIdx.y; index-list product with 31-bit parts.
template <int R>
__global__ void __launch_bounds__(kBlock) k_client_keyrows(
    const KeyRow *__restrict__ rows, const int8_t *__restrict__ msgs,
    const uint16_t *__restrict__ sidx, uint32_t npos, uint32_t nneg, uint32_t n, uint32_t limbs,
    uint64_t q0, uint64_t q1) {
  extern __shared__ __align__(16) int32_t smem[];
  int32_t *ext = smem;
  uint16_t *sl = reinterpret_cast<uint16_t *>(smem + 2 * 2 * n);
  const KeyRow row = rows[blockIdx.x / limbs];
  const uint32_t limb = blockIdx.x % limbs;
  const uint64_t q = limb ? q1 : q0;
  const uint64_t kn = static_cast<uint64_t>(limbs) * n;
  const uint64_t *x = row.a + static_cast<uint64_t>(limb) * n;
  stage_ext<2, 31>(x, q, n, ext);
  for (uint32_t u = threadIdx.x; u < npos + nneg; u += blockDim.x) sl[u] = sidx[u];
  __syncthreads();
  const uint32_t i0 = blockIdx.y * (n / gridDim.y) + threadIdx.x;
  int64_t acc[2][R];
  list_product<2, R>(ext, sl, npos, nneg, n, i0, acc);
  uint64_t *c0 = row.out + static_cast<uint64_t>(limb) * n;
  uint64_t *c1 = c0 + kn;
  const int8_t *m = msgs + static_cast<uint64_t>(row.msg) * n;
  const uint64_t sc = row.scale[limb];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t i = i0 + kBlock * r;
    const uint64_t prod = reduce_parts<2, 31, R>(acc, r, q);
    const uint64_t em = signed_mod(row.e[i], q);
    const uint64_t term = m[i] == 1 ? sc : (m[i] == -1 && sc ? q - sc : 0);
    uint64_t v = prod ? q - prod : 0;                        // -(a s)
    if (row.esign > 0) {
      v += em;
      if (v >= q) v -= q;
    } else {
      v = v >= em ? v - em : v + (q - em);
    }
    uint64_t w = x[i] % q;
    if (row.half == 0) {
      v += term;
      if (v >= q) v -= q;
    } else {
      w += term;
      if (w >= q) w -= q;
    }
    c0[i] = v;
    c1[i] = w;
  }
}

// In-place forward negacyclic NTT of polynomial blockIdx.x (limb = index % K)
// in the reference's convention: Cooley-Tukey from natural order, output in
// bit-reversed order, twiddle at butterfly group m + i = root^BitRev(m + i)
// (fw, per limb), every value canonical in [0, q).
__global__ void __launch_bounds__(kBlock) k_client_ntt(uint64_t *__restrict__ polys, uint32_t n,
                                                       uint32_t limbs, const uint64_t *__restrict__ fw,
                                                       uint64_t q0, uint64_t q1) {
  extern __shared__ __align__(16) uint64_t sp[];
  const uint32_t limb = blockIdx.x % limbs;
  const uint64_t q = limb ? q1 : q0;
  const uint64_t *w = fw + static_cast<uint64_t>(limb) * n;
  uint64_t *a = polys + static_cast<uint64_t>(blockIdx.x) * n;
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) sp[i] = a[i];
  __syncthreads();
  for (uint32_t m = 1, t = n >> 1; m < n; m <<= 1, t >>= 1) {
    for (uint32_t b = threadIdx.x; b < n / 2; b += blockDim.x) {
      const uint32_t g = b / t, j = b % t;
      const uint32_t xi = 2 * g * t + j, yi = xi + t;
      const uint64_t u = sp[xi];
      const uint64_t v = static_cast<uint64_t>(static_cast<unsigned __int128>(sp[yi]) * w[m + g] % q);
      const uint64_t s = u + v;
      sp[xi] = s >= q ? s - q : s;
      sp[yi] = u >= v ? u - v : u + (q - v);
    }
    __syncthreads();
  }
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) a[i] = sp[i];
}

// ------------------------------------------------- tensor-core product
// (x s)_i = sum_j S[i][j] x_j with S[i][j] = s[i - j] (i >= j) or
// -s[N + i - j], so with A = S + 1 (entries 0, 1, 2: one unsigned byte plane)
// x s = A x - sum_j x_j, a GEMM over a batch's columns. x comes as NP byte
// planes (3 for a 22-bit small_q, 7 for 50 bits, 8 for a ciphertext modulus),
// so the tensor cores give S_p = A x_p exactly (int32: below 2 N 255 < 2^23)
// and A x = sum_p 2^(8p) S_p is an exact integer; only the finish reduces.
__global__ void __launch_bounds__(kBlock) k_client_secret_matrix(const int8_t *__restrict__ s,
                                                                 uint32_t n,
                                                                 uint8_t *__restrict__ a) {
  const uint32_t i = blockIdx.x;
  for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) {
    const int v = i >= j ? s[i - j] : -s[n + i - j];
    a[static_cast<uint64_t>(i) * n + j] = static_cast<uint8_t>(v + 1);
  }
}

// Byte planes [NP][cols][n] of column blockIdx.x, four coefficients per
// thread and store, and its sums of low and high 32-bit words. Column c is the
// polynomial at x + c x_stride (reduced mod `mod` with mu = floor(2^64 / mod)
// when mod is given), copied to copy + polynomial_of(c) when `copy` is given
// (a query's c1 = a: query c / limbs, limb c % limbs).
template <int NP>
__global__ void __launch_bounds__(kBlock) k_client_planes(
    const uint64_t *__restrict__ x, uint64_t x_stride, uint32_t n, uint32_t cols, uint64_t mod,
    uint64_t mu, uint8_t *__restrict__ planes, uint64_t *__restrict__ colsum,
    uint64_t *__restrict__ copy, uint32_t limbs) {
  __shared__ uint64_t part[2][kBlock / 32];
  const uint64_t c = blockIdx.x;
  const uint64_t *src = x + c * x_stride;
  uint64_t *dst = copy ? copy + ((c / limbs) * 2 * limbs + limbs + c % limbs) * n : nullptr;
  uint64_t lo = 0, hi = 0;
  for (uint32_t j = 4 * threadIdx.x; j < n; j += 4 * kBlock) {
    uint64_t v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = src[j + k];
    if (dst) {
#pragma unroll
      for (int k = 0; k < 4; ++k) dst[j + k] = v[k];
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (mod) {
        v[k] -= __umul64hi(v[k], mu) * mod;
        v[k] = v[k] >= mod ? v[k] - mod : v[k];
      }
      lo += static_cast<uint32_t>(v[k]);
      hi += v[k] >> 32;
    }
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      uint32_t w = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) w |= static_cast<uint32_t>((v[k] >> (8 * p)) & 0xFF) << (8 * k);
      *reinterpret_cast<uint32_t *>(planes + (static_cast<uint64_t>(p) * cols + c) * n + j) = w;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo += __shfl_xor_sync(0xFFFFFFFFu, lo, o);
    hi += __shfl_xor_sync(0xFFFFFFFFu, hi, o);
  }
  if ((threadIdx.x & 31) == 0) {
    part[0][threadIdx.x >> 5] = lo;
    part[1][threadIdx.x >> 5] = hi;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    uint64_t tot = 0;
    for (int w = 0; w < kBlock / 32; ++w) tot += part[threadIdx.x][w];
    colsum[2 * c + threadIdx.x] = tot;
  }
}

// The finish of one output, x s = lo + 2^32 hi of column c at coefficient i:
// compute() is branch-free over a warp's eight columns so that their chains
// interleave, store() follows for the columns that exist. A warp holds 32
// adjacent coefficients of one column.
struct FinishDecrypt {  // pt = round(phase t / sq) and the response's max noise
  const uint64_t *resp;
  uint64_t *pt;
  unsigned long long *noise;
  DecConst dc;
  BigMod mod;     // sq (seven planes)
  uint64_t bias;  // the multiple 2 n + 1 of sq (three planes): |x s| <= n sq
  uint32_t n;
  __device__ __forceinline__ uint64_t operand(uint32_t c, uint32_t i) const {
    return __ldg(resp + static_cast<uint64_t>(c) * (2 * n) + i);
  }
  template <int NP>
  __device__ __forceinline__ uint64_t compute(uint32_t, int64_t lo, int64_t hi, uint64_t c0,
                                              uint64_t &worst) const {
    if (NP == 3) {
      const uint64_t v = static_cast<uint64_t>(lo) + bias;  // below 2^38
      const uint32_t sq = static_cast<uint32_t>(dc.sq);
      uint32_t w = 0;
      const uint32_t m = decrypt_narrow(static_cast<uint32_t>(v) - div_narrow(v, sq, dc.m_sq) * sq, c0, dc, w);
      worst = w;
      return m;
    }
    worst = 0;
    return decrypt_coeff(mod(lo, hi), c0, dc, worst);
  }
  template <int NP>
  __device__ __forceinline__ void store(uint32_t c, uint32_t i, uint64_t v, uint64_t worst) const {
    pt[static_cast<uint64_t>(c) * n + i] = v;
    if (!noise) return;
    if (NP == 3) {
      worst = __reduce_max_sync(0xFFFFFFFFu, static_cast<uint32_t>(worst));
    } else {
      for (int o = 16; o > 0; o >>= 1) {
        const uint64_t w = __shfl_xor_sync(0xFFFFFFFFu, worst, o);
        worst = w > worst ? w : worst;
      }
    }
    if ((threadIdx.x & 31) == 0) atomicMax(noise + c, static_cast<unsigned long long>(worst));
  }
};
struct FinishPack {  // c0 = -(a s + e) mod q_limb (the constants follow)
  const int64_t *e;
  uint64_t *out;
  BigMod mod[2];  // per limb
  uint32_t n, limbs;
  __device__ __forceinline__ uint64_t operand(uint32_t c, uint32_t i) const {
    return static_cast<uint64_t>(__ldg(reinterpret_cast<const long long *>(e) +
                                       static_cast<uint64_t>(limbs == 2 ? c >> 1 : c) * n + i));
  }
  template <int NP>
  __device__ __forceinline__ uint64_t compute(uint32_t c, int64_t lo, int64_t hi, uint64_t ei,
                                              uint64_t &) const {
    const BigMod &b = mod[limbs == 2 ? c & 1 : 0];
    return pack_coeff(b(lo, hi), static_cast<int64_t>(ei), b.q);
  }
  template <int NP>
  __device__ __forceinline__ void store(uint32_t c, uint32_t i, uint64_t v, uint64_t) const {
    const uint32_t query = limbs == 2 ? c >> 1 : c, k = limbs == 2 ? c & 1 : 0;
    out[(static_cast<uint64_t>(query) * 2 * limbs + k) * n + i] = v;
  }
};

struct SecretArgs {
  uint32_t n, cols;
  uint32_t ntile, col_tiles, k_tiles, stages;
  const uint64_t *colsum;
  uint32_t *err;  // one bit per kind of wait
};
constexpr int kSecretThreads = 64 + 256;  // producer, MMA issuer, 8 finishing warps
constexpr uint32_t kMaxSecretStages = 8;

// One CTA: one 128-row tile of A times one tile of ntile columns. Warp 0
// streams 128-byte K slices of the A rows and of the NP planes through a ring
// of shared-memory stages (TMA), warp 1 issues one MMA of N = NP ntile per 32
// bytes of K (all planes of a column tile are one B operand), then eight
// warps read the sums from TMEM, recombine and finish. A CTA takes half an
// SM's shared memory and TMEM, so that one CTA's set-up and finish run beside
// another's loop: at 1024 decryptions the loop and set-up take about 17 us
// alone, the finish 13 (6 of them its DRAM traffic). All waits are bounded; a
// wait that runs out sets its bit of the error word, and the CTA drains its copies and
// MMAs, frees TMEM and returns.
template <int NP, class Fin>
__global__ void __launch_bounds__(kSecretThreads, 2)
k_client_secret_gemm(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_x,
                     SecretArgs a, Fin fin) {
  using namespace opir::tc;
  extern __shared__ __align__(1024) uint8_t sraw[];
  uint8_t *sm = sraw + ((1024u - (sa(sraw) & 1023u)) & 1023u);
  const uint32_t x_plane = a.ntile * 128, stage_bytes = 16384 + NP * x_plane;
  uint64_t *full = reinterpret_cast<uint64_t *>(sm + a.stages * stage_bytes);
  uint64_t *empty = full + kMaxSecretStages, *done = empty + kMaxSecretStages;
  uint32_t *slot = reinterpret_cast<uint32_t *>(done + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ct = blockIdx.x % a.col_tiles, row0 = blockIdx.x / a.col_tiles * 128;
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < a.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sa(slot)),
                 "r"(256u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *slot;
  if (warp == 0) {
    uint32_t issued = 0;
    for (uint32_t kt = 0; kt < a.k_tiles; ++kt) {
      const uint32_t s = kt % a.stages, ph = (kt / a.stages) & 1;
      if (!mbar_wait(&empty[s], ph ^ 1, abort_flag)) {
        if (lane == 0) { *abort_flag = 1; atomicOr(a.err, 1u); }
        break;
      }
      if (lane == 0) {
        uint8_t *st = sm + s * stage_bytes;
        mbar_expect_tx(&full[s], stage_bytes);
        tma_load_3d(st, &tm_a, &full[s], kt * 128, row0, 0);
        for (int p = 0; p < NP; ++p)
          tma_load_3d(st + 16384 + p * x_plane, &tm_x, &full[s], kt * 128, ct * a.ntile, p);
      }
      __syncwarp();
      ++issued;
    }
    for (uint32_t s = 0; s < a.stages; ++s) {  // copies in flight must land before the CTA exits
      const uint32_t uses = (issued + a.stages - 1 - s) / a.stages;
      if (uses == 0) continue;
      const long long t0 = clock64();
      while (!mbar_try(&full[s], (uses - 1) & 1))
        if (clock64() - t0 > kWaitCycles) { if (lane == 0) atomicOr(a.err, 8u); break; }
    }
  } else if (warp == 1) {
    const uint32_t idesc = (2u << 4) | ((NP * a.ntile >> 3) << 17) | (8u << 24);  // u8 x u8 -> s32
    for (uint32_t kt = 0; kt < a.k_tiles; ++kt) {
      const uint32_t s = kt % a.stages, ph = (kt / a.stages) & 1;
      if (!mbar_wait(&full[s], ph, abort_flag)) {
        if (lane == 0) { *abort_flag = 1; atomicOr(a.err, 2u); }
        break;
      }
      fence_after();
      if (lane == 0) {
        const uint32_t base = sa(sm + s * stage_bytes);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          mma_u8(tmem, smem_desc<128>(base + 32 * ks), smem_desc<128>(base + 16384 + 32 * ks), idesc, kt + ks);
        mma_commit(&empty[s]);
      }
      __syncwarp();
    }
    if (lane == 0) mma_commit(done);
    __syncwarp();
    const long long t0 = clock64();
    while (!mbar_try(done, 0))
      if (clock64() - t0 > kWaitCycles) { if (lane == 0) atomicOr(a.err, 16u); break; }
  } else {
    const uint32_t quad = warp & 3, part = (warp - 2) >> 2, chunks = a.ntile / 8;
    const uint32_t i = row0 + quad * 32 + lane;
    // a chunk is eight columns; its operands (c0 of a response, the error of
    // a query) come from DRAM, so they are read one chunk ahead, the first
    // under the main loop
    const auto load = [&](uint64_t (&v)[8], uint32_t u) {
      const uint32_t c = ct * a.ntile + 8 * u;
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = u < chunks && c + k < a.cols ? fin.operand(c + k, i) : 0;
    };
    uint64_t next[8];
    load(next, part);
    const bool ok = mbar_wait(done, 0, abort_flag);
    if (!ok && lane == 0) { *abort_flag = 1; atomicOr(a.err, 4u); }
    fence_after();
    for (uint32_t u = part; ok && u < chunks; u += 2) {
      const uint32_t col0 = ct * a.ntile + 8 * u;
      uint64_t v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = next[k];
      uint32_t S[NP][8];
#pragma unroll
      for (int p = 0; p < NP; ++p)
        tmem_ld8(tmem + (quad << 21) + 8 * u + p * a.ntile, S[p]);
      load(next, u + 2);
      tmem_wait_ld();
      uint64_t worst[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t c = min(col0 + k, a.cols - 1);
        int64_t w[2];  // sums of byte planes 0..3 and 4..7, below 2^47
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (4 * h >= NP) continue;
          uint64_t y = 0;
#pragma unroll
          for (int p = 3; p >= 0; --p)
            if (4 * h + p < NP) y = (y << 8) + S[4 * h + p][k];
          w[h] = static_cast<int64_t>(y) - static_cast<int64_t>(__ldg(a.colsum + 2ull * c + h));
        }
        v[k] = fin.template compute<NP>(c, w[0], NP > 4 ? w[1] : 0, v[k], worst[k]);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (col0 + k < a.cols) fin.template store<NP>(col0 + k, i, v[k], worst[k]);  // uniform
    }
    fence_before();
  }
  __syncthreads();
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u)
                 : "memory");
  }
}

// What the device needs to place a query's plaintext constants itself.
struct PackLayout {
  uint64_t n0, other;      // first-dimension size, rows
  uint32_t num_dims, h;    // dimensions, expansion height
  uint32_t l_ep, pad;
  uint64_t one[2];         // the one-hot's value per limb
  uint64_t gadget[16][2];  // B^(L_EP-1-k) (2^h)^-1 mod q_limb
};

__device__ __forceinline__ uint32_t bitrev_dev(uint64_t x, uint32_t bits) {
  return bits ? static_cast<uint32_t>(__brevll(x) >> (64 - bits)) : 0u;
}

// get_query_indices (src/client.cpp:48-98) for selector bit i >= 1 of index
// idx: the leaf's parity on the incomplete last level, then the perfect-tree
// path MSB first.
__device__ __forceinline__ uint32_t selector_bit(const PackLayout &L, uint64_t idx, uint32_t i) {
  const uint64_t row = idx / L.n0;
  const uint64_t hd = L.num_dims - 1;
  const uint64_t r = 2 * L.other - (1ull << hd), sl = L.other - r;
  uint64_t perfect, first;
  if (row < sl) {
    first = 0;
    perfect = row;
  } else {
    first = (row - sl) % 2;
    perfect = sl + (row - sl) / 2;
  }
  return static_cast<uint32_t>(i == 1 ? first : (perfect >> (hd - i)) & 1ull);
}

// Adds query blockIdx.x's constants (client.cpp:128-225) to its c0 from the
// index: the one-hot at BitRev(col, h), and for each set selector bit i the
// L_EP gadget rows at BitRev(N0 + (i-1) L_EP + k, h), per limb.
__global__ void __launch_bounds__(128) k_client_pack_constants(
    const uint64_t *__restrict__ pt_idx, PackLayout L, uint32_t n, uint32_t limbs, uint64_t q0,
    uint64_t q1, uint64_t *__restrict__ out) {
  const uint64_t b = blockIdx.x;
  uint64_t *c0 = out + b * 2 * limbs * n;
  const uint64_t idx = pt_idx[b];
  const uint32_t nconst = 1 + (L.num_dims - 1) * L.l_ep;
  for (uint32_t u = threadIdx.x; u < limbs * nconst; u += blockDim.x) {
    const uint32_t k = u / nconst, cu = u % nconst;
    const uint64_t q = k ? q1 : q0;
    uint32_t pos;
    uint64_t val;
    if (cu == 0) {
      pos = bitrev_dev(idx % L.n0, L.h);
      val = L.one[k];
    } else {
      const uint32_t i = 1 + (cu - 1) / L.l_ep, r = (cu - 1) % L.l_ep;
      if (!selector_bit(L, idx, i)) continue;
      pos = bitrev_dev(L.n0 + static_cast<uint64_t>(i - 1) * L.l_ep + r, L.h);
      val = L.gadget[r][k];
    }
    uint64_t *cell = c0 + static_cast<uint64_t>(k) * n + pos;
    const uint64_t v = *cell + val;
    *cell = v >= q ? v - q : v;
  }
}


uint64_t bitrev(uint64_t x, uint32_t bits) {
  uint64_t r = 0;
  for (uint32_t i = 0; i < bits; ++i) r |= ((x >> i) & 1ull) << (bits - 1 - i);
  return r;
}

uint64_t mulmod(uint64_t a, uint64_t b, uint64_t m) {
  return static_cast<uint64_t>(static_cast<unsigned __int128>(a) * b % m);
}

}  // namespace

struct opir_client {
  opir_params params{};
  int device = 0;
  int sms = 148;
  uint32_t n = 0, limbs = 1;
  uint64_t mods[2]{};        // ciphertext moduli: the logical q (K = 1) or the two limbs
  DevBuf<uint16_t> sidx;     // [P | M] secret index lists
  uint32_t npos = 0, nneg = 0;
  DevBuf<uint32_t> code;     // [kBlock]: s[jl + kBlock jh] 2 bits each (window product)
  DevBuf<int8_t> msgs;       // [1 + h][n]: s, then sigma_{N/2^i + 1}(s) for i < h
  DevBuf<uint64_t> fw;       // [K][n]: forward NTT twiddles per limb
  DevBuf<KeyRow> keyrows;
  // tensor-core product: A = S + 1 and the error word (built on first use),
  // per-call scratch
  DevBuf<uint8_t> tc_a, tc_q;
  DevBuf<uint64_t> tc_colsum;
  DevBuf<uint32_t> tc_err;
  DevBuf<uint64_t> pk_idx;
  uint64_t *idx_staging = nullptr;   // pinned copy of the last call's indices
  size_t idx_staging_cap = 0;
  // host-buffer calls: the handle's stream and device copies of their buffers
  cudaStream_t io_stream = nullptr;
  DevBuf<uint64_t> io_u0, io_u1, io_out, io_noise;
  DevBuf<int64_t> io_e0, io_e1;
  uint32_t nconst = 1;       // constant slots per query
  uint64_t one_val[2]{};     // the one-hot's value per limb
  std::vector<uint64_t> gadget_val;  // [k][limb]: B^(L_EP-1-k) (2^h)^-1 mod q_limb
  DevBuf<ConstEntry> consts;
  ConstEntry *staging = nullptr;     // pinned host copy of the last call's constants
  size_t staging_cap = 0;
  cudaEvent_t staged = nullptr;      // that copy has been consumed
  std::string last_error;
};

namespace {

template <typename F>
opir_status client_guarded(opir_client *c, F &&f) {
  std::string msg;
  opir_status st = OPIR_OK;
  try {
    f();
  } catch (const std::invalid_argument &e) {
    st = OPIR_ERR_INVALID_ARGUMENT, msg = e.what();
  } catch (const std::out_of_range &e) {
    st = OPIR_ERR_OUT_OF_RANGE, msg = e.what();
  } catch (const std::bad_alloc &) {
    st = OPIR_ERR_NO_MEMORY, msg = "device or host allocation failed";
  } catch (const opir::CudaError &e) {
    cudaGetLastError();
    st = OPIR_ERR_CUDA, msg = e.what();
  } catch (const std::exception &e) {
    cudaGetLastError();
    st = OPIR_ERR_RUNTIME, msg = e.what();
  } catch (...) {
    st = OPIR_ERR_RUNTIME, msg = "unknown error";
  }
  if (c) c->last_error = msg;
  return st;
}

// The layout must be one opir_params_init[_config] produces.
opir_params checked_layout(const opir_params &p) {
  const bool c4 = p.num_limbs == 2 && p.poly_degree == 4096;
  if (!c4 && !(p.num_limbs == 1 && p.poly_degree == 2048 && p.q1 != 0))
    throw std::invalid_argument("unsupported parameter set (CONFIG_N2048_K1_COMP or CONFIG_N4096_K2_MP)");
  if (p.view != OPIR_VIEW_LAYOUT)
    throw std::invalid_argument("a client needs a database layout (opir_params_init[_config])");
  const opir_layout lay{p.target_num_pt, p.expansion_height, p.fst_dim_pow2};
  const opir_params d = c4 ? opir::derive_params_c4(lay) : opir::derive_params(lay);
  if (d.num_pt != p.num_pt || d.q != p.q || d.q1 != p.q1 || d.q2 != p.q2 ||
      d.fst_dim_sz != p.fst_dim_sz || d.num_dims != p.num_dims)
    throw std::invalid_argument("params do not match their layout");
  return d;
}

// get_query_indices (src/client.cpp:48-98): the first-dimension column, then
// one selector bit per further dimension (the leaf's parity on the
// incomplete last level, then the perfect-tree path MSB first).
std::vector<uint64_t> query_indices(const opir_params &p, uint64_t idx) {
  std::vector<uint64_t> out;
  const uint64_t col = idx % p.fst_dim_sz, row = idx / p.fst_dim_sz;
  out.push_back(col);
  if (p.num_dims == 1) return out;
  const uint64_t h = p.num_dims - 1, other = p.other_dim_sz;
  const uint64_t r = 2 * other - (1ull << h), sl = other - r;
  uint64_t perfect;
  if (row < sl) {
    out.push_back(0);
    perfect = row;
  } else {
    const uint64_t corr = row - sl;
    out.push_back(corr % 2);
    perfect = sl + corr / 2;
  }
  for (uint64_t k = h - 1; k-- > 0;) out.push_back((perfect >> k) & 1ull);
  return out;
}

// The values of a query's plaintext constants (client.cpp:128-225), fixed
// per parameter set: the first dimension's one-hot is the BFV lift of
// (2^h)^-1 mod t (under Q = q0 q1 when K = 2, reduced per limb), and selector
// gadget row k is B^(L_EP-1-k) (2^h)^-1 mod q_k.
void prepare_constants(opir_client &c) {
  const opir_params &p = c.params;
  const uint32_t h = p.expansion_height;
  const uint64_t t = p.plain_mod, cap = 1ull << h;
  uint64_t inv_t = 0;
  if (!opir::invert_mod(cap % t, t, inv_t)) throw std::invalid_argument("2^h is not invertible mod t");
  if (c.limbs == 1) {
    const uint64_t q = c.mods[0];
    c.one_val[0] = static_cast<uint64_t>(
        ((static_cast<unsigned __int128>(q) * inv_t + (t >> 1)) / t) % q);
  } else {
    const unsigned __int128 Q = static_cast<unsigned __int128>(c.mods[0]) * c.mods[1];
    const unsigned __int128 delta = Q / t;
    const uint64_t rem = static_cast<uint64_t>(Q - delta * t);
    const uint64_t rem_round =
        static_cast<uint64_t>((static_cast<unsigned __int128>(rem) * inv_t + (t >> 1)) / t);
    const unsigned __int128 scaled = delta * inv_t + rem_round;
    for (uint32_t k = 0; k < 2; ++k) c.one_val[k] = static_cast<uint64_t>(scaled % c.mods[k]);
  }
  c.gadget_val.assign(static_cast<size_t>(p.l_ep) * 2, 0);
  for (uint32_t m = 0; m < c.limbs; ++m) {
    const uint64_t q = c.mods[m];
    uint64_t inv_q = 0;
    if (!opir::invert_mod(cap % q, q, inv_q)) throw std::invalid_argument("2^h is not invertible mod q");
    uint64_t g = 1;  // B^(L_EP-1-k) mod q, k from L_EP - 1 down
    for (uint32_t k = p.l_ep; k-- > 0;) {
      c.gadget_val[2 * k + m] = mulmod(g, inv_q, q);
      g = static_cast<uint64_t>((static_cast<unsigned __int128>(g) << p.base_log2) % q);
    }
  }
}

// The constants of one query: the one-hot at BitRev(col, h), and for each set
// selector bit i the L_EP gadget rows at BitRev(N0 + (i-1) L_EP + k, h).
void query_constants(const opir_client &c, uint64_t idx, ConstEntry *out) {
  const opir_params &p = c.params;
  for (uint32_t u = 0; u < c.nconst; ++u) out[u] = ConstEntry{kNoPos, 0, {0, 0}};
  const std::vector<uint64_t> qi = query_indices(p, idx);
  const uint32_t h = p.expansion_height;
  out[0].pos = static_cast<uint32_t>(bitrev(qi[0], h));
  out[0].val[0] = c.one_val[0];
  out[0].val[1] = c.one_val[1];
  uint32_t at = 1;
  for (size_t i = 1; i < qi.size(); ++i) {
    if (qi[i] != 1) continue;
    for (uint32_t k = 0; k < p.l_ep; ++k) {
      ConstEntry &ce = out[at++];
      ce.pos = static_cast<uint32_t>(bitrev(p.fst_dim_sz + (i - 1) * p.l_ep + k, h));
      ce.val[0] = c.gadget_val[2 * k];
      ce.val[1] = c.gadget_val[2 * k + 1];
    }
  }
}

// make_tree_query's plaintext constants (tree_query.cpp:70-140) for one
// query, W = 2^h_q: the alpha one-hot as the BFV lift of W^-1 mod t at
// BitRev(alpha, h_q) (add_bfv_query_constant), and for every set bit of group
// g (b beta bits, then r gamma bits) the L_EP gadget rows times W^-1 mod q_k
// at BitRev(N0 + g L_EP + row, h_q) (add_rlwe_star_constant).
void tree_query_constants(const opir_client &c, uint64_t n0, uint32_t h_q, uint64_t alpha,
                          const uint8_t *bits, uint32_t groups, ConstEntry *out) {
  const opir_params &p = c.params;
  const uint32_t nconst = 1 + groups * p.l_ep;
  for (uint32_t u = 0; u < nconst; ++u) out[u] = ConstEntry{kNoPos, 0, {0, 0}};
  const uint64_t t = p.plain_mod, W = 1ull << h_q;
  uint64_t w_inv_t = 0;
  if (!opir::invert_mod(W % t, t, w_inv_t)) throw std::invalid_argument("W is not invertible mod t");
  out[0].pos = static_cast<uint32_t>(bitrev(alpha, h_q));
  if (c.limbs == 1) {
    const uint64_t q = c.mods[0];
    out[0].val[0] = static_cast<uint64_t>(
        ((static_cast<unsigned __int128>(q) * w_inv_t + (t >> 1)) / t) % q);
  } else {
    const unsigned __int128 Q = static_cast<unsigned __int128>(c.mods[0]) * c.mods[1];
    const unsigned __int128 delta = Q / t;
    const uint64_t rem = static_cast<uint64_t>(Q - delta * t);
    const uint64_t rem_round =
        static_cast<uint64_t>((static_cast<unsigned __int128>(rem) * w_inv_t + (t >> 1)) / t);
    const unsigned __int128 scaled = delta * w_inv_t + rem_round;
    for (uint32_t k = 0; k < 2; ++k) out[0].val[k] = static_cast<uint64_t>(scaled % c.mods[k]);
  }
  uint64_t w_inv_q[2] = {0, 0};
  for (uint32_t m = 0; m < c.limbs; ++m)
    if (!opir::invert_mod(W % c.mods[m], c.mods[m], w_inv_q[m]))
      throw std::invalid_argument("W is not invertible mod q");
  uint32_t at = 1;
  for (uint32_t g = 0; g < groups; ++g) {
    if (!bits[g]) continue;
    for (uint32_t row = 0; row < p.l_ep; ++row) {
      ConstEntry &ce = out[at++];
      ce.pos = static_cast<uint32_t>(bitrev(n0 + static_cast<uint64_t>(g) * p.l_ep + row, h_q));
      for (uint32_t m = 0; m < c.limbs; ++m) {
        uint64_t gd = 1;  // B^(L_EP-1-row) mod q_m
        for (uint32_t s2 = 0; s2 + 1 + row < p.l_ep; ++s2)
          gd = static_cast<uint64_t>((static_cast<unsigned __int128>(gd) << p.base_log2) % c.mods[m]);
        ce.val[m] = mulmod(gd, w_inv_q[m], c.mods[m]);
      }
    }
  }
}

// Output slices per item so that a batch fills the GPU (index-list
// product); R = n / (s kBlock) outputs per thread, at most kMaxR.
constexpr uint32_t kMaxR = 8;
uint32_t slices_for(uint64_t items, uint32_t n, int sms) {
  uint32_t s = 1;
  while (n / (s * kBlock) > kMaxR) s *= 2;
  while (items * s < 2ull * sms && s * 2 * kBlock <= n) s *= 2;
  return s;
}

// The window product pays when each thread keeps R >= 4 outputs (R + J - 1
// loads serve R J terms); decryption uses it when those slices still give
// every SM a CTA. Query packing keeps the index-list product: its moduli need
// three 20-bit parts in the window form, which issued as many instructions
// per term as the list form at half the occupancy. OPIR_CLIENT_WINDOW=0 keeps
// the index-list product everywhere.
bool window_enabled() {
  const char *v = std::getenv("OPIR_CLIENT_WINDOW");
  return !(v && v[0] == '0');
}
uint32_t window_r(uint64_t items, uint32_t n, int sms) {
  if (!window_enabled() || (n != 2048 && n != 4096)) return 0;
  for (uint32_t R : {8u, 4u})
    if (items * (n / (kBlock * R)) >= static_cast<uint64_t>(sms)) return R;
  return 0;
}

template <typename K>
void set_smem(K kernel, size_t smem, const char *what) {
  ck(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          static_cast<int>(smem)),
     what);
}

void launched(const char *what) {
  ck(cudaGetLastError(), what);
  opir::note_launches(1);
}

DecConst dec_const(const opir_params &p) {
  DecConst dc{};
  dc.sq = p.small_q;
  dc.t = p.plain_mod;
  dc.mu_sq = static_cast<uint64_t>((static_cast<unsigned __int128>(1) << 64) / dc.sq);
  dc.mu_t = static_cast<uint64_t>((static_cast<unsigned __int128>(1) << 64) / dc.t);
  dc.wide = static_cast<unsigned __int128>(dc.sq) * dc.t + dc.sq >= (static_cast<unsigned __int128>(1) << 63);
  dc.inv_sq = 1.0 / static_cast<double>(dc.sq);
  dc.inv_t = 1.0 / static_cast<double>(dc.t);
  dc.narrow = dc.sq < (1ull << 24) && dc.sq > 64 && dc.t > 64 && dc.t < (1ull << 24) &&
              dc.sq * (dc.t + 1) < (1ull << 38) && dc.sq * (3ull * p.poly_degree + 1) < (1ull << 38);
  if (dc.narrow) {
    dc.m_sq = static_cast<uint32_t>((1ull << 38) / dc.sq);
    dc.m_t = static_cast<uint32_t>((1ull << 38) / dc.t);
  }
  return dc;
}

// Reduction of lo + 2^32 hi with |lo| <= 2 n 2^lo_bits, |hi| <= 2 n 2^hi_bits.
BigMod big_mod(uint64_t q, uint32_t n, uint32_t lo_bits, uint32_t hi_bits) {
  uint32_t ln = 1;  // 2 n <= 2^ln
  while ((1ull << ln) < 2ull * n) ++ln;
  using u128 = unsigned __int128;
  BigMod b{};
  b.q = q;
  // hi' + lo' / 2^32 < 2^(hi_bits + ln + 2) + 2^(lo_bits + ln + 2 - 32)
  const uint32_t top = std::max(hi_bits + ln + 3, lo_bits + ln + 3 > 32 ? lo_bits + ln + 3 - 32 : 1);
  b.sh = top > 32 ? top - 32 : 0;
  // the estimate's error and m in 32 bits both need q above 2^(32 + sh), the
  // remainder 3 q in a word
  if (q <= 1ull << (32 + b.sh) || q >> 62)
    throw std::invalid_argument("client product: modulus out of range");
  b.m = static_cast<uint32_t>((static_cast<u128>(1) << (64 + b.sh)) / q);
  // the least multiple of q at or above the magnitude of both parts, split
  // with lb >= 2 n 2^lo_bits
  const u128 need = (static_cast<u128>(1) << (hi_bits + ln + 32)) + (static_cast<u128>(1) << (lo_bits + ln + 1));
  const u128 bias = (need + q - 1) / q * q;
  b.lb = static_cast<uint64_t>(bias & 0xFFFFFFFFu) + (1ull << std::max<uint32_t>(lo_bits + ln, 32));
  b.hb = static_cast<uint64_t>((bias - b.lb) >> 32);
  return b;
}

// The tensor-core form serves decryption and packing batches of at least
// kTcMinResponses (OPIR_CLIENT_TC=0 turns it off).
constexpr uint64_t kTcMinResponses = 32;
bool tc_enabled(uint64_t items) {
  const char *v = std::getenv("OPIR_CLIENT_TC");
  return !(v && v[0] == '0') && window_enabled() && items >= kTcMinResponses;
}

void ensure_secret_matrix(opir_client &c, cudaStream_t st) {
  if (c.tc_a.p) return;
  const uint32_t n = c.n;
  opir::DevBuf<uint8_t> a;
  a.alloc(static_cast<size_t>(n) * n);
  c.tc_err.alloc(1);
  ck(cudaMemsetAsync(c.tc_err.p, 0, sizeof(uint32_t), st), "client error word");
  k_client_secret_matrix<<<n, kBlock, 0, st>>>(c.msgs.p, n, a.p);
  launched("secret matrix launch");
  std::swap(c.tc_a.p, a.p);
  std::swap(c.tc_a.n, a.n);
}

// Columns per tile of the secret product (16, 32 or 64, NP ntile <= 256): the
// largest that leaves one and a half CTAs per SM (an SM holds two), since a
// larger tile reads A fewer times, else the smallest. At 1024 decryptions
// (N = 2048) 64 columns give 256 CTAs and 30 us, 32 give 512 and 33 us; at
// 777 packings 32 columns give 400 CTAs and 46 us.
uint32_t secret_ntile(uint32_t np, uint32_t n, uint64_t cols, int sms) {
  for (uint32_t nt : {64u, 32u})
    if (np * nt <= 256 && n / 128 * ((cols + nt - 1) / nt) >= 3ull * sms / 2) return nt;
  return 16;
}

// planes [NP][cols][n] and colsum as k_client_planes writes them
template <int NP, class Fin>
void secret_product(const opir_client &c, uint64_t cols, const uint8_t *planes,
                    const uint64_t *colsum, const Fin &fin, cudaStream_t st) {
  constexpr size_t kLimit = 113 * 1024;  // half an SM
  const uint32_t n = c.n;
  SecretArgs a{};
  a.n = n;
  a.cols = static_cast<uint32_t>(cols);
  a.ntile = secret_ntile(NP, n, cols, c.sms);
  a.col_tiles = static_cast<uint32_t>((cols + a.ntile - 1) / a.ntile);
  a.k_tiles = n / 128;
  const size_t stage = 16384 + NP * a.ntile * 128;
  a.stages = static_cast<uint32_t>(std::min<size_t>(kMaxSecretStages, (kLimit - 1024 - 256) / stage));
  a.colsum = colsum;
  a.err = c.tc_err.p;
  CUtensorMap map_a, map_x;
  opir::make_plane_map(&map_a, c.tc_a.p, n, n, 1, 128, 128);
  opir::make_plane_map(&map_x, planes, n, cols, NP, a.ntile, 128);
  auto kern = k_client_secret_gemm<NP, Fin>;
  ck(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kLimit)),
     "cudaFuncSetAttribute");
  kern<<<a.col_tiles * (n / 128), kSecretThreads, 1024 + a.stages * stage + 256, st>>>(map_a, map_x,
                                                                                      a, fin);
  launched("client secret product launch");
}

// Synchronises the stream and reports a product whose bounded wait ran out. A
// wait runs out after kWaitCycles SM cycles, so a call that is back sooner than
// these take at 8 GHz, four times the clock, cannot have set the error word,
// and only a later one reads it. The read would add 9 us to every call of 38;
// the word in mapped host memory took no read, but pinning it and giving it
// back took 2.9 ms a client (created, one batch of 64, destroyed: 3.6 ms).
using Clock = std::chrono::steady_clock;
constexpr std::chrono::nanoseconds kReadErrorAfter{opir::tc::kWaitCycles / 8};
void check_product_error(const opir_client &c, cudaStream_t st, Clock::time_point begin,
                         const char *what) {
  ck(cudaStreamSynchronize(st), what);
  if (Clock::now() - begin < kReadErrorAfter) return;
  uint32_t err = 0;
  ck(cudaMemcpyAsync(&err, c.tc_err.p, sizeof(err), cudaMemcpyDeviceToHost, st), what);
  ck(cudaStreamSynchronize(st), what);
  if (err) {
    ck(cudaMemsetAsync(c.tc_err.p, 0, sizeof(err), st), what);
    ck(cudaStreamSynchronize(st), what);
    throw std::runtime_error(std::string(what) + ": tensor-core product gave up (error bits " +
                             std::to_string(err) + ")");
  }
}

// Byte planes and column sums for `cols` columns of np planes.
void ensure_planes(opir_client &c, uint32_t np, uint64_t cols, cudaStream_t st) {
  const uint64_t bytes = static_cast<uint64_t>(np) * cols * c.n;
  if (c.tc_q.n >= bytes && c.tc_colsum.n >= 2 * cols) return;
  ck(cudaStreamSynchronize(st), "client sync");
  if (c.tc_q.n < bytes) c.tc_q.alloc(bytes);
  if (c.tc_colsum.n < 2 * cols) c.tc_colsum.alloc(2 * cols);
}

void launch_pack_tc(uint64_t n_q, const uint64_t *pt_idx, cudaStream_t st, const uint64_t *a,
                    const int64_t *e, opir_client &c, uint64_t *out) {
  const uint32_t n = c.n, limbs = c.limbs;
  const opir_params &p = c.params;
  if (p.l_ep > 16) throw std::runtime_error("client pack: L_EP above 16");
  const Clock::time_point begin = Clock::now();
  ensure_secret_matrix(c, st);
  const uint64_t cols = n_q * limbs;  // one column per query and limb
  ensure_planes(c, 8, cols, st);
  if (c.pk_idx.n < n_q) {
    ck(cudaStreamSynchronize(st), "client sync");
    c.pk_idx.alloc(n_q);
  }
  // the previous call's index upload must have left the staging buffer
  ck(cudaEventSynchronize(c.staged), "client staging wait");
  if (c.idx_staging_cap < n_q) {
    if (c.idx_staging) cudaFreeHost(c.idx_staging);
    c.idx_staging = nullptr;
    c.idx_staging_cap = 0;
    ck(cudaMallocHost(&c.idx_staging, n_q * sizeof(uint64_t)), "client index staging");
    c.idx_staging_cap = n_q;
  }
  std::memcpy(c.idx_staging, pt_idx, n_q * sizeof(uint64_t));
  ck(cudaMemcpyAsync(c.pk_idx.p, c.idx_staging, n_q * sizeof(uint64_t), cudaMemcpyHostToDevice, st),
     "client index upload");
  ck(cudaEventRecord(c.staged, st), "client staging record");
  PackLayout L{};
  L.n0 = p.fst_dim_sz;
  L.other = p.other_dim_sz;
  L.num_dims = p.num_dims;
  L.h = p.expansion_height;
  L.l_ep = p.l_ep;
  L.one[0] = c.one_val[0];
  L.one[1] = c.one_val[1];
  for (uint32_t k = 0; k < p.l_ep; ++k) {
    L.gadget[k][0] = c.gadget_val[2 * k];
    L.gadget[k][1] = c.gadget_val[2 * k + 1];
  }
  k_client_planes<8><<<static_cast<unsigned>(cols), kBlock, 0, st>>>(
      a, n, n, static_cast<uint32_t>(cols), 0, 0, c.tc_q.p, c.tc_colsum.p, out, limbs);
  launched("client planes launch");
  FinishPack fin{};
  fin.e = e;
  fin.out = out;
  fin.n = n;
  fin.limbs = limbs;
  // words of any 64-bit a: both halves below 2^32
  for (uint32_t k = 0; k < limbs; ++k) fin.mod[k] = big_mod(c.mods[k], n, 32, 32);
  secret_product<8>(c, cols, c.tc_q.p, c.tc_colsum.p, fin, st);
  k_client_pack_constants<<<static_cast<unsigned>(n_q), 128, 0, st>>>(c.pk_idx.p, L, n, limbs,
                                                                     c.mods[0], c.mods[1], out);
  launched("client constants launch");
  check_product_error(c, st, begin, "client pack");
}

// Plane counts of a reduced response: 3 (narrow moduli: CONFIG_N2048_K1_COMP's
// 22 bits) or 7 (up to 2^50: CONFIG_N4096_K2_MP's).
void launch_decrypt_tc(uint64_t n_resp, cudaStream_t st, const uint64_t *resp, opir_client &c,
                       uint64_t *pt, unsigned long long *noise) {
  const uint32_t n = c.n, nr = static_cast<uint32_t>(n_resp);
  const Clock::time_point begin = Clock::now();
  ensure_secret_matrix(c, st);
  FinishDecrypt fin{};
  fin.resp = resp;
  fin.pt = pt;
  fin.noise = noise;
  fin.dc = dec_const(c.params);
  fin.n = n;
  const uint64_t sq = c.params.small_q;
  fin.bias = sq * (2ull * n + 1);
  const auto run = [&](auto np) {
    constexpr int NP = decltype(np)::value;
    ensure_planes(c, NP, n_resp, st);
    if (NP > 4) {
      if (sq >> 50) throw std::invalid_argument("client product: small_q above 50 bits");
      fin.mod = big_mod(sq, n, 32, 18);
    }
    k_client_planes<NP><<<nr, kBlock, 0, st>>>(resp + n, 2ull * n, n, nr, sq, fin.dc.mu_sq, c.tc_q.p,
                                               c.tc_colsum.p, nullptr, 1);
    launched("client planes launch");
    secret_product<NP>(c, n_resp, c.tc_q.p, c.tc_colsum.p, fin, st);
  };
  if (fin.dc.narrow) run(std::integral_constant<int, 3>{});
  else run(std::integral_constant<int, 7>{});
  check_product_error(c, st, begin, "client decrypt");
}

void launch_decrypt(uint64_t n_resp, cudaStream_t st, const uint64_t *resp, const opir_client &c,
                    uint64_t *pt, unsigned long long *noise) {
  const uint32_t n = c.n;
  const uint64_t sq = c.params.small_q;
  const DecConst dc = dec_const(c.params);
  const uint32_t nb = static_cast<uint32_t>(n_resp);
  const uint32_t R = sq < (1ull << 50) ? window_r(n_resp, n, c.sms) : 0;
  if (R) {
    const int np = sq < (1ull << 25) ? 1 : 2;
    const dim3 grid(nb, n / (kBlock * R));
    const size_t smem = np * 2 * n * sizeof(int32_t) + kBlock * sizeof(uint32_t);
#define OPIR_DECW(NP, RR, JJ)                                                                  \
  if (np == NP && R == RR && n == kBlock * JJ) {                                              \
    set_smem(k_client_decrypt_w<NP, 25, RR, JJ>, smem, "client decrypt smem");               \
    k_client_decrypt_w<NP, 25, RR, JJ><<<grid, kBlock, smem, st>>>(resp, c.code.p, n, dc, pt, \
                                                                   noise);                    \
    return launched("client decrypt launch");                                                 \
  }
    OPIR_DECW(1, 8, 8) OPIR_DECW(1, 4, 8) OPIR_DECW(1, 8, 16) OPIR_DECW(1, 4, 16)
    OPIR_DECW(2, 8, 8) OPIR_DECW(2, 4, 8) OPIR_DECW(2, 8, 16) OPIR_DECW(2, 4, 16)
#undef OPIR_DECW
    throw std::runtime_error("client decrypt: no window kernel for this shape");
  }
  const uint32_t s = slices_for(n_resp, n, c.sms);
  const uint32_t Rl = n / (s * kBlock);
  const dim3 grid(nb, s);
  const size_t lists = (c.npos + c.nneg + 8) * sizeof(uint16_t);
  const int np = sq < (1ull << 31) ? 1 : 2;
  const size_t smem = np * 2 * n * sizeof(int32_t) + lists;
#define OPIR_DEC(NP, RR)                                                                      \
  if (np == NP && Rl == RR) {                                                                 \
    set_smem(k_client_decrypt<NP, RR>, smem, "client decrypt smem");                          \
    k_client_decrypt<NP, RR><<<grid, kBlock, smem, st>>>(resp, c.sidx.p, c.npos, c.nneg, n,   \
                                                         dc, pt, noise);                      \
    return launched("client decrypt launch");                                                 \
  }
  OPIR_DEC(1, 1) OPIR_DEC(1, 2) OPIR_DEC(1, 4) OPIR_DEC(1, 8)
  OPIR_DEC(2, 1) OPIR_DEC(2, 2) OPIR_DEC(2, 4) OPIR_DEC(2, 8)
#undef OPIR_DEC
  throw std::runtime_error("client decrypt: unsupported slice width");
}

void launch_pack(uint64_t items, cudaStream_t st, const uint64_t *a, const int64_t *e,
                 const opir_client &c, const ConstEntry *consts, uint32_t nconst, uint64_t *out) {
  const uint32_t n = c.n;
  const uint32_t ni = static_cast<uint32_t>(items);
  const uint32_t s = slices_for(items, n, c.sms);
  const uint32_t Rl = n / (s * kBlock);
  const dim3 grid(ni, s);
  const size_t smem = 2 * 2 * n * sizeof(int32_t) + (c.npos + c.nneg + 8) * sizeof(uint16_t);
#define OPIR_PACK(RR)                                                                         \
  if (Rl == RR) {                                                                             \
    set_smem(k_client_pack<RR>, smem, "client pack smem");                                    \
    k_client_pack<RR><<<grid, kBlock, smem, st>>>(a, e, consts, nconst, c.sidx.p,             \
                                                  c.npos, c.nneg, n, c.limbs, c.mods[0],      \
                                                  c.mods[1], out);                            \
    return launched("client pack launch");                                                    \
  }
  OPIR_PACK(1) OPIR_PACK(2) OPIR_PACK(4) OPIR_PACK(8)
#undef OPIR_PACK
  throw std::runtime_error("client pack: unsupported slice width");
}

void launch_keygen(const opir_client &c, const std::vector<KeyRow> &rows, uint64_t *bv,
                   uint64_t bv_polys, uint64_t *gsw, uint64_t gsw_polys, cudaStream_t st) {
  const uint32_t n = c.n;
  const uint64_t items = rows.size() * c.limbs;
  const uint32_t s = slices_for(items, n, c.sms);
  const uint32_t Rl = n / (s * kBlock);
  const dim3 grid(static_cast<uint32_t>(items), s);
  const size_t smem = 2 * 2 * n * sizeof(int32_t) + (c.npos + c.nneg + 8) * sizeof(uint16_t);
  bool done = false;
#define OPIR_KEYROWS(RR)                                                                      \
  if (!done && Rl == RR) {                                                                    \
    set_smem(k_client_keyrows<RR>, smem, "client keygen smem");                               \
    k_client_keyrows<RR><<<grid, kBlock, smem, st>>>(c.keyrows.p, c.msgs.p, c.sidx.p, c.npos, \
                                                     c.nneg, n, c.limbs, c.mods[0],          \
                                                     c.mods[1]);                              \
    launched("client keygen launch");                                                         \
    done = true;                                                                              \
  }
  OPIR_KEYROWS(1) OPIR_KEYROWS(2) OPIR_KEYROWS(4) OPIR_KEYROWS(8)
#undef OPIR_KEYROWS
  if (!done) throw std::runtime_error("client keygen: unsupported slice width");
  for (const auto &part : {std::make_pair(bv, bv_polys), std::make_pair(gsw, gsw_polys)}) {
    if (part.second == 0) continue;
    k_client_ntt<<<static_cast<uint32_t>(part.second), kBlock, n * sizeof(uint64_t), st>>>(
        part.first, n, c.limbs, c.fw.p, c.mods[0], c.mods[1]);
    launched("client keygen NTT launch");
  }
}

}  // namespace

namespace opir {

std::vector<uint64_t> forward_twiddles(const opir_params &p) {
  const uint32_t n = p.poly_degree, limbs = p.num_limbs;
  uint32_t lg = 0;
  while ((1u << lg) < n) ++lg;
  std::vector<uint64_t> fw(static_cast<size_t>(limbs) * n);
  for (uint32_t m = 0; m < limbs; ++m) {
    const uint64_t q = limbs == 1 ? p.q : (m == 0 ? p.q1 : p.q2);
    const uint64_t root = limbs == 1 ? p.w_crt % q : (m == 0 ? p.w1 : p.w2);
    std::vector<uint64_t> pw(n);
    pw[0] = 1 % q;
    for (uint32_t e = 1; e < n; ++e) pw[e] = mulmod(pw[e - 1], root, q);
    for (uint32_t k = 0; k < n; ++k) fw[static_cast<size_t>(m) * n + k] = pw[bitrev(k, lg)];
  }
  return fw;
}

void forward_ntt_polys(uint64_t *d_polys, uint64_t count, const opir_params &p,
                       const uint64_t *d_fw, cudaStream_t st) {
  if (count == 0) return;
  const uint32_t n = p.poly_degree, limbs = p.num_limbs;
  const uint64_t q0 = limbs == 1 ? p.q : p.q1, q1 = limbs == 1 ? 0 : p.q2;
  for (uint64_t done = 0; done < count;) {
    const uint32_t chunk = static_cast<uint32_t>(std::min<uint64_t>(count - done, 1u << 30));
    // chunks keep the limb of polynomial i at i % limbs (chunk sizes are multiples of limbs)
    k_client_ntt<<<chunk, kBlock, n * sizeof(uint64_t), st>>>(d_polys + done * n, n, limbs, d_fw,
                                                            q0, q1);
    launched("NTT launch");
    done += chunk;
  }
}

}  // namespace opir

// Helpers of the host-buffer calls.
namespace {

template <typename T>
T *upload(DevBuf<T> &buf, const T *host, size_t count, cudaStream_t st) {
  buf.alloc(std::max<size_t>(count, 1));
  if (count)
    ck(cudaMemcpyAsync(buf.p, host, count * sizeof(T), cudaMemcpyHostToDevice, st), "upload");
  return buf.p;
}

void ensure_io_stream(opir_client &c) {
  if (!c.io_stream) ck(cudaStreamCreateWithFlags(&c.io_stream, cudaStreamNonBlocking), "client stream");
}

void download(void *host, const void *dev, size_t bytes, cudaStream_t st) {
  ck(cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st), "download");
  ck(cudaStreamSynchronize(st), "client call");
}

}  // namespace

extern "C" {

opir_status opir_client_create(const opir_params *params, const int8_t *secret, int device,
                               opir_client **out) {
  if (!params || !secret || !out) return OPIR_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  opir_client *c = new (std::nothrow) opir_client();
  if (!c) return OPIR_ERR_NO_MEMORY;
  const opir_status st = client_guarded(c, [&] {
    c->params = checked_layout(*params);
    c->device = device;
    c->n = c->params.poly_degree;
    c->limbs = c->params.num_limbs;
    if (c->limbs == 1) {
      c->mods[0] = c->params.q;
    } else {
      c->mods[0] = c->params.q1;
      c->mods[1] = c->params.q2;
    }
    std::vector<uint16_t> lists;
    lists.reserve(c->n);
    for (uint32_t j = 0; j < c->n; ++j) {
      if (secret[j] < -1 || secret[j] > 1)
        throw std::invalid_argument("secret coefficients must be -1, 0 or 1");
      if (secret[j] == 1) lists.push_back(static_cast<uint16_t>(j));
    }
    c->npos = static_cast<uint32_t>(lists.size());
    for (uint32_t j = 0; j < c->n; ++j)
      if (secret[j] == -1) lists.push_back(static_cast<uint16_t>(j));
    c->nneg = static_cast<uint32_t>(lists.size()) - c->npos;
    std::vector<uint32_t> code(kBlock, 0);
    if (c->n % kBlock == 0 && c->n / kBlock <= 16)
      for (uint32_t j = 0; j < c->n; ++j)
        if (secret[j] != 0)
          code[j % kBlock] |= (secret[j] == 1 ? 1u : 2u) << (2 * (j / kBlock));
    c->nconst = 1 + (c->params.num_dims - 1) * c->params.l_ep;
    prepare_constants(*c);
    DeviceGuard g(device);
    ck(cudaEventCreateWithFlags(&c->staged, cudaEventDisableTiming), "client event");
    ck(cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, device), "SM count");
    c->sidx.alloc(std::max<size_t>(lists.size(), 1));
    if (!lists.empty())
      ck(cudaMemcpy(c->sidx.p, lists.data(), lists.size() * sizeof(uint16_t),
                    cudaMemcpyHostToDevice),
         "secret upload");
    c->code.alloc(kBlock);
    ck(cudaMemcpy(c->code.p, code.data(), kBlock * sizeof(uint32_t), cudaMemcpyHostToDevice),
       "secret code upload");
    // key generation: s and its automorphisms sigma_k(s), k = N/2^i + 1
    // (utils.cpp:58-72: coefficient j moves to j k mod 2N, negated past N)
    const uint32_t h = c->params.expansion_height;
    std::vector<int8_t> msgs(static_cast<size_t>(1 + h) * c->n, 0);
    std::copy(secret, secret + c->n, msgs.begin());
    for (uint32_t i = 0; i < h; ++i) {
      const uint64_t k = (c->n >> i) + 1, two_n = 2ull * c->n;
      int8_t *o = msgs.data() + static_cast<size_t>(1 + i) * c->n;
      for (uint64_t j = 0; j < c->n; ++j) {
        const uint64_t dest = j * k % two_n;
        if (dest < c->n) o[dest] = secret[j];
        else o[dest - c->n] = static_cast<int8_t>(-secret[j]);
      }
    }
    c->msgs.alloc(msgs.size());
    ck(cudaMemcpy(c->msgs.p, msgs.data(), msgs.size(), cudaMemcpyHostToDevice), "message upload");
    const std::vector<uint64_t> fw = opir::forward_twiddles(c->params);
    c->fw.alloc(fw.size());
    ck(cudaMemcpy(c->fw.p, fw.data(), fw.size() * sizeof(uint64_t), cudaMemcpyHostToDevice),
       "twiddle upload");
  });
  if (st != OPIR_OK) {
    // device resources exist once the event does; release them on their device
    if (c->staged) opir_client_destroy(c);
    else delete c;
    return st;
  }
  *out = c;
  return OPIR_OK;
}

void opir_client_destroy(opir_client *c) {
  if (!c) return;
  {
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(c->device);
    cudaDeviceSynchronize();
    c->sidx.reset();
    c->code.reset();
    c->msgs.reset();
    c->fw.reset();
    c->keyrows.reset();
    c->tc_a.reset();
    c->tc_q.reset();
    c->tc_colsum.reset();
    c->tc_err.reset();
    c->pk_idx.reset();
    if (c->idx_staging) cudaFreeHost(c->idx_staging);
    c->consts.reset();
    if (c->staging) cudaFreeHost(c->staging);
    if (c->staged) cudaEventDestroy(c->staged);
    c->io_u0.reset();
    c->io_u1.reset();
    c->io_out.reset();
    c->io_noise.reset();
    c->io_e0.reset();
    c->io_e1.reset();
    if (c->io_stream) cudaStreamDestroy(c->io_stream);
    if (prev >= 0) cudaSetDevice(prev);
  }
  delete c;
}

const char *opir_client_last_error(const opir_client *c) {
  return c ? c->last_error.c_str() : "null client handle";
}

opir_status opir_client_generate_queries_device(opir_client *c, uint32_t n,
                                                const uint64_t *pt_idx, const uint64_t *d_a,
                                                const int64_t *d_e, uint64_t *d_queries,
                                                void *stream) {
  if (!c) return OPIR_ERR_INVALID_ARGUMENT;
  return client_guarded(c, [&] {
    if (n == 0) return;
    if (!pt_idx || !d_a || !d_e || !d_queries) throw std::invalid_argument("null buffer");
    for (uint32_t i = 0; i < n; ++i)
      if (pt_idx[i] >= c->params.num_pt)
        throw std::out_of_range("PIR plaintext index exceeds the runtime layout");
    DeviceGuard g(c->device);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (tc_enabled(n)) {
      launch_pack_tc(n, pt_idx, st, d_a, d_e, *c, d_queries);
      return;
    }
    const size_t count = static_cast<size_t>(n) * c->nconst;
    // the previous call's upload must have left the staging buffer
    ck(cudaEventSynchronize(c->staged), "client staging wait");
    if (c->staging_cap < count) {
      if (c->staging) cudaFreeHost(c->staging);
      c->staging = nullptr;
      c->staging_cap = 0;
      ck(cudaMallocHost(&c->staging, count * sizeof(ConstEntry)), "client staging");
      c->staging_cap = count;
    }
    for (uint32_t i = 0; i < n; ++i)
      query_constants(*c, pt_idx[i], c->staging + static_cast<size_t>(i) * c->nconst);
    if (c->consts.n < count) {
      ck(cudaStreamSynchronize(st), "client sync");
      c->consts.alloc(count);
    }
    ck(cudaMemcpyAsync(c->consts.p, c->staging, count * sizeof(ConstEntry),
                       cudaMemcpyHostToDevice, st),
       "client constants upload");
    ck(cudaEventRecord(c->staged, st), "client staging record");
    launch_pack(static_cast<uint64_t>(n) * c->limbs, st, d_a, d_e, *c, c->consts.p, c->nconst,
                d_queries);
  });
}

opir_status opir_client_decrypt_device(opir_client *c, uint32_t n, const uint64_t *d_responses,
                                       uint64_t *d_plaintexts, uint64_t *d_max_noise,
                                       void *stream) {
  if (!c) return OPIR_ERR_INVALID_ARGUMENT;
  return client_guarded(c, [&] {
    if (n == 0) return;
    if (!d_responses || !d_plaintexts) throw std::invalid_argument("null buffer");
    DeviceGuard g(c->device);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (d_max_noise)
      ck(cudaMemsetAsync(d_max_noise, 0, static_cast<size_t>(n) * sizeof(uint64_t), st),
         "noise reset");
    auto *noise = reinterpret_cast<unsigned long long *>(d_max_noise);
    if (tc_enabled(n))
      launch_decrypt_tc(n, st, d_responses, *c, d_plaintexts, noise);
    else
      launch_decrypt(n, st, d_responses, *c, d_plaintexts, noise);
  });
}

opir_status opir_client_keygen_device(opir_client *c, const uint64_t *d_bv_a,
                                      const int64_t *d_bv_e, const uint64_t *d_gsw_a,
                                      const int64_t *d_gsw_e, uint64_t *d_bv_keys,
                                      uint64_t *d_gsw_key, void *stream) {
  if (!c) return OPIR_ERR_INVALID_ARGUMENT;
  return client_guarded(c, [&] {
    const opir_params &p = c->params;
    const uint32_t h = p.expansion_height, K = c->limbs, n = c->n;
    if (h && (!d_bv_a || !d_bv_e || !d_bv_keys)) throw std::invalid_argument("null BV buffer");
    if (!d_gsw_a || !d_gsw_e || !d_gsw_key) throw std::invalid_argument("null RGSW buffer");
    const uint64_t kn = static_cast<uint64_t>(K) * n;
    auto power = [&](uint32_t bits, uint32_t m) {  // 2^bits mod q_m
      uint64_t v = 1 % c->mods[m];
      for (uint32_t b = 0; b < bits; ++b) v = mulmod(v, 2, c->mods[m]);
      return v;
    };
    std::vector<KeyRow> rows;
    for (uint32_t i = 0; i < h; ++i)
      for (uint32_t r = 0; r < p.l_ks; ++r) {
        const uint64_t at = static_cast<uint64_t>(i) * p.l_ks + r;
        KeyRow kr{d_bv_a + at * kn, d_bv_e + at * n, d_bv_keys + at * 2 * kn, 1 + i, 0, 1, 0, {0, 0}};
        for (uint32_t m = 0; m < K; ++m) kr.scale[m] = power(r * p.base_log2_ks, m);
        rows.push_back(kr);
      }
    for (uint32_t half = 0; half < 2; ++half)
      for (uint32_t r = 0; r < p.l_key; ++r) {
        const uint64_t at = static_cast<uint64_t>(half) * p.l_key + r;
        KeyRow kr{d_gsw_a + at * kn, d_gsw_e + at * n, d_gsw_key + at * 2 * kn, 0, half, -1, 0, {0, 0}};
        for (uint32_t m = 0; m < K; ++m) kr.scale[m] = power(p.base_log2_key * (p.l_key - 1 - r), m);
        rows.push_back(kr);
      }
    DeviceGuard g(c->device);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (c->keyrows.n < rows.size()) {
      ck(cudaStreamSynchronize(st), "client sync");
      c->keyrows.alloc(rows.size());
    }
    ck(cudaMemcpyAsync(c->keyrows.p, rows.data(), rows.size() * sizeof(KeyRow),
                       cudaMemcpyHostToDevice, st),
       "key row upload");
    launch_keygen(*c, rows, d_bv_keys, static_cast<uint64_t>(h) * p.l_ks * 2 * K, d_gsw_key,
                  2ull * p.l_key * 2 * K, st);
  });
}

// ---- host-buffer forms: the same calls on host arrays (same layouts), on
// the handle's own stream; each returns when its results are in host memory.

opir_status opir_client_generate_queries(opir_client *c, uint32_t n, const uint64_t *pt_idx,
                                         const uint64_t *a, const int64_t *e,
                                         uint64_t *queries) {
  if (!c) return OPIR_ERR_INVALID_ARGUMENT;
  if (n == 0) return OPIR_OK;
  const size_t kn = static_cast<size_t>(c->limbs) * c->n;
  opir_status st = client_guarded(c, [&] {
    if (!pt_idx || !a || !e || !queries) throw std::invalid_argument("null buffer");
    DeviceGuard g(c->device);
    ensure_io_stream(*c);
    upload(c->io_u0, a, n * kn, c->io_stream);
    upload(c->io_e0, e, static_cast<size_t>(n) * c->n, c->io_stream);
    c->io_out.alloc(n * 2 * kn);
  });
  if (st != OPIR_OK) return st;
  st = opir_client_generate_queries_device(c, n, pt_idx, c->io_u0.p, c->io_e0.p, c->io_out.p,
                                           c->io_stream);
  if (st != OPIR_OK) return st;
  return client_guarded(c, [&] {
    DeviceGuard g(c->device);
    download(queries, c->io_out.p, n * 2 * kn * sizeof(uint64_t), c->io_stream);
  });
}

opir_status opir_client_decrypt(opir_client *c, uint32_t n, const uint64_t *responses,
                                uint64_t *plaintexts, uint64_t *max_noise) {
  if (!c) return OPIR_ERR_INVALID_ARGUMENT;
  if (n == 0) return OPIR_OK;
  opir_status st = client_guarded(c, [&] {
    if (!responses || !plaintexts) throw std::invalid_argument("null buffer");
    DeviceGuard g(c->device);
    ensure_io_stream(*c);
    upload(c->io_u0, responses, static_cast<size_t>(n) * 2 * c->n, c->io_stream);
    c->io_out.alloc(static_cast<size_t>(n) * c->n);
    if (max_noise) c->io_noise.alloc(n);
  });
  if (st != OPIR_OK) return st;
  st = opir_client_decrypt_device(c, n, c->io_u0.p, c->io_out.p, max_noise ? c->io_noise.p : nullptr,
                                  c->io_stream);
  if (st != OPIR_OK) return st;
  return client_guarded(c, [&] {
    DeviceGuard g(c->device);
    if (max_noise)
      ck(cudaMemcpyAsync(max_noise, c->io_noise.p, n * sizeof(uint64_t), cudaMemcpyDeviceToHost,
                         c->io_stream),
         "download");
    download(plaintexts, c->io_out.p, static_cast<size_t>(n) * c->n * sizeof(uint64_t),
             c->io_stream);
  });
}

opir_status opir_client_keygen(opir_client *c, const uint64_t *bv_a, const int64_t *bv_e,
                               const uint64_t *gsw_a, const int64_t *gsw_e, uint64_t *bv_keys,
                               uint64_t *gsw_key) {
  if (!c) return OPIR_ERR_INVALID_ARGUMENT;
  const opir_params &p = c->params;
  const size_t kn = static_cast<size_t>(c->limbs) * c->n;
  const size_t bv_rows = static_cast<size_t>(p.expansion_height) * p.l_ks;
  const size_t gsw_rows = 2ull * p.l_key;
  opir_status st = client_guarded(c, [&] {
    if (bv_rows && (!bv_a || !bv_e || !bv_keys)) throw std::invalid_argument("null BV buffer");
    if (!gsw_a || !gsw_e || !gsw_key) throw std::invalid_argument("null RGSW buffer");
    DeviceGuard g(c->device);
    ensure_io_stream(*c);
    upload(c->io_u0, bv_a, bv_rows * kn, c->io_stream);
    upload(c->io_e0, bv_e, bv_rows * c->n, c->io_stream);
    upload(c->io_u1, gsw_a, gsw_rows * kn, c->io_stream);
    upload(c->io_e1, gsw_e, gsw_rows * c->n, c->io_stream);
    c->io_out.alloc((bv_rows + gsw_rows) * 2 * kn);
  });
  if (st != OPIR_OK) return st;
  st = opir_client_keygen_device(c, bv_rows ? c->io_u0.p : nullptr, bv_rows ? c->io_e0.p : nullptr,
                                 c->io_u1.p, c->io_e1.p, bv_rows ? c->io_out.p : nullptr,
                                 c->io_out.p + bv_rows * 2 * kn, c->io_stream);
  if (st != OPIR_OK) return st;
  return client_guarded(c, [&] {
    DeviceGuard g(c->device);
    if (bv_rows)
      ck(cudaMemcpyAsync(bv_keys, c->io_out.p, bv_rows * 2 * kn * sizeof(uint64_t),
                         cudaMemcpyDeviceToHost, c->io_stream),
         "download");
    download(gsw_key, c->io_out.p + bv_rows * 2 * kn, gsw_rows * 2 * kn * sizeof(uint64_t),
             c->io_stream);
  });
}

opir_status opir_client_generate_tree_queries(opir_client *c, const opir_tree_params *tree,
                                              uint32_t n, const uint64_t *alpha,
                                              const uint8_t *bits, uint32_t groups,
                                              const uint64_t *a, const int64_t *e,
                                              uint64_t *queries) {
  if (!c) return OPIR_ERR_INVALID_ARGUMENT;
  return client_guarded(c, [&] {
    if (n == 0) return;
    if (!tree || !alpha || (groups && !bits) || !a || !e || !queries)
      throw std::invalid_argument("null buffer");
    const opir_params &p = c->params;
    const uint64_t n0 = tree->N0;
    const uint32_t h_q = static_cast<uint32_t>(tree->h_q);
    if ((1ull << h_q) > c->n || n0 + static_cast<uint64_t>(groups) * p.l_ep > (1ull << h_q))
      throw std::invalid_argument("tree query shape does not fit the polynomial");
    for (uint32_t i = 0; i < n; ++i)
      if (alpha[i] >= n0) throw std::out_of_range("tree query alpha exceeds N0");
    const uint32_t nconst = 1 + groups * p.l_ep;
    const size_t count = static_cast<size_t>(n) * nconst;
    const size_t kn = static_cast<size_t>(c->limbs) * c->n;
    DeviceGuard g(c->device);
    ensure_io_stream(*c);
    cudaStream_t st = c->io_stream;
    ck(cudaEventSynchronize(c->staged), "client staging wait");
    if (c->staging_cap < count) {
      if (c->staging) cudaFreeHost(c->staging);
      c->staging = nullptr;
      c->staging_cap = 0;
      ck(cudaMallocHost(&c->staging, count * sizeof(ConstEntry)), "client staging");
      c->staging_cap = count;
    }
    for (uint32_t i = 0; i < n; ++i)
      tree_query_constants(*c, n0, h_q, alpha[i], bits + static_cast<size_t>(i) * groups, groups,
                           c->staging + static_cast<size_t>(i) * nconst);
    if (c->consts.n < count) {
      ck(cudaStreamSynchronize(st), "client sync");
      c->consts.alloc(count);
    }
    ck(cudaMemcpyAsync(c->consts.p, c->staging, count * sizeof(ConstEntry),
                       cudaMemcpyHostToDevice, st),
       "client constants upload");
    ck(cudaEventRecord(c->staged, st), "client staging record");
    upload(c->io_u0, a, n * kn, st);
    upload(c->io_e0, e, static_cast<size_t>(n) * c->n, st);
    c->io_out.alloc(n * 2 * kn);
    launch_pack(static_cast<uint64_t>(n) * c->limbs, st, c->io_u0.p, c->io_e0.p, *c, c->consts.p,
                nconst, c->io_out.p);
    download(queries, c->io_out.p, n * 2 * kn * sizeof(uint64_t), st);
  });
}

}  // extern "C"
