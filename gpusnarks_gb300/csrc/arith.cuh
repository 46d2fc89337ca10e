// Device field arithmetic for the NTT path: Montgomery multiplication and
// modular add/sub written as PTX carry chains.
//
// Replaces the reference's generic C++ limb loops (cuda/device_field_operators.h:
// _add :104-117, _subtract :120-137, ciosMontgomeryMultiply :151-187,
// Scalar::add/subtract/mul :190-214) with register-resident carry chains:
//   * products:  mad.lo.cc / madc.lo.cc / mad.hi.cc / madc.hi.cc
//   * add / sub: add.cc / addc, sub.cc / subc, then a branch-free select
// and uses the correct CIOS constant -p^-1 mod 2^32 per field (the reference
// hard-codes 0xFFFFFFFF, device_field_operators.h:47).
//
// Element layout is the reference's: uint32_t limbs, little-endian
// (cuda/device_field.h:75).  Values are canonical, in [0, p), where a function's
// comment gives no wider range (K = 2: below 2p; the unreduced sums: below 2^k p).
// Montgomery products compute a*b*R^-1 mod p with R = 2^(32*N); they serve
// products of two data elements.  The transform's products are by table
// constants: fe_mul_tw computes x*w whatever representation x is held in
// (the one-limb field stores w*R and takes the Montgomery product).
#pragma once
#include <cstdint>

#include "fields_gen.h"

namespace gsn {
namespace ptx {

// Every carry-chain step is its own volatile asm statement: the carry flag is
// invisible to the compiler, and volatile keeps the statements of one chain in
// program order.
__device__ __forceinline__ void mad_lo_cc(uint32_t& d, uint32_t a, uint32_t b, uint32_t c) {
  asm volatile("mad.lo.cc.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
}
__device__ __forceinline__ void madc_lo_cc(uint32_t& d, uint32_t a, uint32_t b, uint32_t c) {
  asm volatile("madc.lo.cc.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
}
__device__ __forceinline__ void mad_hi_cc(uint32_t& d, uint32_t a, uint32_t b, uint32_t c) {
  asm volatile("mad.hi.cc.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
}
__device__ __forceinline__ void madc_hi_cc(uint32_t& d, uint32_t a, uint32_t b, uint32_t c) {
  asm volatile("madc.hi.cc.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
}
__device__ __forceinline__ void madc_hi(uint32_t& d, uint32_t a, uint32_t b, uint32_t c) {
  asm volatile("madc.hi.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
}
__device__ __forceinline__ void mad_lo(uint32_t& d, uint32_t a, uint32_t b, uint32_t c) {
  asm volatile("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
}
__device__ __forceinline__ void madc_lo(uint32_t& d, uint32_t a, uint32_t b, uint32_t c) {
  asm volatile("madc.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
}
__device__ __forceinline__ void add_cc(uint32_t& d, uint32_t a, uint32_t b) {
  asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
}
__device__ __forceinline__ void addc_cc(uint32_t& d, uint32_t a, uint32_t b) {
  asm volatile("addc.cc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
}
__device__ __forceinline__ void addc(uint32_t& d, uint32_t a, uint32_t b) {
  asm volatile("addc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
}
__device__ __forceinline__ void sub_cc(uint32_t& d, uint32_t a, uint32_t b) {
  asm volatile("sub.cc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
}
__device__ __forceinline__ void subc_cc(uint32_t& d, uint32_t a, uint32_t b) {
  asm volatile("subc.cc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
}
__device__ __forceinline__ void subc(uint32_t& d, uint32_t a, uint32_t b) {
  asm volatile("subc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
}
__device__ __forceinline__ uint32_t mul_hi(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.hi.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

}  // namespace ptx

template <class P>
struct Fe {
  uint32_t l[P::N];
};

// ---------------------------------------------------------------------------
// One-limb fields (p32).  p > 2^31, so there is no headroom for lazy sums:
// every operation returns a canonical value.
// ---------------------------------------------------------------------------
template <class P>
__device__ __forceinline__ uint32_t mul1(uint32_t a, uint32_t b) {
  // Montgomery product with R = 2^32, subtractive form: m = lo * p^-1, so
  // a*b - m*p has a zero low word and equals (hi - mulhi(m,p)) * 2^32,
  // which lies in (-p*2^32, p*2^32).
  constexpr uint32_t p = P::mod(0);
  constexpr uint32_t pinv_pos = 0u - P::PINV;  // +p^-1 mod 2^32
  uint32_t lo = a * b;
  uint32_t hi = ptx::mul_hi(a, b);
  uint32_t m = lo * pinv_pos;
  uint32_t mh = ptx::mul_hi(m, p);
  uint32_t r = hi - mh;
  return (hi < mh) ? r + p : r;
}
// mul1 with w' = w * p^-1 mod 2^32 supplied: Montgomery's m = (a w mod 2^32) p^-1 equals a w' mod 2^32,
// so a product with a reused w costs one multiply less.  Same result as mul1(a, w).
template <class P>
__device__ __forceinline__ uint32_t mul1_pre(uint32_t a, uint32_t w, uint32_t wp) {
  constexpr uint32_t p = P::mod(0);
  const uint32_t hi = ptx::mul_hi(a, w);
  const uint32_t m = a * wp;
  const uint32_t mh = ptx::mul_hi(m, p);
  const uint32_t r = hi - mh;
  return (hi < mh) ? r + p : r;
}
template <class P>
__device__ __forceinline__ uint32_t mul1_wp(uint32_t w) {  // w' for mul1_pre
  return w * (0u - P::PINV);
}
template <class P>
__device__ __forceinline__ uint32_t add1(uint32_t a, uint32_t b) {
  constexpr uint32_t p = P::mod(0);
  uint32_t t = p - b;  // in [1, p]
  uint32_t r = a - t;
  return (a < t) ? r + p : r;
}
template <class P>
__device__ __forceinline__ uint32_t sub1(uint32_t a, uint32_t b) {
  constexpr uint32_t p = P::mod(0);
  uint32_t r = a - b;
  return (a < b) ? r + p : r;
}

// ---------------------------------------------------------------------------
// Multi-limb fields, one element per thread.
// ---------------------------------------------------------------------------

// Limb i of K p, K = 1 or 2 (2p fits the limbs: HEADROOM >= 2).
template <class P, int K>
__host__ __device__ constexpr uint32_t mod_times(int i) {
  static_assert(K == 1 || (K == 2 && P::HEADROOM >= 2), "K p must fit the limbs");
  return K == 1 ? P::mod(i) : (P::mod(i) << 1) | (i > 0 ? P::mod(i - 1) >> 31 : 0u);
}

// r = a + b mod K p.  Inputs below K p.
template <class P, int K = 1>
__device__ __forceinline__ void fe_add(Fe<P>& r, const Fe<P>& a, const Fe<P>& b) {
  constexpr int N = P::N;
  if constexpr (N == 1) {
    r.l[0] = add1<P>(a.l[0], b.l[0]);
  } else {
    uint32_t s[N], d[N], c, mask;
    ptx::add_cc(s[0], a.l[0], b.l[0]);
#pragma unroll
    for (int j = 1; j < N; ++j) ptx::addc_cc(s[j], a.l[j], b.l[j]);
    ptx::addc(c, 0u, 0u);
    ptx::sub_cc(d[0], s[0], mod_times<P, K>(0));
#pragma unroll
    for (int j = 1; j < N; ++j) ptx::subc_cc(d[j], s[j], mod_times<P, K>(j));
    ptx::subc(mask, c, 0u);  // 0xFFFFFFFF iff s < K p (no carry and a borrow)
#pragma unroll
    for (int j = 0; j < N; ++j) r.l[j] = (s[j] & mask) | (d[j] & ~mask);
  }
}

// r = a - b mod K p.  Inputs below K p.
template <class P, int K = 1>
__device__ __forceinline__ void fe_sub(Fe<P>& r, const Fe<P>& a, const Fe<P>& b) {
  constexpr int N = P::N;
  if constexpr (N == 1) {
    r.l[0] = sub1<P>(a.l[0], b.l[0]);
  } else {
    uint32_t d[N], mask;
    ptx::sub_cc(d[0], a.l[0], b.l[0]);
#pragma unroll
    for (int j = 1; j < N; ++j) ptx::subc_cc(d[j], a.l[j], b.l[j]);
    ptx::subc(mask, 0u, 0u);  // 0xFFFFFFFF iff a < b
    ptx::add_cc(r.l[0], d[0], mod_times<P, K>(0) & mask);
#pragma unroll
    for (int j = 1; j < N - 1; ++j) ptx::addc_cc(r.l[j], d[j], mod_times<P, K>(j) & mask);
    ptx::addc(r.l[N - 1], d[N - 1], mod_times<P, K>(N - 1) & mask);
  }
}

// Sums and differences without a reduction, for a field whose limbs have room for many multiples of p (MNT4-753 r: 2^15).
// Values below 2^k p in, below 2^(k+1) p out; a difference adds 2^k p to stay positive.
constexpr int kMaxLazyLog = 12;
template <class P>
struct ShiftedMod {
  uint32_t limb[kMaxLazyLog + 1][P::N];
  constexpr ShiftedMod() : limb{} {
    for (int k = 0; k <= kMaxLazyLog; ++k)
      for (int j = 0; j < P::N; ++j)
        limb[k][j] = (P::mod(j) << k) | (k > 0 && j > 0 ? P::mod(j - 1) >> (32 - k) : 0u);
  }
};
template <class P>
static __constant__ ShiftedMod<P> c_shifted_mod{};

template <class P>
__device__ __forceinline__ void fe_add_lazy(Fe<P>& r, const Fe<P>& a, const Fe<P>& b) {
  constexpr int N = P::N;
  ptx::add_cc(r.l[0], a.l[0], b.l[0]);
#pragma unroll
  for (int j = 1; j < N - 1; ++j) ptx::addc_cc(r.l[j], a.l[j], b.l[j]);
  ptx::addc(r.l[N - 1], a.l[N - 1], b.l[N - 1]);
}
template <class P>
__device__ __forceinline__ void fe_sub_lazy(Fe<P>& r, const Fe<P>& a, const Fe<P>& b, int k) {
  constexpr int N = P::N;
  uint32_t d[N];
  ptx::sub_cc(d[0], a.l[0], b.l[0]);
#pragma unroll
  for (int j = 1; j < N - 1; ++j) ptx::subc_cc(d[j], a.l[j], b.l[j]);
  ptx::subc(d[N - 1], a.l[N - 1], b.l[N - 1]);
  const uint32_t* const m = c_shifted_mod<P>.limb[k];
  ptx::add_cc(r.l[0], d[0], m[0]);
#pragma unroll
  for (int j = 1; j < N - 1; ++j) ptx::addc_cc(r.l[j], d[j], m[j]);
  ptx::addc(r.l[N - 1], d[N - 1], m[N - 1]);
}

// -p^-1 mod 2^32, the factor of each reduction row's m = t_0 * (-p^-1).  For a modulus with p_0 = 1
// (BLS12-381 r) it is 0xFFFFFFFF.  When the compiler can see that value it rewrites m = -t_0 and the
// reduction row that uses m, at a cost of about 44 more multiply-pipe instructions per 8-limb product
// (measured on GB300: 180.5 against 139.5 per product, 57 against 64 G products/s, the same outputs).
// There the factor is read from constant memory, whose contents the compiler does not assume; every
// other field keeps the immediate.
template <class P>
static __constant__ uint32_t c_row_pinv = P::PINV;

template <class P>
__device__ __forceinline__ uint32_t row_pinv() {
  if constexpr (P::N > 1 && P::PINV == 0xFFFFFFFFu) {
    return c_row_pinv<P>;
  } else {
    return P::PINV;
  }
}

// One CIOS reduction step on the accumulator t[0..N+1]: m = t0 * (-p^-1),
// t += m*p (t0 becomes 0), then t >>= 32.
template <class P>
__device__ __forceinline__ void cios_reduce_step(uint32_t (&t)[P::N + 2]) {
  constexpr int N = P::N;
  const uint32_t m = t[0] * row_pinv<P>();
  ptx::mad_lo_cc(t[0], m, P::mod(0), t[0]);
#pragma unroll
  for (int j = 1; j < N; ++j) ptx::madc_lo_cc(t[j], m, P::mod(j), t[j]);
  ptx::addc_cc(t[N], t[N], 0u);
  ptx::addc(t[N + 1], t[N + 1], 0u);
  ptx::mad_hi_cc(t[1], m, P::mod(0), t[1]);
#pragma unroll
  for (int j = 1; j < N; ++j) ptx::madc_hi_cc(t[j + 1], m, P::mod(j), t[j + 1]);
  ptx::addc(t[N + 1], t[N + 1], 0u);
#pragma unroll
  for (int j = 0; j <= N; ++j) t[j] = t[j + 1];
  t[N + 1] = 0u;
}

// r = a * b * R^-1 mod p (CIOS, Koc-Acar-Kaliski), lo and hi partial
// products in two carry chains per row.  Inputs canonical; output canonical.
template <class P>
__device__ __forceinline__ void fe_mul_rows(Fe<P>& r, const Fe<P>& a, const Fe<P>& b) {
  constexpr int N = P::N;
  if constexpr (N == 1) {
    r.l[0] = mul1<P>(a.l[0], b.l[0]);
  } else {
    uint32_t t[N + 2];
    {  // row 0: t = a * b0
      const uint32_t bi = b.l[0];
#pragma unroll
      for (int j = 0; j < N; ++j) t[j] = a.l[j] * bi;
      ptx::mad_hi_cc(t[1], a.l[0], bi, t[1]);
#pragma unroll
      for (int j = 1; j < N - 1; ++j) ptx::madc_hi_cc(t[j + 1], a.l[j], bi, t[j + 1]);
      ptx::madc_hi(t[N], a.l[N - 1], bi, 0u);
      t[N + 1] = 0u;
      cios_reduce_step<P>(t);
    }
#pragma unroll
    for (int i = 1; i < N; ++i) {
      const uint32_t bi = b.l[i];
      ptx::mad_lo_cc(t[0], a.l[0], bi, t[0]);
#pragma unroll
      for (int j = 1; j < N; ++j) ptx::madc_lo_cc(t[j], a.l[j], bi, t[j]);
      ptx::addc_cc(t[N], t[N], 0u);
      ptx::addc(t[N + 1], 0u, 0u);
      ptx::mad_hi_cc(t[1], a.l[0], bi, t[1]);
#pragma unroll
      for (int j = 1; j < N; ++j) ptx::madc_hi_cc(t[j + 1], a.l[j], bi, t[j + 1]);
      ptx::addc(t[N + 1], t[N + 1], 0u);
      cios_reduce_step<P>(t);
    }
    // t < 2p: one conditional subtraction
    uint32_t d[N], mask;
    ptx::sub_cc(d[0], t[0], P::mod(0));
#pragma unroll
    for (int j = 1; j < N; ++j) ptx::subc_cc(d[j], t[j], P::mod(j));
    ptx::subc(mask, t[N], 0u);  // 0xFFFFFFFF iff t < p
#pragma unroll
    for (int j = 0; j < N; ++j) r.l[j] = (t[j] & mask) | (d[j] & ~mask);
  }
}

// ---------------------------------------------------------------------------
// Even/odd-accumulator CIOS.  Same result as fe_mul_rows, different schedule:
// every carry chain adds whole 64-bit products a_j*b into a non-overlapping
// pair of accumulator words (mad.lo.cc then madc.hi.cc on the same operands,
// into consecutive words), so each pair can issue as one wide multiply-add.
// Even-indexed limbs accumulate into E, odd-indexed limbs into O one word
// higher: T = E + 2^32 O.  After the reduction row E_0 is zero and
// T / 2^32 = (O + E_1) + 2^32 (E_2 .. E_N), so the accumulators swap roles
// each row (the merge of fe_mul_eo below).
// ---------------------------------------------------------------------------

// acc[0..N] += sum_k x[2k + off] * y * 2^(64 k)
template <int N>
__device__ __forceinline__ void pair_chain(uint32_t (&acc)[N + 1], const uint32_t* x, int off, uint32_t y) {
  ptx::mad_lo_cc(acc[0], x[off], y, acc[0]);
  ptx::madc_hi_cc(acc[1], x[off], y, acc[1]);
#pragma unroll
  for (int k = 1; k < N / 2; ++k) {
    ptx::madc_lo_cc(acc[2 * k], x[2 * k + off], y, acc[2 * k]);
    ptx::madc_hi_cc(acc[2 * k + 1], x[2 * k + off], y, acc[2 * k + 1]);
  }
  ptx::addc(acc[N], acc[N], 0u);
}

// Same on the modulus limbs (compile-time constants).
template <class P>
__device__ __forceinline__ void pair_chain_mod(uint32_t (&acc)[P::N + 1], int off, uint32_t y) {
  constexpr int N = P::N;
  ptx::mad_lo_cc(acc[0], P::mod(off), y, acc[0]);
  ptx::madc_hi_cc(acc[1], P::mod(off), y, acc[1]);
#pragma unroll
  for (int k = 1; k < N / 2; ++k) {
    ptx::madc_lo_cc(acc[2 * k], P::mod(2 * k + off), y, acc[2 * k]);
    ptx::madc_hi_cc(acc[2 * k + 1], P::mod(2 * k + off), y, acc[2 * k + 1]);
  }
  ptx::addc(acc[N], acc[N], 0u);
}

// r = a * b * R^-1 mod p, canonical in and out, N even: the even/odd schedule.
// The merge E <- O + E_1 adds E_1 into O's first word and the carry into the second, and
// the carry out of the second word stays pending as one bit q of weight 2^64 (the third word of the next
// row's frame), instead of running through all N+1 words.  A row's products and reduction do not touch
// that word's position before the next merge, where the shift has brought q down to the second word:
// that merge adds it there (addc with q as the addend), and the final combination adds the last q once.
// 3 carry-chain adds per row instead of N+1 for a full merge, no branch.  The adds run on the ALU pipe, but a
// full merge is a serial chain of N+1 dependent adds between one row's products and the next row's, and it
// cost the 24-limb product a quarter of its time (6.1 against 8.3 G products/s in isolation on GB300).
template <class P>
__device__ __forceinline__ void fe_mul_eo(Fe<P>& r, const Fe<P>& a, const Fe<P>& b) {
  constexpr int N = P::N;
  static_assert(N % 2 == 0 && N >= 4, "even/odd schedule needs an even limb count of at least 4");
  uint32_t E[N + 1], O[N + 1];
  uint32_t q = 0u;  // pending carry, weight 2^64 in the current frame
#pragma unroll
  for (int j = 0; j <= N; ++j) E[j] = O[j] = 0u;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint32_t bi = b.l[i];
    pair_chain<N>(E, a.l, 0, bi);
    pair_chain<N>(O, a.l, 1, bi);
    const uint32_t m = E[0] * row_pinv<P>();
    pair_chain_mod<P>(E, 0, m);
    pair_chain_mod<P>(O, 1, m);
    // E <- O + E_1 + 2^32 q (carry out of the second word pending), O <- E_2..E_N
    const uint32_t e1 = E[1];
    uint32_t Onew[N + 1];
#pragma unroll
    for (int j = 0; j <= N - 2; ++j) Onew[j] = E[j + 2];
    Onew[N - 1] = 0u;
    Onew[N] = 0u;
    ptx::add_cc(E[0], O[0], e1);
    ptx::addc_cc(E[1], O[1], q);
    ptx::addc(q, 0u, 0u);
#pragma unroll
    for (int j = 2; j <= N; ++j) E[j] = O[j];
#pragma unroll
    for (int j = 0; j <= N; ++j) O[j] = Onew[j];
  }
  // t = E + 2^32 O + 2^64 q  (< 2p), then one conditional subtraction
  uint32_t t[N + 1];
  t[0] = E[0];
  ptx::add_cc(t[1], E[1], O[0]);
#pragma unroll
  for (int j = 2; j < N; ++j) ptx::addc_cc(t[j], E[j], O[j - 1]);
  ptx::addc(t[N], E[N], O[N - 1]);
  ptx::add_cc(t[2], t[2], q);
#pragma unroll
  for (int j = 3; j < N; ++j) ptx::addc_cc(t[j], t[j], 0u);
  ptx::addc(t[N], t[N], 0u);
  uint32_t d[N], mask;
  ptx::sub_cc(d[0], t[0], P::mod(0));
#pragma unroll
  for (int j = 1; j < N; ++j) ptx::subc_cc(d[j], t[j], P::mod(j));
  ptx::subc(mask, t[N], 0u);
#pragma unroll
  for (int j = 0; j < N; ++j) r.l[j] = (t[j] & mask) | (d[j] & ~mask);
}

// Montgomery product used by the kernels.  GSN_MONT_SCHEDULE selects the
// multi-limb schedule: 1 = even/odd accumulators (default), 0 = row chains.
#ifndef GSN_MONT_SCHEDULE
#define GSN_MONT_SCHEDULE 1
#endif
template <class P, int S = GSN_MONT_SCHEDULE>
__device__ __forceinline__ void fe_mul(Fe<P>& r, const Fe<P>& a, const Fe<P>& b) {
  if constexpr (P::N == 1) {
    r.l[0] = mul1<P>(a.l[0], b.l[0]);
  } else if constexpr (S == 1 && P::N % 2 == 0) {
    fe_mul_eo<P>(r, a, b);
  } else {
    fe_mul_rows<P>(r, a, b);
  }
}

// Montgomery form helpers (device): x*R and x*R^-1.
template <class P>
__device__ __forceinline__ void fe_to_mont(Fe<P>& r, const Fe<P>& a) {
  Fe<P> r2;
#pragma unroll
  for (int j = 0; j < P::N; ++j) r2.l[j] = P::r2(j);
  fe_mul<P>(r, a, r2);
}

template <class P>
__device__ __forceinline__ void fe_set_one_mont(Fe<P>& r) {
#pragma unroll
  for (int j = 0; j < P::N; ++j) r.l[j] = P::r1(j);
}

// --- loads and stores (16-byte vectors when the element allows) -------------
template <class P>
__device__ __forceinline__ void fe_load(Fe<P>& r, const uint32_t* p) {
  constexpr int N = P::N;
  if constexpr (N % 4 == 0) {
    const uint4* q = reinterpret_cast<const uint4*>(p);
#pragma unroll
    for (int k = 0; k < N / 4; ++k) {
      uint4 v = q[k];
      r.l[4 * k + 0] = v.x;
      r.l[4 * k + 1] = v.y;
      r.l[4 * k + 2] = v.z;
      r.l[4 * k + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < N; ++k) r.l[k] = p[k];
  }
}

// Load that bypasses L1 (ld.global.cg): used for data another CTA of the same
// launch may have written (the batched kernel reads earlier passes' output),
// or a kernel that this one overlaps (chain.cuh).
template <class P>
__device__ __forceinline__ void fe_load_cg(Fe<P>& r, const uint32_t* p) {
  constexpr int N = P::N;
  if constexpr (N % 4 == 0) {
    const uint4* q = reinterpret_cast<const uint4*>(p);
#pragma unroll
    for (int k = 0; k < N / 4; ++k) {
      uint4 v = __ldcg(q + k);
      r.l[4 * k + 0] = v.x;
      r.l[4 * k + 1] = v.y;
      r.l[4 * k + 2] = v.z;
      r.l[4 * k + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < N; ++k) r.l[k] = __ldcg(p + k);
  }
}

template <class P>
__device__ __forceinline__ void fe_store(uint32_t* p, const Fe<P>& a) {
  constexpr int N = P::N;
  if constexpr (N % 4 == 0) {
    uint4* q = reinterpret_cast<uint4*>(p);
#pragma unroll
    for (int k = 0; k < N / 4; ++k) q[k] = make_uint4(a.l[4 * k], a.l[4 * k + 1], a.l[4 * k + 2], a.l[4 * k + 3]);
  } else {
#pragma unroll
    for (int k = 0; k < N; ++k) p[k] = a.l[k];
  }
}

// ---------------------------------------------------------------------------
// Product by a table constant w (Shoup's precomputed quotient; V. Shoup's NTL, and D. Harvey, "Faster arithmetic
// for number-theoretic transforms", 2014).  The table holds w and w' = floor(w R / p), R = 2^(32N).  With
// q ~ floor(x w' / R), r = x w - q p lies in [0, 2p), so only the high half of x w' and the low halves of x w and
// q p are needed: for MNT4-753 852 wide multiply-adds and 47 single-word ones, where a Montgomery product takes
// 1152 wide ones and 24 row factors (BLS12-381: 86 and 14, against 128 and 8).  The transform multiplies only by table
// constants.
//
// Bounds: floor(x w' / R) > x w / p - x / R - 1.  q leaves out the word products below word N-2, together less
// than (N-2) 2^(32(N-1)), which can lower it by one, in (N-2) 2^-32 of all cases.  So
// r < p (1 + x / R + (N-2) 2^-32) + (rounding) <= p (1 + (x / R) + 2^-27) for x < R.  With x < 2p (and 2p < R by a
// margin above 2^-27) that is below 2p and below R, so the arithmetic modulo R is exact and one conditional
// subtraction ends in [0, p).  A caller that keeps its values in [0, 2p) leaves that subtraction out (K = 2).  MNT4-753
// r is below 2^-15 R, so there x may be any value below 2^13 p.
//
// Measured on GB300 as chains of dependent products (G products/s, 128-thread blocks), Montgomery -> this form:
// MNT4-753 7.7 -> 10.5 (16 warps per SM, 124 registers; before its modulus's low limb went to shifts, which took 875
// wide multiply-adds to 852 and the multiply pipe's own limit from 11.2 to 11.5), BLS12-381 66.8 -> 90.3 (81.9 without
// the modulus's two low limbs taken apart below).
//
// The halves are summed by rows into two accumulators per half, one for products at even words and one for odd
// ones, so that every product lands on an aligned register pair (one wide multiply-add) and no accumulator moves.
// ---------------------------------------------------------------------------

// Table layout.  The one-limb field stores w R (its product is mul1), one word per entry.  The others store w and w'
// in blocks of 8 entries, each block chunk-major: 16-byte chunk c (limbs 4c.. of w, then of w') of entry e is at word
// (e / 8) 16N + 32 c + 4 (e mod 8).  Lanes that read neighbouring entries then share 128-byte lines, one line per
// chunk for 8 entries, where entry-major rows take a line per lane.
template <class P>
__device__ __forceinline__ size_t tw_offset(uint32_t e) {
  if constexpr (P::N == 1) {
    return e;
  } else {
    return (size_t)(e >> 3) * (16 * P::N) + ((e & 7u) << 2);
  }
}
constexpr int kTwChunk = 32;  // words from one chunk of an entry to the next

// Limb j of R - p: adding q (R - p) subtracts q p modulo R.  p is odd, so no carry leaves word 0.
template <class P>
__host__ __device__ constexpr uint32_t neg_mod(int j) {
  return j == 0 ? 0u - P::mod(0) : ~P::mod(j);
}

// (lo, hi) += a * b inside a carry chain that `first` opens.
__device__ __forceinline__ void wide_step(uint32_t& lo, uint32_t& hi, uint32_t a, uint32_t b, bool first) {
  if (first) {
    ptx::mad_lo_cc(lo, a, b, lo);
  } else {
    ptx::madc_lo_cc(lo, a, b, lo);
  }
  ptx::madc_hi_cc(hi, a, b, hi);
}

// E + 2^32 O += x * y * 2^(32 i) modulo 2^(32N), for limbs j >= jmin of x.  E[k] is word k, O[k] word k + 1.
template <int N, class X>
__device__ __forceinline__ void low_row(uint32_t (&E)[N], uint32_t (&O)[N], X x, int i, uint32_t y, int jmin = 0) {
  const int je = jmin + ((i + jmin) & 1), jo = jmin + ((i + jmin + 1) & 1);
#pragma unroll
  for (int j = je; i + j <= N - 2; j += 2) wide_step(E[i + j], E[i + j + 1], x(j), y, j == je);
#pragma unroll
  for (int j = jo; i + j <= N - 3; j += 2) wide_step(O[i + j - 1], O[i + j], x(j), y, j == jo);
  const int jt = N - 1 - i;  // word N-1: the low half alone
  if (jt == jo) {
    ptx::mad_lo(O[N - 2], x(jt), y, O[N - 2]);
  } else if (jt > jo) {
    ptx::madc_lo(O[N - 2], x(jt), y, O[N - 2]);
  }
}

// The words from N-2 up of x * y * 2^(32 i): E[k] is word N-2+k, O[k] word N-1+k.  The carry out of a row's chain
// goes into a word that only such carries (one per parity of i) have reached before.
template <int N, class X>
__device__ __forceinline__ void high_row(uint32_t (&E)[N + 2], uint32_t (&O)[N + 2], X x, int i, uint32_t y) {
  const int je = i <= N - 2 ? N - 2 - i : 1, jo = N - 1 - i;
  int k = 0;
#pragma unroll
  for (int j = je; j <= N - 1; j += 2) {
    k = i + j - (N - 2);
    wide_step(E[k], E[k + 1], x(j), y, j == je);
  }
  if (k + 2 <= N + 1) ptx::addc(E[k + 2], E[k + 2], 0u);
#pragma unroll
  for (int j = jo; j <= N - 1; j += 2) {
    k = i + j - (N - 1);
    wide_step(O[k], O[k + 1], x(j), y, j == jo);
  }
  if (k + 2 <= N) ptx::addc(O[k + 2], O[k + 2], 0u);
}

// f(i, limb i) over N limbs of a table entry, read as 16-byte chunks.
template <int N, class F>
__device__ __forceinline__ void each_limb(const uint32_t* p, F f) {
#pragma unroll
  for (int k = 0; k < N / 4; ++k) {
    const uint4 v = *reinterpret_cast<const uint4*>(p + k * kTwChunk);
    f(4 * k + 0, v.x);
    f(4 * k + 1, v.y);
    f(4 * k + 2, v.z);
    f(4 * k + 3, v.w);
  }
}

// r = t mod p for t < 2p.
template <class P>
__device__ __forceinline__ void fe_reduce_once(Fe<P>& r, const uint32_t (&t)[P::N]) {  // t may be r.l
  constexpr int N = P::N;
  uint32_t d[N], mask;
  ptx::sub_cc(d[0], t[0], P::mod(0));
#pragma unroll
  for (int j = 1; j < N; ++j) ptx::subc_cc(d[j], t[j], P::mod(j));
  ptx::subc(mask, 0u, 0u);  // 0xFFFFFFFF iff t < p
#pragma unroll
  for (int j = 0; j < N; ++j) r.l[j] = (t[j] & mask) | (d[j] & ~mask);
}

// r = x mod p for x < 2^(kMaxLazyLog + 1) p of a field with that room. The quotient from the top words alone,
// q = floor(x_top / (p_top + 1)) up to 2^-16, is the true one or one less: the two differ by less than
// 2^13 / p_top + 1 / p_top + 2^-16 < 0.08 before they are rounded down (p_top = 0x1c4c6).
template <class P>
__device__ __forceinline__ void fe_reduce_lazy(Fe<P>& r, const Fe<P>& x) {
  constexpr int N = P::N;
  static_assert(P::mod(N - 1) > (1u << 16) && P::mod(N - 1) < (1u << 18), "the quotient's error bound");
  constexpr uint64_t inv = (1ull << 48) / (P::mod(N - 1) + 1u);
  const uint32_t q = (uint32_t)((x.l[N - 1] * inv) >> 48);
  uint32_t E[N], O[N], t[N];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    E[j] = x.l[j];
    O[j] = 0u;
  }
  low_row<N>(E, O, [](int j) { return neg_mod<P>(j); }, 0, q);
  t[0] = E[0];
  ptx::add_cc(t[1], E[1], O[0]);
#pragma unroll
  for (int j = 2; j < N - 1; ++j) ptx::addc_cc(t[j], E[j], O[j - 1]);
  ptx::addc(t[N - 1], E[N - 1], O[N - 2]);
  fe_reduce_once<P>(r, t);
}

// r = x * w mod p, below K p (K = 1: canonical), for x < 2p and the table entry at `e` (table + tw_offset<P>(index)).
template <class P, int K = 1>
__device__ __forceinline__ void fe_mul_tw(Fe<P>& r, const Fe<P>& x, const uint32_t* e) {
  constexpr int N = P::N;
  if constexpr (N == 1) {
    r.l[0] = mul1<P>(x.l[0], e[0]);
  } else {
    static_assert(N % 4 == 0, "entries are read as 16-byte vectors");
    auto xl = [&](int j) { return x.l[j]; };
    uint32_t q[N];
    {
      uint32_t E[N + 2], O[N + 2], below;
#pragma unroll
      for (int j = 0; j < N + 2; ++j) E[j] = O[j] = 0u;
      each_limb<N>(e + N / 4 * kTwChunk, [&](int i, uint32_t y) { high_row<N>(E, O, xl, i, y); });
      ptx::add_cc(below, E[1], O[0]);
#pragma unroll
      for (int k = 0; k < N - 1; ++k) ptx::addc_cc(q[k], E[k + 2], O[k + 1]);
      ptx::addc(q[N - 1], E[N + 1], O[N]);
    }
    uint32_t E[N], O[N], t[N];
#pragma unroll
    for (int j = 0; j < N; ++j) E[j] = O[j] = 0u;
    each_limb<N>(e, [&](int i, uint32_t y) { low_row<N>(E, O, xl, i, y); });
    // BLS12-381 r has the low limbs 1 and 2^32 - 1, so R - p = (2^32 - 1) + 2^64 (...): its two low limbs'
    // share of q (R - p) is 2^32 q - q, two carry chains on the add pipe instead of 15 word products.
    constexpr bool low_by_adds = P::mod(0) == 1u && P::mod(1) == 0xFFFFFFFFu;
    // MNT4-753 r has the low limb 2^30 + 1: q p = q + 2^30 q + 2^32 q p', p' the limbs above, whose negative modulo R / 2^32
    // multiplies q from word 1 up.
    constexpr bool low_by_shift = P::mod(0) == 0x40000001u && P::mod(1) != 0u;
    auto pl = [&](int j) { return low_by_shift && j == 1 ? 0u - P::mod(1) : neg_mod<P>(j); };
#pragma unroll
    for (int i = 0; i < N; ++i) low_row<N>(E, O, pl, i, q[i], low_by_adds ? 2 : low_by_shift ? 1 : 0);
    t[0] = E[0];
    ptx::add_cc(t[1], E[1], O[0]);
#pragma unroll
    for (int j = 2; j < N - 1; ++j) ptx::addc_cc(t[j], E[j], O[j - 1]);
    ptx::addc(t[N - 1], E[N - 1], O[N - 2]);
    if constexpr (low_by_shift) {
      ptx::sub_cc(t[0], t[0], q[0]);
#pragma unroll
      for (int j = 1; j < N - 1; ++j) ptx::subc_cc(t[j], t[j], q[j]);
      ptx::subc(t[N - 1], t[N - 1], q[N - 1]);
      ptx::sub_cc(t[0], t[0], q[0] << 30);
#pragma unroll
      for (int j = 1; j < N - 1; ++j) ptx::subc_cc(t[j], t[j], __funnelshift_l(q[j - 1], q[j], 30));
      ptx::subc(t[N - 1], t[N - 1], __funnelshift_l(q[N - 2], q[N - 1], 30));
    }
    if constexpr (low_by_adds) {
      ptx::add_cc(t[1], t[1], q[0]);
#pragma unroll
      for (int j = 2; j < N - 1; ++j) ptx::addc_cc(t[j], t[j], q[j - 1]);
      ptx::addc(t[N - 1], t[N - 1], q[N - 2]);
      ptx::sub_cc(t[0], t[0], q[0]);
#pragma unroll
      for (int j = 1; j < N - 1; ++j) ptx::subc_cc(t[j], t[j], q[j]);
      ptx::subc(t[N - 1], t[N - 1], q[N - 1]);
    }
    if constexpr (K == 1) {
      fe_reduce_once<P>(r, t);
    } else {
#pragma unroll
      for (int j = 0; j < N; ++j) r.l[j] = t[j];
    }
  }
}

// Table entry of w from its Montgomery form m = w R mod p.  Reducing m by R, the row factors are the limbs of
// -m p^-1 mod R = (w R - m) / p = w', and what is left is m / R = w mod p (below p, since m < p).
template <class P>
__device__ __forceinline__ void fe_store_tw(uint32_t* e, const Fe<P>& m) {
  constexpr int N = P::N;
  if constexpr (N == 1) {
    e[0] = m.l[0];
  } else {
    Fe<P> w, f;
    uint32_t E[N + 1], O[N + 1];
    uint32_t q = 0u;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      E[j] = m.l[j];
      O[j] = 0u;
    }
    E[N] = O[N] = 0u;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      f.l[i] = E[0] * row_pinv<P>();
      pair_chain_mod<P>(E, 0, f.l[i]);
      pair_chain_mod<P>(O, 1, f.l[i]);
      const uint32_t e1 = E[1];  // the merge of fe_mul_eo
      uint32_t Onew[N + 1];
#pragma unroll
      for (int j = 0; j <= N - 2; ++j) Onew[j] = E[j + 2];
      Onew[N - 1] = 0u;
      Onew[N] = 0u;
      ptx::add_cc(E[0], O[0], e1);
      ptx::addc_cc(E[1], O[1], q);
      ptx::addc(q, 0u, 0u);
#pragma unroll
      for (int j = 2; j <= N; ++j) E[j] = O[j];
#pragma unroll
      for (int j = 0; j <= N; ++j) O[j] = Onew[j];
    }
    w.l[0] = E[0];
    ptx::add_cc(w.l[1], E[1], O[0]);
#pragma unroll
    for (int j = 2; j < N - 1; ++j) ptx::addc_cc(w.l[j], E[j], O[j - 1]);
    ptx::addc(w.l[N - 1], E[N - 1], O[N - 2]);
    ptx::add_cc(w.l[2], w.l[2], q);
#pragma unroll
    for (int j = 3; j < N - 1; ++j) ptx::addc_cc(w.l[j], w.l[j], 0u);
    ptx::addc(w.l[N - 1], w.l[N - 1], 0u);
#pragma unroll
    for (int k = 0; k < N / 4; ++k) {
      *reinterpret_cast<uint4*>(e + k * kTwChunk) =
          make_uint4(w.l[4 * k], w.l[4 * k + 1], w.l[4 * k + 2], w.l[4 * k + 3]);
      *reinterpret_cast<uint4*>(e + (N / 4 + k) * kTwChunk) =
          make_uint4(f.l[4 * k], f.l[4 * k + 1], f.l[4 * k + 2], f.l[4 * k + 3]);
    }
  }
}

// r = x / 2^k mod p, 0 < k < 32: with f = -x p^-1 mod 2^k, x + f p is a multiple of 2^k and below 2^k p for x < p
// (and below (2^k + 1) p for x < 2p, so r < 2p).
// N + 1 multiply-adds, where a product by the inverse of 2^k takes a whole field product.
template <class P>
__device__ __forceinline__ void fe_div_pow2(Fe<P>& r, const Fe<P>& x, int k) {
  constexpr int N = P::N;
  const uint32_t f = (x.l[0] * row_pinv<P>()) & ((1u << k) - 1u);
  if constexpr (N == 1) {
    r.l[0] = (uint32_t)((x.l[0] + (uint64_t)f * P::mod(0)) >> k);
  } else {
    uint32_t E[N + 1], O[N + 1];
#pragma unroll
    for (int j = 0; j < N; ++j) {
      E[j] = x.l[j];
      O[j] = 0u;
    }
    E[N] = O[N] = 0u;
    pair_chain_mod<P>(E, 0, f);
    pair_chain_mod<P>(O, 1, f);
    ptx::add_cc(E[1], E[1], O[0]);
#pragma unroll
    for (int j = 2; j < N; ++j) ptx::addc_cc(E[j], E[j], O[j - 1]);
    ptx::addc(E[N], E[N], O[N - 1]);
#pragma unroll
    for (int j = 0; j < N; ++j) r.l[j] = __funnelshift_r(E[j], E[j + 1], k);
  }
}

}  // namespace gsn
