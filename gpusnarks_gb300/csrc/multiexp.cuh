// Multi-exponentiation over field elements: out = sum_i a[i] * b[i] mod p.
//
// Replaces the reference's multiexp<FieldT, FieldMul> (cuda/multi_exp.cu:86-137): there every thread
// multiplies with the full Scalar product and adds modularly (deviceReduceKernel :86-101), reduces its
// block through warp shuffles and shared memory (blockReduceSum :54-68), and a one-block second launch
// sums the per-block results (deviceReduceKernelSecond :70-84).  Here the two-launch shape stays, but
// the per-element work is half a Montgomery product:
//   * each thread adds the plain 2N-word products a[i]*b[i] into a (2N+1)-word integer accumulator, so
//     the per-element cost is the N^2 word products of a*b (PTX mad.lo.cc/madc.hi.cc pair chains, the
//     even/odd split of arith.cuh, so each pair can issue as one wide multiply-add) and one add chain;
//     there is no reduction and no modular add in the loop. With 24 limbs the multiply pipe bounds it, and
//     one Karatsuba step takes 432 of the 576 (1,000,003 elements on GB300: 78.7 -> 67.0 us);
//   * the threads' accumulators are added as integers, word column by word column in 64 bits: through shared memory in a
//     block, then by the second launch over the blocks. No thread reduces or normalises anything;
//   * one warp of the second launch reduces the total T < 2^40 p^2 by N+2 Montgomery word steps, a lane per column, to
//     T * 2^(-32(N+2)) in [0, 2p), and one Montgomery product by a host constant, again a lane per column, turns that into
//     the requested representation:
//       canonical   (inputs x, y as integers):           T mod p,        fix = 2^(32(2N+2)) mod p
//       Montgomery  (inputs xR, yR, output (sum x y) R):  T R^-1 mod p,   fix = 2^(32(N+2)) mod p.
// Before, every thread reduced its own accumulator and multiplied it by the constant, and the canonical results went
// through modular shuffle trees: about 10 us of a 24-limb call whatever its length.
// The 32-bit field accumulates 64-bit products (mul.wide) into a 96-bit sum with 16-byte loads.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>

#include "arith.cuh"
#include "chain.cuh"
#include "ntt_common.h"

namespace gsn {
namespace mexp {

// The plain product a * b (N even) into two accumulators whose 64-bit pairs always start at an even word,
// so every mad.lo.cc / madc.hi.cc pair on the same operands is register-pair aligned and can issue as one
// wide multiply-add:  a * b = A + 2^32 B,  A taking the word products a_j b_i with i + j even (pairs at
// words (i+j, i+j+1)) and B those with i + j odd (pair at A-words (i+j, i+j+1) stored at B[i+j-1], B[i+j]).
// Row i adds one chain into each.  A chain that ends at pair word w carries into word w + 1, which before
// that row holds at most the 1-bit carry of the row before (the chains of each accumulator end one word
// apart on alternate rows), so no carry is lost: A needs 2N+1 words, B 2N-1.
template <int N, int I, bool INTO_A>
__device__ __forceinline__ void pair_row(uint32_t* acc, const uint32_t* a, uint32_t bi) {
  // j runs over one parity: (I + j) even for A, odd for B; words of acc are (I + j - off, I + j + 1 - off)
  constexpr int j0 = INTO_A ? (I & 1) : ((I + 1) & 1);
  constexpr int off = INTO_A ? 0 : 1;
  constexpr int jlast = ((N - 1 - j0) / 2) * 2 + j0;
  ptx::mad_lo_cc(acc[I + j0 - off], a[j0], bi, acc[I + j0 - off]);
  ptx::madc_hi_cc(acc[I + j0 + 1 - off], a[j0], bi, acc[I + j0 + 1 - off]);
#pragma unroll
  for (int j = j0 + 2; j <= jlast; j += 2) {
    ptx::madc_lo_cc(acc[I + j - off], a[j], bi, acc[I + j - off]);
    ptx::madc_hi_cc(acc[I + j + 1 - off], a[j], bi, acc[I + j + 1 - off]);
  }
  ptx::addc(acc[I + jlast + 2 - off], acc[I + jlast + 2 - off], 0u);
}

template <int N, int I>
__device__ __forceinline__ void rows(uint32_t (&A)[2 * N + 1], uint32_t (&B)[2 * N - 1], const uint32_t* a,
                                     const uint32_t* b) {
  if constexpr (I < N) {
    pair_row<N, I, true>(A, a, b[I]);
    pair_row<N, I, false>(B, a, b[I]);
    rows<N, I + 1>(A, B, a, b);
  }
}

// T[0..2N] += a * b (plain product, no reduction).
template <int N>
__device__ __forceinline__ void mul_acc(uint32_t (&T)[2 * N + 1], const uint32_t* a, const uint32_t* b) {
  static_assert(N % 2 == 0, "the pair-aligned product needs an even limb count");
  uint32_t A[2 * N + 1], B[2 * N - 1];
#pragma unroll
  for (int k = 0; k < 2 * N + 1; ++k) A[k] = 0u;
#pragma unroll
  for (int k = 0; k < 2 * N - 1; ++k) B[k] = 0u;
  rows<N, 0>(A, B, a, b);
  // T += A, then T += 2^32 B (the product is below 2^(64N), so A's top word and the final carries fit)
  ptx::add_cc(T[0], T[0], A[0]);
#pragma unroll
  for (int k = 1; k < 2 * N + 1; ++k) ptx::addc_cc(T[k], T[k], A[k]);
  ptx::add_cc(T[1], T[1], B[0]);
#pragma unroll
  for (int k = 2; k < 2 * N; ++k) ptx::addc_cc(T[k], T[k], B[k - 1]);
  ptx::addc(T[2 * N], T[2 * N], 0u);
}

// The accumulator of one thread: T += a * b, and T's words at the end.
template <int N>
struct Accumulator {
  uint32_t T[2 * N + 1];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int k = 0; k <= 2 * N; ++k) T[k] = 0u;
  }
  __device__ __forceinline__ void add(const uint32_t* a, const uint32_t* b) { mul_acc<N>(T, a, b); }
  __device__ __forceinline__ void words(uint32_t (&out)[2 * N + 1]) const {
#pragma unroll
    for (int k = 0; k <= 2 * N; ++k) out[k] = T[k];
  }
};

// 24 limbs: one Karatsuba step, kept apart over the whole sum. With halves a = a0 + a1 B, B = 2^384, the thread adds up
// a0 b0, a1 b1 and (a0 + a1)(b0 + b1), 432 word products an element for 576, and takes the middle part out once at the end.
// The sums of halves have a carry bit each, whose products are masked additions on the add pipe.
template <>
struct Accumulator<24> {
  static constexpr int H = 12;
  uint32_t L[2 * H + 1], U[2 * H + 1], M[2 * H + 2];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int k = 0; k <= 2 * H; ++k) L[k] = U[k] = M[k] = 0u;
    M[2 * H + 1] = 0u;
  }
  __device__ __forceinline__ void add(const uint32_t* a, const uint32_t* b) {
    uint32_t s[H], t[H], cs, ct;
    ptx::add_cc(s[0], a[0], a[H]);
#pragma unroll
    for (int k = 1; k < H; ++k) ptx::addc_cc(s[k], a[k], a[H + k]);
    ptx::addc(cs, 0u, 0u);
    ptx::add_cc(t[0], b[0], b[H]);
#pragma unroll
    for (int k = 1; k < H; ++k) ptx::addc_cc(t[k], b[k], b[H + k]);
    ptx::addc(ct, 0u, 0u);
    uint32_t low[2 * H + 1];
#pragma unroll
    for (int k = 0; k <= 2 * H; ++k) low[k] = M[k];
    mul_acc<H>(low, s, t);  // the sum of fewer than 2^32 such products fits with M's last word
    const bool wrapped = low[2 * H] < M[2 * H];
#pragma unroll
    for (int k = 0; k <= 2 * H; ++k) M[k] = low[k];
    M[2 * H + 1] += wrapped ? 1u : 0u;
    // + 2^384 (cs t + ct s) + 2^768 cs ct
    const uint32_t ms = 0u - cs, mt = 0u - ct;
    ptx::add_cc(M[H], M[H], t[0] & ms);
#pragma unroll
    for (int k = 1; k < H; ++k) ptx::addc_cc(M[H + k], M[H + k], t[k] & ms);
    ptx::addc_cc(M[2 * H], M[2 * H], cs & ct);
    ptx::addc(M[2 * H + 1], M[2 * H + 1], 0u);
    ptx::add_cc(M[H], M[H], s[0] & mt);
#pragma unroll
    for (int k = 1; k < H; ++k) ptx::addc_cc(M[H + k], M[H + k], s[k] & mt);
    ptx::addc_cc(M[2 * H], M[2 * H], 0u);
    ptx::addc(M[2 * H + 1], M[2 * H + 1], 0u);
    mul_acc<H>(L, a, b);
    mul_acc<H>(U, a + H, b + H);
  }
  __device__ __forceinline__ void words(uint32_t (&out)[4 * H + 1]) const {
    uint32_t m[2 * H + 2];  // the middle part, M - L - U >= 0
    ptx::sub_cc(m[0], M[0], L[0]);
#pragma unroll
    for (int k = 1; k <= 2 * H; ++k) ptx::subc_cc(m[k], M[k], L[k]);
    ptx::subc(m[2 * H + 1], M[2 * H + 1], 0u);
    ptx::sub_cc(m[0], m[0], U[0]);
#pragma unroll
    for (int k = 1; k <= 2 * H; ++k) ptx::subc_cc(m[k], m[k], U[k]);
    ptx::subc(m[2 * H + 1], m[2 * H + 1], 0u);
    // L + 2^768 U overlap in word 2H
#pragma unroll
    for (int k = 0; k < 2 * H; ++k) out[k] = L[k];
    ptx::add_cc(out[2 * H], L[2 * H], U[0]);
#pragma unroll
    for (int k = 1; k < 2 * H; ++k) ptx::addc_cc(out[2 * H + k], U[k], 0u);
    ptx::addc(out[4 * H], U[2 * H], 0u);
    ptx::add_cc(out[H], out[H], m[0]);
#pragma unroll
    for (int k = 1; k < 2 * H + 2; ++k) ptx::addc_cc(out[H + k], out[H + k], m[k]);
#pragma unroll
    for (int k = 3 * H + 2; k < 4 * H; ++k) ptx::addc_cc(out[k], out[k], 0u);
    ptx::addc(out[4 * H], out[4 * H], 0u);
  }
};

// Threads per block: 256 up to 8 limbs, 128 for 24 (register-bound).
template <class P>
__host__ __device__ constexpr int multiexp_block() {
  return P::N > 8 ? 128 : 256;
}

// Word columns of an accumulator.
template <class P>
__host__ __device__ constexpr int columns() {
  return 2 * P::N + 1;
}

// Sums over `count` rows of W columns, load(r * W + k) the word of row r and column k: thread k < W of the block gets column
// k's.  `part` holds blockDim.x values.  W is odd, so rows in shared memory conflict neither in their stores nor here.
template <int W, class Load>
__device__ __forceinline__ uint64_t column_sum(Load load, int count, uint64_t* part) {
  const int segs = blockDim.x / W, k = threadIdx.x % W, seg = threadIdx.x / W;
  uint64_t sum = 0;
  if (seg < segs) {
#pragma unroll 8
    for (int r = seg; r < count; r += segs) sum += load((size_t)r * W + k);
    part[threadIdx.x] = sum;
  }
  __syncthreads();
  sum = 0;
  if (threadIdx.x < W) {
#pragma unroll 4
    for (int g = 0; g < segs; ++g) sum += part[g * W + threadIdx.x];
  }
  return sum;
}

// The same for the few columns of the one-limb field, each thread's in registers: shuffles, then over the warps.
template <int W>
__device__ __forceinline__ uint64_t thread_columns_sum(uint64_t (&v)[W], uint64_t* part) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int k = 0; k < W; ++k) v[k] += __shfl_down_sync(0xFFFFFFFFu, v[k], off);
  }
  if ((threadIdx.x & 31u) == 0) {
#pragma unroll
    for (int k = 0; k < W; ++k) part[(threadIdx.x >> 5) * W + k] = v[k];
  }
  __syncthreads();
  uint64_t sum = 0;
  if (threadIdx.x < W) {
#pragma unroll 8
    for (unsigned g = 0; g < blockDim.x / 32; ++g) sum += part[g * W + threadIdx.x];
  }
  return sum;
}

// One warp, a lane per 32-bit column (columns may hold more than 32 bits): acc = (acc + m p) / 2^32 with the m that makes
// it whole, plus `lo` in each column and `hi` one column up.  `in` enters at lane 31.
__device__ __forceinline__ uint64_t lane_step(uint64_t acc, uint32_t p_lane, uint32_t pinv, uint64_t hi, uint64_t in) {
  const int lane = threadIdx.x & 31;
  const uint32_t m = __shfl_sync(0xFFFFFFFFu, (uint32_t)acc * pinv, 0);
  const uint64_t prod = (uint64_t)m * p_lane;
  acc += (uint32_t)prod;
  const uint64_t up = __shfl_down_sync(0xFFFFFFFFu, acc, 1);
  return (lane == 31 ? in : up) + (prod >> 32) + hi + (lane == 0 ? acc >> 32 : 0u);
}

// The lanes' columns, a value below 2p, as a canonical element in every lane.  `cols` holds 32 values.
template <class P>
__device__ __forceinline__ void lane_gather(Fe<P>& x, uint64_t acc, uint64_t* cols) {
  constexpr int N = P::N;
  __syncwarp();
  cols[threadIdx.x & 31] = acc;
  __syncwarp();
  uint32_t t[N], d[N], mask;
  uint64_t c = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    c += cols[j];
    t[j] = (uint32_t)c;
    c >>= 32;
  }
  const uint32_t top = (uint32_t)(c + cols[N]);
  ptx::sub_cc(d[0], t[0], P::mod(0));
#pragma unroll
  for (int j = 1; j < N; ++j) ptx::subc_cc(d[j], t[j], P::mod(j));
  ptx::subc(mask, top, 0u);  // 0xFFFFFFFF iff the value is below p
#pragma unroll
  for (int j = 0; j < N; ++j) x.l[j] = (t[j] & mask) | (d[j] & ~mask);
}

// First launch: per-block sums of a[i] * b[i] (grid-stride over i) as columns()<P> columns each, in `partial`.
// PF: load the next element's operands before the current product (more registers, overlapped latency).
template <class P, bool PF>
__global__ void __launch_bounds__(256) multiexp_kernel(const uint32_t* a, const uint32_t* b, uint64_t n,
                                                       uint64_t* partial) {
  constexpr int N = P::N, W = columns<P>();
  __shared__ uint32_t sums[N > 1 ? multiexp_block<P>() * W : 1];
  __shared__ uint64_t part[multiexp_block<P>()];
  chain_wait();
  uint32_t T[2 * N + 1];
#pragma unroll
  for (int k = 0; k <= 2 * N; ++k) T[k] = 0u;
  Accumulator<N> sum_ab;
  sum_ab.clear();
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if constexpr (N == 1) {
    // four elements per step with 16-byte loads when both arrays allow it, then the tail one by one
    const bool vec = ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0;
    uint64_t done = 0;
    if (vec) {
      const uint64_t quads = n >> 2;
      const uint4* a4 = reinterpret_cast<const uint4*>(a);
      const uint4* b4 = reinterpret_cast<const uint4*>(b);
      for (uint64_t q = i; q < quads; q += stride) {
        const uint4 x = __ldcs(a4 + q), y = __ldcs(b4 + q);
        const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          uint32_t lo, hi;
          lo = xs[e] * ys[e];
          hi = ptx::mul_hi(xs[e], ys[e]);
          ptx::add_cc(T[0], T[0], lo);
          ptx::addc_cc(T[1], T[1], hi);
          ptx::addc(T[2], T[2], 0u);
        }
      }
      done = quads << 2;
    }
    for (uint64_t k = done + i; k < n; k += stride) {
      const uint32_t x = __ldcs(a + k), y = __ldcs(b + k);
      ptx::add_cc(T[0], T[0], x * y);
      ptx::addc_cc(T[1], T[1], ptx::mul_hi(x, y));
      ptx::addc(T[2], T[2], 0u);
    }
  } else if constexpr (!PF) {
    for (; i < n; i += stride) {
      Fe<P> x, y;
      fe_load_cg<P>(x, a + i * N);
      fe_load_cg<P>(y, b + i * N);
      sum_ab.add(x.l, y.l);
    }
  } else {
    // the next element's operands are loaded before the current product, so their memory latency overlaps it
    Fe<P> x, y;
    if (i < n) {
      fe_load_cg<P>(x, a + i * N);
      fe_load_cg<P>(y, b + i * N);
    }
    for (; i < n; i += stride) {
      const uint64_t next = i + stride;
      Fe<P> xn, yn;
      if (next < n) {
        fe_load_cg<P>(xn, a + next * N);
        fe_load_cg<P>(yn, b + next * N);
      }
      sum_ab.add(x.l, y.l);
      x = xn;
      y = yn;
    }
  }
  chain_next();
  if constexpr (N > 1) sum_ab.words(T);
  uint64_t sum;
  if constexpr (N == 1) {
    uint64_t v[W];
#pragma unroll
    for (int k = 0; k < W; ++k) v[k] = T[k];
    sum = thread_columns_sum<W>(v, part);
  } else {
#pragma unroll
    for (int k = 0; k < W; ++k) sums[threadIdx.x * W + k] = T[k];
    __syncthreads();
    sum = column_sum<W>([&](size_t at) { return sums[at]; }, (int)blockDim.x, part);
  }
  if (threadIdx.x < W) partial[(uint64_t)blockIdx.x * W + threadIdx.x] = sum;
}

// Second launch (one block): the columns of all blocks, then the reduction of their sum in one warp.
constexpr int kFinalBlock = 1024;
template <class P>
__global__ void __launch_bounds__(kFinalBlock) multiexp_final_kernel(const uint64_t* partial, int count, uint32_t* out,
                                                                     Fe<P> fix) {
  constexpr int N = P::N, W = columns<P>(), ROWS = N + 2;
  __shared__ uint64_t part[kFinalBlock], cols[ROWS + 32 > W ? ROWS + 32 : W], gather[32];
  if (threadIdx.x >= W && threadIdx.x < ROWS + 32) cols[threadIdx.x] = 0u;
  chain_wait();
  uint64_t sum;
  if constexpr (N == 1) {
    uint64_t v[W] = {0u, 0u, 0u};
    for (int r = threadIdx.x; r < count; r += kFinalBlock) {
#pragma unroll
      for (int k = 0; k < W; ++k) v[k] += __ldcg(partial + (size_t)r * W + k);
    }
    sum = thread_columns_sum<W>(v, part);
  } else {
    sum = column_sum<W>([&](size_t at) { return __ldcg(partial + at); }, count, part);
  }
  if (threadIdx.x < W) cols[threadIdx.x] = sum;
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  uint32_t p_lane = 0u, fix_lane = 0u;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    if (lane == j) {
      p_lane = P::mod(j);
      fix_lane = fix.l[j];
    }
  }
  uint64_t acc = cols[lane];
#pragma unroll 1
  for (int r = 0; r < ROWS; ++r) acc = lane_step(acc, p_lane, P::PINV, 0u, cols[r + 32]);
  Fe<P> x;
  lane_gather<P>(x, acc, gather);
  acc = 0u;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint64_t prod = (uint64_t)x.l[i] * fix_lane;
    acc = lane_step(acc + (uint32_t)prod, p_lane, P::PINV, prod >> 32, 0u);
  }
  lane_gather<P>(x, acc, gather);
  if (lane == 0) fe_store<P>(out, x);
}

}  // namespace mexp
}  // namespace gsn

namespace gsn {

// Host launchers, instantiated per field.
template <class P>
struct MultiexpKernels {
  // CTAs of the first launch for n elements: enough to fill every SM, at most one thread per element.
  // Prefetching variant: on for the multi-limb fields (the 24-limb loop gained 23% from it on GB300);
  // GSN_MEXP_PREFETCH=0/1 overrides.
  static bool prefetch() {
    static const int v = [] {
      const char* e = getenv("GSN_MEXP_PREFETCH");
      return e ? atoi(e) : -1;
    }();
    return v < 0 ? P::N > 1 : v != 0;
  }
  static int grid(uint64_t n) {
    auto k = prefetch() ? mexp::multiexp_kernel<P, true> : mexp::multiexp_kernel<P, false>;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, mexp::multiexp_block<P>(), 0) != cudaSuccess) {
      cudaGetLastError();
      per_sm = 1;
    }
    const uint64_t full = (uint64_t)current_device_sms() * (uint64_t)(per_sm > 0 ? per_sm : 1);
    const uint64_t need = (n + mexp::multiexp_block<P>() - 1) / mexp::multiexp_block<P>();
    return (int)(need < 1 ? 1 : (need < full ? need : full));
  }
  static size_t partial_bytes(int grid) { return (size_t)grid * mexp::columns<P>() * sizeof(uint64_t); }
  static cudaError_t run(const uint32_t* a, const uint32_t* b, uint64_t n, void* partial, int grid, uint32_t* out,
                         const uint32_t* fix_limbs, cudaStream_t s) {
    Fe<P> fix;
    for (int j = 0; j < P::N; ++j) fix.l[j] = fix_limbs[j];
    uint64_t* const sums = static_cast<uint64_t*>(partial);
    auto k = prefetch() ? mexp::multiexp_kernel<P, true> : mexp::multiexp_kernel<P, false>;
    cudaError_t e = launch_chained(k, (unsigned)grid, mexp::multiexp_block<P>(), 0, s, a, b, n, sums);
    if (e != cudaSuccess) return e;
    return launch_chained(mexp::multiexp_final_kernel<P>, 1, mexp::kFinalBlock, 0, s, sums, grid, out, fix);
  }
};

}  // namespace gsn
