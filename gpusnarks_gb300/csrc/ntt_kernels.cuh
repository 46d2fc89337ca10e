// NTT kernels, templated on the field.  Included by one .cu per field so the
// fields compile in parallel.
//
// Replaces cuda_fft (cuda/fft_kernel.cu:52-115).  The reference launches 1280
// threads that each run a 1024-term direct sum and a 64-point radix-2 loop in
// local memory (O(n * 1024) products); here each pass is a radix-2^r
// sub-transform of a shared-memory tile (see ntt_common.h for the
// decomposition), so a transform costs (n/2) log2 n products plus one
// twiddle product per element per pass boundary.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "arith.cuh"
#include "chain.cuh"
#include "ntt_common.h"

namespace gsn {

// Dynamic shared memory above this is requested explicitly with
// cudaFuncAttributeMaxDynamicSharedMemorySize.  It is below the 48 KB default
// so that kernels with a little static shared memory (the batch kernel keeps
// its ticket and pass arguments there) never exceed the default limit.
constexpr size_t kDefaultSmemOptIn = 32 * 1024;

__device__ __forceinline__ uint32_t bitrev_bits(uint32_t x, int bits) {
  return bits == 0 ? 0u : (__brev(x) >> (32 - bits));
}

// Indices are 32-bit: every transform has at most 2^28 elements (the fields' size limits), and so does every table.

// e, or -e modulo the table's 2^log entries for the one-limb field's inverse transforms.
template <class P>
__device__ __forceinline__ uint32_t tw_sign(uint32_t e, int log, int inverse) {
  return P::N == 1 && inverse ? (0u - e) & ((1u << log) - 1u) : e;
}

// Stage twiddle w_R^e of a pass, e < R/2.
template <class P>
__device__ __forceinline__ const uint32_t* stage_entry(const PassArgs& A, uint32_t e) {
  return A.stage_tw + tw_offset<P>(tw_sign<P>(e << A.stage_shift, A.tw_log, A.inverse));
}

// Four-step factor w^(outer j k) of output k in column j.
template <class P>
__device__ __forceinline__ const uint32_t* step_entry(const PassArgs& A, uint32_t j, uint32_t k) {
  if (P::N > 1 && A.step_tw) return A.step_tw + tw_offset<P>((k << A.log_inner) + j);
  const uint32_t e = (j * k) << (A.log_outer + A.tw_log - A.log_n);  // < 2^tw_log
  return A.tw + tw_offset<P>(tw_sign<P>(e, A.tw_log, A.inverse));
}

// Position of output k of the last pass: -k mod n for the multi-limb fields' inverse transforms.
template <class P>
__device__ __forceinline__ uint32_t out_pos(const PassArgs& A, uint32_t k) {
  return P::N > 1 && A.inverse ? (0u - k) & ((1u << A.log_n) - 1u) : k;
}

// Multi-limb tile elements in shared memory: blocks of 8 slots, each block chunk-major (16-byte chunk c of slot s at
// word (s / 8) 8N + 32 c + 4 (s mod 8)), so that a quarter warp's 16-byte accesses to 8 slots of different s mod 8 take
// one pass over the banks; with element-major rows of 32 or 96 bytes every access was a two-way conflict.  Element
// (row, jj) has slot (row 2^lj + jj) ^ tile_hash(row): with fewer than 8 columns the bits of s mod 8 above the column
// also take in the higher row bits, because a quarter warp's rows are 2^m apart in the late stages and the bit-reversed
// reads.  tile_hash is linear over xor, and 0 for row 1.
template <int LJ>
__device__ __forceinline__ uint32_t tile_hash(uint32_t row, int lj) {
  const int l = LJ >= 0 ? LJ : lj;
  if (l >= 3) return 0u;
  if (l == 2) return (uint32_t)(__popc(row >> 1) & 1) << 2;
  if (l == 1) {
    row >>= 2;
    row ^= row >> 4;
    row ^= row >> 2;
    return ((row ^ (row >> 8)) & 3u) << 1;
  }
  row >>= 3;
  row ^= row >> 6;
  return (row ^ (row >> 3)) & 7u;
}
template <int LJ>
__device__ __forceinline__ uint32_t tile_slot(uint32_t row, uint32_t jj, int lj) {
  return ((row << (LJ >= 0 ? LJ : lj)) + jj) ^ tile_hash<LJ>(row, lj);
}
template <class P>
__device__ __forceinline__ uint32_t* tile_at(uint32_t* sm, uint32_t slot) {
  return sm + (slot >> 3) * (8 * P::N) + ((slot & 7u) << 2);
}
template <class P>
__device__ __forceinline__ void tile_load(Fe<P>& x, const uint32_t* p) {
#pragma unroll
  for (int c = 0; c < P::N / 4; ++c) {
    const uint4 v = *reinterpret_cast<const uint4*>(p + 32 * c);
    x.l[4 * c + 0] = v.x;
    x.l[4 * c + 1] = v.y;
    x.l[4 * c + 2] = v.z;
    x.l[4 * c + 3] = v.w;
  }
}
template <class P>
__device__ __forceinline__ void tile_store(uint32_t* p, const Fe<P>& x) {
#pragma unroll
  for (int c = 0; c < P::N / 4; ++c)
    *reinterpret_cast<uint4*>(p + 32 * c) = make_uint4(x.l[4 * c], x.l[4 * c + 1], x.l[4 * c + 2], x.l[4 * c + 3]);
}

// Mixed-radix digit reversal of the last pass's "rest" prefix index
// (digits k_1..k_{P-2}, row-major) into the output offset
// k_1 + n_1 k_2 + ... (before the final multiplication by n_0).
__device__ __forceinline__ uint64_t rest_offset(uint64_t rest, int npass, const int* radix_log) {
  uint64_t off = 0;
  int shift_before[kMaxPasses];
  int acc = 0;
  for (int i = 1; i < npass - 1; ++i) {
    shift_before[i] = acc;
    acc += radix_log[i];
  }
  for (int i = npass - 2; i >= 1; --i) {
    const uint64_t digit = rest & (((uint64_t)1 << radix_log[i]) - 1);
    rest >>= radix_log[i];
    off += digit << shift_before[i];
  }
  return off;
}

// Where a tile's elements come from and go to.
struct TileGeom {
  uint32_t base = 0;    // non-last: first element of the tile
  uint32_t jbase = 0;   // non-last: first suffix index j'
  uint32_t rowpre = 0;  // last: prefix_lin of row 0 = (k0_first << (outer_log - lo0)) + rest
  uint32_t obase = 0;   // last: output offset of row 0 (k_0 = k0_first, k = 0)
  int row_shift = 0;    // last: log2 of the distance between two rows' prefixes

  __device__ __forceinline__ TileGeom(const PassArgs& A, uint32_t tile) {
    if (!A.last) {
      const int per_prefix_log = A.log_inner - A.log_j;
      const uint32_t prefix = tile >> per_prefix_log;
      jbase = (tile & ((1u << per_prefix_log) - 1u)) << A.log_j;
      base = (prefix << (A.log_r + A.log_inner)) + jbase;
    } else {
      const int lo0 = (A.npass == 1) ? 0 : A.radix_log[0];
      const int k0b_log = lo0 - A.log_j;
      const uint32_t rest = tile >> k0b_log;
      const uint32_t k0 = (tile & ((1u << k0b_log) - 1u)) << A.log_j;
      row_shift = A.log_outer - lo0;
      rowpre = (k0 << row_shift) + rest;
      obase = k0 + ((uint32_t)rest_offset(rest, A.npass, A.radix_log) << lo0);
    }
  }
  // position of tile element (k, jj) in the source array
  __device__ __forceinline__ uint32_t src(const PassArgs& A, uint32_t k, uint32_t jj) const {
    return !A.last ? base + (k << A.log_inner) + jj : ((rowpre + (jj << row_shift)) << A.log_r) + k;
  }
  // position of output k of column (last pass: row) jj in the destination array
  template <class P>
  __device__ __forceinline__ uint32_t dst(const PassArgs& A, uint32_t k, uint32_t jj) const {
    return !A.last ? base + (k << A.log_inner) + jj : out_pos<P>(A, obase + jj + (k << A.log_outer));
  }
};

// CHAIN: the block's last stores are those of this tile, so the next kernel on the stream may be set up before them.  A
// pass's block has one tile up to 2^20 of them.  Blocks of the batched kernel take tiles until none are left and let the
// next kernel start as they end.

// One tile of one pass, one-limb field.  `sm` holds 2^(log_r + log_j) words.  Small transforms and batches of them come
// here (ntt_p32.cuh has the large ones), so latency and instructions count: a load phase (times the powers of the shift on
// the first pass of a coset transform), radix-4 sub-steps of 4 rows a thread (one radix-2 stage first for odd log_r), and
// a last phase with the four-step factor (non-last) or the division by n and the post table (last) and the store.  With a
// butterfly per thread and stage a warp took 977 instructions for a radix-2^8 tile and twice the barriers and exchanges.
// Products by 1 are computed (the table's entry 0) rather than branched around.
//
// Element (row, jj) is word word_slot((row << lj) + jj): the low 5 bits take in the higher ones so that a sub-step's rows
// at any distance and (mostly) the bit-reversed reads fall on 32 banks.  The map is linear over xor, so the rows of a
// sub-step differ by constants.
__device__ __forceinline__ uint32_t word_slot(uint32_t i) {
  const uint32_t u = i >> 5;
  return i ^ ((u ^ (u << 2) ^ (u << 3) ^ (u >> 5)) & 31u);
}

template <class P, bool CHAIN>
__device__ void word_tile(const PassArgs& A, unsigned array, uint32_t tile, uint32_t* sm) {
  static_assert(P::N == 1, "one limb");
  const int lr = A.log_r, lj = A.log_j;
  const uint32_t R = 1u << lr, J = 1u << lj, nthr = blockDim.x;
  const TileGeom G(A, tile);
  const bool pre = A.first && A.pre_table;
#pragma unroll 4
  for (uint32_t e = threadIdx.x; e < R * J; e += nthr) {
    // input rows are contiguous on the last pass
    const uint32_t k = !A.last ? e >> lj : e & (R - 1u), jj = !A.last ? e & (J - 1u) : e >> lr;
    const uint32_t pos = G.src(A, k, jj);
    uint32_t x = __ldcg(A.arrays.src[array] + pos);
    if (pre) x = mul1<P>(x, A.pre_table[pos]);
    sm[word_slot((k << lj) + jj)] = x;
  }
  __syncthreads();
  if (lr & 1) {
    const uint32_t half = word_slot(R * J >> 1);
    for (uint32_t u = threadIdx.x; u < R * J >> 1; u += nthr) {
      const uint32_t w = *stage_entry<P>(A, lr > 1 ? u >> lj : 0u);
      const uint32_t s = word_slot(u), x = sm[s], y = sm[s ^ half];
      sm[s] = add1<P>(x, y);
      sm[s ^ half] = mul1<P>(sub1<P>(x, y), w);
    }
    __syncthreads();
  }
  for (int s0 = lr & 1; s0 < lr; s0 += 2) {  // stages s0 and s0 + 1 on rows row + m 2^ls
    const int ls = lr - s0 - 2;
    const uint32_t d1 = word_slot(1u << (ls + lj)), d2 = word_slot(2u << (ls + lj));
    for (uint32_t u = threadIdx.x; u < R * J >> 2; u += nthr) {
      const uint32_t low = (u >> lj) & ((1u << ls) - 1u);
      const uint32_t w1 = *stage_entry<P>(A, (low + (1u << ls)) << s0);
      const uint32_t s = word_slot(((u >> (ls + lj)) << (ls + lj + 2)) + (u & ((1u << (ls + lj)) - 1u)));
      uint32_t x0 = sm[s], x1 = sm[s ^ d1], x2 = sm[s ^ d2], x3 = sm[s ^ d1 ^ d2];
      const uint32_t t0 = add1<P>(x0, x2), t1 = add1<P>(x1, x3);
      x2 = sub1<P>(x0, x2);
      x3 = mul1<P>(sub1<P>(x1, x3), w1);
      x0 = add1<P>(t0, t1);
      x1 = sub1<P>(t0, t1);
      if (ls != 0) {
        x2 = mul1<P>(x2, *stage_entry<P>(A, low << s0));
        const uint32_t w = *stage_entry<P>(A, low << (s0 + 1));
        x1 = mul1<P>(x1, w);
        const uint32_t t2 = sub1<P>(x2, x3);
        x2 = add1<P>(x2, x3);
        x3 = mul1<P>(t2, w);
      } else {
        const uint32_t t2 = sub1<P>(x2, x3);
        x2 = add1<P>(x2, x3);
        x3 = t2;
      }
      sm[s] = x0;
      sm[s ^ d1] = x1;
      sm[s ^ d2] = x2;
      sm[s ^ d1 ^ d2] = x3;
    }
    __syncthreads();
  }
  if constexpr (CHAIN) chain_next();
#pragma unroll 4
  for (uint32_t e = threadIdx.x; e < R * J; e += nthr) {
    const uint32_t k = e >> lj, jj = e & (J - 1u), pos = G.dst<P>(A, k, jj);
    Fe<P> x;
    x.l[0] = sm[word_slot((bitrev_bits(k, lr) << lj) + jj)];
    if (!A.last) {
      fe_mul_tw<P>(x, x, step_entry<P>(A, G.jbase + jj, k));
    } else {
      if (A.div_log) fe_div_pow2<P>(x, x, A.div_log);
      if (A.post_table) fe_mul_tw<P>(x, x, A.post_table + pos);
    }
    A.arrays.dst[array][pos] = x.l[0];
  }
  __syncthreads();
}

// One tile of one pass, multi-limb fields: a radix-2 DIF stage per phase, the first reading global memory itself (its
// product hides the latency), the last fused with the four-step factors and the store.  `sm` holds 2^(log_r + log_j)
// elements (tile_words).  LJ: the tile's log_j at compile time, or -1.
//
// Bound: the multiply pipe.  Each phase has its own product and straight code.  Sharing one product between the phases
// cost register moves where their values meet, and with them went generic addresses and run-time column counts: a
// BLS12-381 butterfly took 394 instructions, of which 218 are arithmetic, and 156 of them on the multiply pipe instead
// of 111 (GB300, ncu); here it takes about 300, 120 on that pipe.  With the table layout and the swizzle above, BLS12-381
// 2^20 went from 184 to 163 us and MNT4-753 2^18 / 2^20 from 302 / 1167 (inverse) to 294 / 1110 (chained launches, the
// low limb by shifts and the unreduced sums below have since made that 159 and 283 / 1090).  Barriers were not what
// was left of the 294 / 1110 and 163 (without them in the stages: 283 / 1119 and 162), nor was memory (every table and
// source read from L1: 4% less).  At 2^18 a pass is 1024 tiles on 152 SMs; an SM's seventh tile runs alone, one warp per
// scheduler, and one warp of carry chains reaches 66% of the pipe where two reach 96%.
//
// Values stay in [0, 2p) between the phases and the passes (a product's last subtraction is left out) until the last
// pass's store.
//
// The 24-limb field has room for 2^15 p: its sums and differences are not reduced at all. Stage ph takes values below
// 2^(ph+1) p (2p from the pass before), the last one gives values below 2^(log_r+1) p, and a four-step product brings them
// below 2p again; the last pass reduces by a quotient from the top word. log_r is at most 11 (shared memory), and 2^12 p
// bounds what kMaxLazyLog names.
template <class P>
__host__ __device__ constexpr bool tile_lazy() {
  return P::N >= 16;
}
template <class P>
__device__ __forceinline__ void tile_add(Fe<P>& r, const Fe<P>& x, const Fe<P>& y) {
  if constexpr (tile_lazy<P>()) {
    fe_add_lazy<P>(r, x, y);
  } else {
    fe_add<P, 2>(r, x, y);
  }
}
template <class P>
__device__ __forceinline__ void tile_sub(Fe<P>& r, const Fe<P>& x, const Fe<P>& y, int k) {  // x, y < 2^k p if lazy
  if constexpr (tile_lazy<P>()) {
    fe_sub_lazy<P>(r, x, y, k);
  } else {
    fe_sub<P, 2>(r, x, y);
  }
}

template <class P, int LJ, bool CHAIN>
__device__ __forceinline__ void field_tile(const PassArgs& A, unsigned array, uint32_t tile, uint32_t* sm) {
  constexpr int N = P::N;
  const int lr = A.log_r, lj = LJ >= 0 ? LJ : A.log_j;
  const uint32_t R = 1u << lr, J = 1u << lj, nthr = blockDim.x;
  const TileGeom G(A, tile);
  bool in_tile = false;  // the elements are in shared memory

  auto src = [&](uint32_t row, uint32_t jj) { return A.arrays.src[array] + (size_t)G.src(A, row, jj) * N; };
  auto at = [&](uint32_t slot) { return tile_at<P>(sm, slot); };

  if (A.first && A.pre_table) {  // coset transform: times the powers of the shift
#pragma unroll 1
    for (uint32_t b = threadIdx.x; b < R << lj; b += nthr) {
      const uint32_t jj = b & (J - 1u), t = b >> lj, pos = G.src(A, t, jj);
      Fe<P> x, r;
      fe_load_cg<P>(x, A.arrays.src[array] + (size_t)pos * N);
      fe_mul_tw<P, 2>(r, x, A.pre_table + tw_offset<P>(pos));
      tile_store<P>(at(tile_slot<LJ>(t, jj, lj)), r);
    }
    in_tile = true;
    __syncthreads();
  }

  // radix-2 DIF stages 0 .. lr-2 (natural order in, bit-reversed out)
#pragma unroll 1
  for (int ph = 0; ph < lr - 1; ++ph) {
    const uint32_t half = R >> (ph + 1), flip = tile_slot<LJ>(half, 0, lj);
#pragma unroll 1
    for (uint32_t b = threadIdx.x; b < (R >> 1) << lj; b += nthr) {
      // butterfly b = (i, group, jj) with the twiddle index i slowest, so that in the late stages, where 2^ph of the
      // butterflies have twiddle 1, whole warps skip the product
      const uint32_t jj = b & (J - 1u), t = b >> lj, i = t >> ph;
      const uint32_t u = ((t & ((1u << ph) - 1u)) << (lr - ph)) + i;
      const uint32_t su = tile_slot<LJ>(u, jj, lj);
      uint32_t *const pu = at(su), *const pv = at(su ^ flip);
      Fe<P> x, y, s;
      if (in_tile) {
        tile_load<P>(x, pu);
        tile_load<P>(y, pv);
      } else {
        fe_load_cg<P>(x, src(u, jj));
        fe_load_cg<P>(y, src(u + half, jj));
      }
      tile_add<P>(s, x, y);
      tile_store<P>(pu, s);
      tile_sub<P>(s, x, y, ph + 1);
      if (i != 0) {
        Fe<P> r;
        fe_mul_tw<P, 2>(r, s, stage_entry<P>(A, i << ph));
        tile_store<P>(pv, r);
      } else {
        tile_store<P>(pv, s);
      }
    }
    in_tile = true;
    __syncthreads();
  }

  // Last stage (twiddle 1): rows r and r + 1, r = bitrev(t) even, give outputs t and t + R/2; then the four-step factor
  // (non-last), or the division by n, the post table and the canonical form (last), and the store.
  auto emit = [&](Fe<P>& x, uint32_t t, uint32_t jj) {
    const uint32_t pos = G.dst<P>(A, t, jj);
    uint32_t* const out = A.arrays.dst[array] + (size_t)pos * N;
    if constexpr (tile_lazy<P>()) {
      if (A.last) fe_reduce_lazy<P>(x, x);
    }
    if (A.last && A.div_log) fe_div_pow2<P>(x, x, A.div_log);
    if (!A.last || A.post_table) {
      Fe<P> v;
      fe_mul_tw<P, 2>(v, x, A.last ? A.post_table + tw_offset<P>(pos) : step_entry<P>(A, G.jbase + jj, t));
      if (A.last) fe_reduce_once<P>(v, v.l);
      fe_store<P>(out, v);
    } else {
      if (!tile_lazy<P>()) fe_reduce_once<P>(x, x.l);
      fe_store<P>(out, x);
    }
  };
  if constexpr (CHAIN) chain_next();
#pragma unroll 1
  for (uint32_t b = threadIdx.x; b < (lr > 0 ? (R >> 1) << lj : J); b += nthr) {
    const uint32_t jj = b & (J - 1u), t = b >> lj, r = bitrev_bits(t, lr);
    Fe<P> x, y, s;
    if (in_tile) {
      const uint32_t su = tile_slot<LJ>(r, jj, lj);
      tile_load<P>(x, at(su));
      if (lr > 0) tile_load<P>(y, at(su ^ (1u << lj)));
    } else {
      fe_load_cg<P>(x, src(r, jj));
      if (lr > 0) fe_load_cg<P>(y, src(r + 1u, jj));
    }
    if (lr > 0) {
      tile_add<P>(s, x, y);
      tile_sub<P>(y, x, y, lr);
      emit(s, t, jj);
      emit(y, t + (R >> 1), jj);
    } else {
      emit(x, t, jj);
    }
  }
  __syncthreads();
}

// Register cap of the per-pass kernel.  24 limbs: 128, 4 CTAs of 128 threads per SM; GB300, MNT4 2^18 / 2^20 in us:
// 294 / 1104 at 128, 298 / 1141 at 144, 297 / 1137 at 168 (3 CTAs); a later form's 2^20 1113 at 128, 1114 at 120, 1128
// at 112.  8 limbs: 64, 8 CTAs: BLS 2^20 158.6 us, 157.3 at 56, 160.8 at 72, 163.9 at 80 and 96; the tile's first form
// 197 without a cap (84 registers), 184.3 at 64.  One limb:
// 64, so that blocks of 1024 threads launch.
template <class P>
constexpr int pass_max_regs() {
  return P::N >= 16 ? 128 : 64;
}

// MANY: the grid has a block row per array (PassArrays).  With one array its addresses stay in the parameter bank: the
// 8-limb passes run 1% slower with them in registers; the 24-limb ones do not notice and have the one form.
template <class P, int LJ, bool MANY>
__global__ void __maxnreg__(pass_max_regs<P>()) ntt_pass_kernel(const __grid_constant__ PassArgs A) {
  extern __shared__ uint4 gsn_smem[];
  uint32_t* sm = reinterpret_cast<uint32_t*>(gsn_smem);
  const unsigned array = MANY ? blockIdx.y : 0u;
  chain_wait();
  for (uint64_t t = blockIdx.x; t < A.tiles; t += gridDim.x) {  // tiles < 2^28
    if constexpr (P::N == 1) {
      word_tile<P, true>(A, array, (uint32_t)t, sm);
    } else {
      field_tile<P, LJ, true>(A, array, (uint32_t)t, sm);
    }
  }
}

// Entry e of `out`: base^e, for e in [0, count), in the form fe_mul_tw takes.
// `base` is canonical.  Each thread produces `chunk` consecutive powers: one
// square-and-multiply for the first, then one product (and for the multi-limb
// fields one reduction, the quotient) per entry.
template <class P>
__global__ void gen_powers_kernel(uint32_t* out, uint64_t count, Fe<P> base, int chunk) {
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t e0 = t * chunk;
  if (e0 >= count) return;
  Fe<P> bm, acc;
  fe_to_mont<P>(bm, base);
  fe_set_one_mont<P>(acc);
  // acc = bm^e0 (left to right over the bits of e0)
  if (e0 != 0) {
    for (int bit = 63 - __clzll((long long)e0); bit >= 0; --bit) {
      fe_mul<P>(acc, acc, acc);
      if ((e0 >> bit) & 1) fe_mul<P>(acc, acc, bm);
    }
  }
  const uint64_t end = (e0 + chunk < count) ? e0 + chunk : count;
  for (uint64_t e = e0; e < end; ++e) {
    fe_store_tw<P>(out + tw_offset<P>((uint32_t)e), acc);
    fe_mul<P>(acc, acc, bm);
  }
}

// Entry k 2^inner + j of `out`: entry (j k) << shift of `tw`, or j << shift where STAGE (r = 0).  One thread per 16-byte
// chunk, 8 threads a line.  Stage twiddles are copied too: computed as powers, and with the host exponentiations that named
// them, they took 510 us of a first call on a root of MNT4-753 2^18 (1515 us in all).
template <class P, bool STAGE>
__global__ void step_table_kernel(uint32_t* out, const uint32_t* tw, int r, int inner, int shift) {
  constexpr int CH = P::N / 2;  // chunks per entry
  const uint64_t count = (uint64_t)1 << (r + inner);
  const uint64_t total = ((count + 7) >> 3) * CH * 8;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t c = (uint32_t)((t >> 3) % CH);
    const uint32_t e = (uint32_t)((t >> 3) / CH * 8 + (t & 7));
    if (e >= count) continue;
    const uint32_t from = (STAGE ? e : (e & ((1u << inner) - 1u)) * (e >> inner)) << shift;
    *reinterpret_cast<uint4*>(out + tw_offset<P>(e) + c * kTwChunk) =
        *reinterpret_cast<const uint4*>(tw + tw_offset<P>(from) + c * kTwChunk);
  }
}

// Uniform elements of [0, p): limb j of attempt a of element i is the low
// word of splitmix64's finaliser applied to
//   seed + (i * 64 * N + a * N + j + 1) * 0x9E3779B97F4A7C15,
// the top limb is masked to bitlen(p) and attempts repeat until the value is
// below p (64 attempts at most; the acceptance rate is at least 1/2).
__device__ __forceinline__ uint64_t splitmix_mix(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

template <class P>
__global__ void fill_random_kernel(uint32_t* out, uint64_t n, uint64_t seed) {
  constexpr int N = P::N;
  constexpr int top_bits = P::BITS - 32 * (N - 1);
  constexpr uint32_t top_mask = top_bits >= 32 ? 0xFFFFFFFFu : ((1u << top_bits) - 1u);
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    Fe<P> x;
    bool ok = false;
    for (int a = 0; a < 64 && !ok; ++a) {
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const uint64_t ctr = i * 64ull * N + (uint64_t)a * N + j + 1;
        x.l[j] = (uint32_t)splitmix_mix(seed + ctr * 0x9E3779B97F4A7C15ull);
      }
      x.l[N - 1] &= top_mask;
      bool lt = false, decided = false;
#pragma unroll
      for (int j = N - 1; j >= 0; --j) {
        if (!decided && x.l[j] != P::mod(j)) {
          lt = x.l[j] < P::mod(j);
          decided = true;
        }
      }
      ok = lt;
    }
    if (!ok)
#pragma unroll
      for (int j = 0; j < N; ++j) x.l[j] = 0;
    fe_store<P>(out + i * N, x);
  }
}

// Element format conversions, in place:
//   mode 0: x -> x*R mod p      (enter Montgomery form: one product by R^2)
//   mode 1: x -> x*R^-1 mod p   (leave Montgomery form: one product by 1)
//   mode 2: reverse the limb order of each element (big-endian limb arrays,
//           as the reference's cpu_fields::Field stores them, fields/field.h:48,56,
//           <-> the little-endian im_rep of cuda/device_field.h:75)
template <class P>
__global__ void convert_kernel(uint32_t* data, uint64_t n, int mode) {
  chain_wait();
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    Fe<P> x, r;
    fe_load_cg<P>(x, data + i * P::N);
    if (mode == 0) {
      fe_to_mont<P>(r, x);
    } else if (mode == 1) {
      Fe<P> one;
#pragma unroll
      for (int j = 0; j < P::N; ++j) one.l[j] = j == 0 ? 1u : 0u;
      fe_mul<P>(r, x, one);
    } else {
#pragma unroll
      for (int j = 0; j < P::N; ++j) r.l[j] = x.l[P::N - 1 - j];
    }
    fe_store<P>(data + i * P::N, r);
  }
}

// a[i] = a[i] * b[i] mod p (canonical in, canonical out): two Montgomery
// products, the second by R^2.
template <class P>
__global__ void pointwise_mul_kernel(uint32_t* a, const uint32_t* b, uint64_t n) {
  chain_wait();
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    Fe<P> x, y, r;
    fe_load_cg<P>(x, a + i * P::N);
    fe_load_cg<P>(y, b + i * P::N);
    fe_mul<P>(r, x, y);
    fe_to_mont<P>(r, r);
    fe_store<P>(a + i * P::N, r);
  }
}

// Coset quotient of the QAP witness map: a[i] = (a[i] * b[i] - c[i]) * z, with
// z = 1 / Z(shift * w^i) = 1 / (shift^n - 1) the same for every point of a
// radix-2 coset.  Inputs canonical; zr2 = z * R^2 (Montgomery, twice), so
//   (mont(a, b) - mont(c, 1)) = (a b - c) / R  and  mont(that, z R^2) = (a b - c) z.
template <class P>
__global__ void coset_quotient_kernel(uint32_t* a, const uint32_t* b, const uint32_t* c, uint64_t n, Fe<P> zr2) {
  chain_wait();
  Fe<P> one;
#pragma unroll
  for (int j = 0; j < P::N; ++j) one.l[j] = j == 0 ? 1u : 0u;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    Fe<P> x, y, z, t, u;
    fe_load_cg<P>(x, a + i * P::N);
    fe_load_cg<P>(y, b + i * P::N);
    fe_load_cg<P>(z, c + i * P::N);
    fe_mul<P>(t, x, y);
    fe_mul<P>(u, z, one);
    fe_sub<P>(t, t, u);
    fe_mul<P>(t, t, zr2);
    fe_store<P>(a + i * P::N, t);
  }
}

// ---------------------------------------------------------------------------
// Batched transforms: one persistent launch over many jobs.
//
// work[t] = job << 32 | pass << 28 | tile, ordered by pass level (every
// level-0 tile of every job, then level 1, ...).  CTAs claim tickets in order
// from counters[0]; a tile of pass p > 0 first waits until
// counters[1 + job*kMaxPasses + p-1] reaches the tile count of pass p-1 of
// that job.  Those tiles hold smaller tickets, so they are already claimed by
// running CTAs that wait only on even smaller tickets: the waits always end.
// Each wait is still bounded (wait_cycles of clock64, kWaitBudgetCycles by
// default); on expiry the CTA records GSN_ERR_TIMEOUT in *status and carries
// on, so the launch always terminates.
// ---------------------------------------------------------------------------
constexpr long long kWaitBudgetCycles = 2LL * 1000 * 1000 * 1000;  // ~1 s at 2 GHz

__device__ __forceinline__ uint32_t ld_volatile_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.volatile.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

__device__ __forceinline__ void job_pass_args(PassArgs& A, const BatchJob& J, int pass) {
  int outer = 0;
  for (int i = 0; i < pass; ++i) outer += J.radix_log[i];
  A.first = pass == 0;
  A.last = pass == J.npass - 1;
  A.arrays.src[0] = A.first ? J.data : J.scratch;
  A.arrays.dst[0] = A.last ? J.data : J.scratch;
  A.tw = J.tw;
  A.tw_log = J.tw_log;
  A.stage_tw = J.stage_tw[pass];
  A.stage_shift = J.stage_shift[pass];
  A.step_tw = J.step_tw[pass];
  A.log_n = J.log_n;
  A.log_r = J.radix_log[pass];
  A.log_outer = outer;
  A.log_inner = J.log_n - outer - J.radix_log[pass];
  A.log_j = J.log_j[pass];
  A.inverse = J.inverse;
  A.npass = J.npass;
  for (int i = 0; i < kMaxPasses; ++i) A.radix_log[i] = J.radix_log[i];
  A.pre_table = A.first ? J.pre_table : nullptr;
  A.post_table = A.last ? J.post_table : nullptr;
  A.div_log = A.last ? J.div_log : 0;
  A.tiles = (uint64_t)1 << (J.log_n - A.log_r - A.log_j);
}

// Register cap of the persistent kernel: the per-pass kernel's, so the same
// occupancy, 4 CTAs of 128 threads per SM for the 753-bit field and 32 warps
// below.  256 BLS12-381 jobs of 2^10..2^16 take 495 us at 64, 512 at 56, 494
// at 72.
template <class P>
constexpr int batch_max_regs() {
  return P::N >= 16 ? 128 : 64;
}

template <class P>
__global__ void __maxnreg__(batch_max_regs<P>())
    batch_kernel(const BatchJob* __restrict__ jobs, const uint64_t* __restrict__ work,
                             uint64_t nwork, uint32_t* counters, uint32_t* status, long long wait_cycles) {
  extern __shared__ uint4 gsn_smem[];
  uint32_t* sm = reinterpret_cast<uint32_t*>(gsn_smem);
  __shared__ uint32_t s_ticket;
  __shared__ PassArgs s_args;
  for (;;) {
    if (threadIdx.x == 0) s_ticket = atomicAdd(&counters[0], 1u);
    __syncthreads();
    const uint32_t t = s_ticket;
    if (t >= nwork) return;
    const uint64_t w = work[t];
    const uint32_t job = (uint32_t)(w >> 32);
    const int pass = (int)((w >> 28) & 0xF);
    const uint32_t tile = (uint32_t)w & 0x0FFFFFFFu;
    if (threadIdx.x == 0) {
      const BatchJob& J = jobs[job];
      job_pass_args(s_args, J, pass);
      if (pass > 0) {
        const uint32_t need = (uint32_t)((uint64_t)1 << (J.log_n - J.radix_log[pass - 1] - J.log_j[pass - 1]));
        const uint32_t* cnt = &counters[1 + (uint64_t)job * kMaxPasses + pass - 1];
        const long long start = clock64();
        while (ld_volatile_u32(cnt) < need) {
          if (clock64() - start > wait_cycles) {
            atomicExch(status, 8u);  // GSN_ERR_TIMEOUT
            break;
          }
          __nanosleep(256);
        }
        __threadfence();
      }
    }
    __syncthreads();
    // each ends with __syncthreads(); s_args is rewritten only after it
    if constexpr (P::N == 1) {
      word_tile<P, false>(s_args, 0, tile, sm);
    } else {
      field_tile<P, -1, false>(s_args, 0, tile, sm);
    }
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(&counters[1 + (uint64_t)job * kMaxPasses + pass], 1u);
    }
  }
}

// --- host-side launchers, instantiated per field ---------------------------
// Elementwise grid-stride kernels launch at most this many CTAs per SM.
constexpr uint64_t kGridPerSm = 64;

// Multi-limb tables of powers up to this size have 8 entries a thread and one warp a block: they do not fill the chip, and a
// thread's chain of entries is their time. First call on a shift, GB300, us, 32 entries and 8: MNT4-753 2^10 355 and 185,
// 2^14 495 and 322, 2^18 785 and 760, 2^20 1950 and 2550; BLS12-381 2^16 178 and 157, 2^20 366 and 389.
constexpr uint64_t kPowSmall = (uint64_t)1 << 18;

template <class P>
struct Kernels {
  using PassKernel = void (*)(PassArgs);
  static constexpr bool kManyOnly = P::N >= 16;  // one array goes by the many-array form too
  template <bool MANY>
  static PassKernel kernel_for(int log_j) {
    if constexpr (P::N > 1) {
      if (log_j == 2) return ntt_pass_kernel<P, 2, MANY>;
    }
    if constexpr (P::N == 8) {
      if (log_j == 0) return ntt_pass_kernel<P, 0, MANY>;
      if (log_j == 1) return ntt_pass_kernel<P, 1, MANY>;
    }
    return ntt_pass_kernel<P, -1, MANY>;
  }
  static cudaError_t pass(const PassArgs& A, int arrays, int block, cudaStream_t s) {
    const size_t smem = tile_words(P::N, (uint64_t)1 << (A.log_r + A.log_j)) * sizeof(uint32_t);
    auto k = arrays == 1 ? kernel_for<kManyOnly>(A.log_j) : kernel_for<true>(A.log_j);
    if (smem > kDefaultSmemOptIn) {
      cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
    }
    const uint64_t grid = A.tiles < (1u << 20) ? A.tiles : (1u << 20);
    // a plan's block may be larger than the register cap lets a block be; the tile loops over any block
    const int most = 65536 / pass_max_regs<P>() / 32 * 32;
    return launch_chained(k, dim3((unsigned)grid, (unsigned)arrays), (unsigned)std::min(block, most), smem, s, A);
  }
  static cudaError_t powers(uint32_t* out, uint64_t count, const uint32_t* base_canon, cudaStream_t s) {
    Fe<P> b;
    for (int i = 0; i < P::N; ++i) b.l[i] = base_canon[i];
    const bool small = P::N > 1 && count <= kPowSmall;
    const int chunk = small ? 8 : 32, block = small ? 32 : 128;
    const uint64_t threads = (count + chunk - 1) / chunk;
    gen_powers_kernel<P><<<(unsigned)((threads + block - 1) / block), block, 0, s>>>(out, count, b, chunk);
    return cudaGetLastError();
  }
  static cudaError_t step_table(uint32_t* out, const uint32_t* tw, int r, int inner, int shift, cudaStream_t s) {
    return copy_table<false>(out, tw, r, inner, shift, s);
  }
  static cudaError_t stage_table(uint32_t* out, const uint32_t* tw, int log_count, int shift, cudaStream_t s) {
    return copy_table<true>(out, tw, 0, log_count, shift, s);
  }
  template <bool STAGE>
  static cudaError_t copy_table(uint32_t* out, const uint32_t* tw, int r, int inner, int shift, cudaStream_t s) {
    if constexpr (P::N == 1) {
      return cudaErrorInvalidValue;  // its passes read `tw` itself
    } else {
      const int block = 256;
      const uint64_t threads = ((uint64_t)1 << (r + inner)) * (P::N / 2);
      const uint64_t grid =
          std::min<uint64_t>(threads / block + 1, kGridPerSm * (uint64_t)current_device_sms());
      step_table_kernel<P, STAGE><<<(unsigned)grid, block, 0, s>>>(out, tw, r, inner, shift);
      return cudaGetLastError();
    }
  }
  static cudaError_t batch(const BatchJob* jobs_dev, const uint64_t* work_dev, uint64_t nwork,
                           uint32_t* counters_dev, uint32_t* status_dev, int grid, int block, size_t smem,
                           cudaStream_t s, long long wait_cycles) {
    auto k = batch_kernel<P>;
    if (smem > kDefaultSmemOptIn) {
      cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
    }
    k<<<grid, block, smem, s>>>(jobs_dev, work_dev, nwork, counters_dev, status_dev,
                                wait_cycles > 0 ? wait_cycles : kWaitBudgetCycles);
    return cudaGetLastError();
  }
  // Loads code that CUDA otherwise loads at each kernel's first launch: the batched kernel's and that of the passes that
  // transform one array.
  static cudaError_t load() {
    cudaFuncAttributes attr;
    cudaError_t e = cudaFuncGetAttributes(&attr, batch_kernel<P>);
    for (int lj = 0; lj <= 3 && e == cudaSuccess; ++lj)
      e = cudaFuncGetAttributes(&attr, kernel_for<kManyOnly>(lj));
    return e;
  }
  static int batch_occupancy(int block, size_t smem) {
    auto k = batch_kernel<P>;
    if (smem > kDefaultSmemOptIn) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, block, smem) != cudaSuccess) return 0;
    return nb;
  }
  static cudaError_t convert(uint32_t* data, uint64_t n, int mode, cudaStream_t s) {
    const int block = 256;
    uint64_t grid = (n + block - 1) / block;
    if (grid > kGridPerSm * (uint64_t)current_device_sms()) grid = kGridPerSm * (uint64_t)current_device_sms();
    if (grid == 0) return cudaSuccess;
    return launch_chained(convert_kernel<P>, (unsigned)grid, block, 0, s, data, n, mode);
  }
  static cudaError_t fill(uint32_t* out, uint64_t n, uint64_t seed, cudaStream_t s) {
    const int block = 256;
    uint64_t grid = (n + block - 1) / block;
    if (grid > kGridPerSm * (uint64_t)current_device_sms()) grid = kGridPerSm * (uint64_t)current_device_sms();
    if (grid == 0) return cudaSuccess;
    fill_random_kernel<P><<<(unsigned)grid, block, 0, s>>>(out, n, seed);
    return cudaGetLastError();
  }
  static cudaError_t pointwise(uint32_t* a, const uint32_t* b, uint64_t n, cudaStream_t s) {
    const int block = 256;
    uint64_t grid = (n + block - 1) / block;
    if (grid > kGridPerSm * (uint64_t)current_device_sms()) grid = kGridPerSm * (uint64_t)current_device_sms();
    return launch_chained(pointwise_mul_kernel<P>, (unsigned)grid, block, 0, s, a, b, n);
  }
  static cudaError_t quotient(uint32_t* a, const uint32_t* b, const uint32_t* c, uint64_t n, const uint32_t* zr2,
                              cudaStream_t s) {
    Fe<P> z;
    for (int i = 0; i < P::N; ++i) z.l[i] = zr2[i];
    const int block = 256;
    uint64_t grid = (n + block - 1) / block;
    if (grid > kGridPerSm * (uint64_t)current_device_sms()) grid = kGridPerSm * (uint64_t)current_device_sms();
    if (grid == 0) return cudaSuccess;
    return launch_chained(coset_quotient_kernel<P>, (unsigned)grid, block, 0, s, a, b, c, n, z);
  }
};

}  // namespace gsn
