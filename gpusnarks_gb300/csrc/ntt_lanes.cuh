// Pass kernel of small 24-limb transforms: four lanes per product.
//
// A small transform leaves most SMs with one warp per scheduler or none, and its time is the chain of dependent products
// (log2 n + passes). One warp alone takes 5,410 cycles for a 24-limb product, 899 multiply-adds on carry chains at 6.0
// cycles a step (GB300); the product below takes it 1,920. Four neighbouring lanes share a product: lane g takes rows
// i = g mod 4 of its three limb products, a quarter of the chain. Rows of one warp instruction have to start at one word, so each lane holds the operand shifted
// up by g words (27 words) and multiplies row 4c of that by limb 4c + g of the constant. The partial sums are added
// across the lanes by shuffles, which leaves the quotient and the product in all four. Additions, subtractions and the
// tile's addressing are done by all four alike. Total work grows by half, so this is for sizes that do not fill the
// chip; the plan says which kernel a size takes.
//
// The quotient leaves out the same word products as fe_mul_tw's, so it is the same number and so are the bounds and the
// results, values in [0, 2p) until the last pass's store. The modulus's low limb is multiplied like the others here (by
// limbs of R - p), where fe_mul_tw shifts and subtracts: modulo R that is the same. Tables, tiles and phases are field_tile's.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "arith.cuh"
#include "chain.cuh"
#include "ntt_common.h"
#include "ntt_kernels.cuh"

namespace gsn {
namespace lanes {

constexpr int kLanes = 4;
constexpr int kMaxBlock = 256;

// out[j] = x[j - g], j < COUNT, g = 0..3 (zero below and above x).
template <int N, int COUNT>
__device__ __forceinline__ void shift_words(uint32_t (&out)[COUNT], const uint32_t (&x)[N], uint32_t g) {
  auto word = [&](int j) { return j >= 0 && j < N ? x[j] : 0u; };
  uint32_t t[COUNT];
#pragma unroll
  for (int j = 0; j < COUNT; ++j) t[j] = (g & 1u) ? word(j - 1) : word(j);
#pragma unroll
  for (int j = 0; j < COUNT; ++j) out[j] = (g & 2u) ? (j >= 2 ? t[j - 2] : 0u) : t[j];
}

// v = sum of v over the four lanes, modulo 2^(32 COUNT).
template <int COUNT>
__device__ __forceinline__ void sum_lanes(uint32_t (&v)[COUNT]) {
#pragma unroll
  for (int m = 1; m < kLanes; m <<= 1) {
    uint32_t o[COUNT];
#pragma unroll
    for (int j = 0; j < COUNT; ++j) o[j] = __shfl_xor_sync(0xFFFFFFFFu, v[j], m);
    ptx::add_cc(v[0], v[0], o[0]);
#pragma unroll
    for (int j = 1; j < COUNT - 1; ++j) ptx::addc_cc(v[j], v[j], o[j]);
    ptx::addc(v[COUNT - 1], v[COUNT - 1], o[COUNT - 1]);
  }
}

// A lane's limbs 4c + g of a table entry's w and w'.
template <class P>
struct Factor {
  uint32_t w[P::N / 4], wq[P::N / 4];
};
template <class P>
__device__ __forceinline__ void load_factor(Factor<P>& f, const uint32_t* e, uint32_t g) {
#pragma unroll
  for (int c = 0; c < P::N / 4; ++c) {
    f.w[c] = e[c * kTwChunk + g];
    f.wq[c] = e[(P::N / 4 + c) * kTwChunk + g];
  }
}

// r = x * w mod p, below 2p, in all four lanes; all of a warp's lanes call it.  neg: limbs 4c + g of R - p.
template <class P>
__device__ __forceinline__ void mul(Fe<P>& r, const Fe<P>& x, const Factor<P>& f, const uint32_t (&neg)[P::N / 4],
                                    uint32_t g) {
  constexpr int N = P::N;
  uint32_t xs[N + 3], h[N + 2];
  shift_words<N, N + 3>(xs, x.l, g);
  {
    // words N-2 .. 2N-1 of the lane's rows, as high_row: E[k] is word N-2+k, O[k] word N-1+k
    uint32_t E[N + 2], O[N + 2];
#pragma unroll
    for (int j = 0; j < N + 2; ++j) E[j] = O[j] = 0u;
#pragma unroll
    for (int c = 0; c < N / 4; ++c) {
      const int i = 4 * c, je = i < N - 2 ? N - 2 - i : 0, jo = i < N - 1 ? N - 1 - i : 1;
      int k = 0;
#pragma unroll
      for (int j = je; j <= N + 2; j += 2) {
        k = i + j - (N - 2);
        wide_step(E[k], E[k + 1], xs[j], f.wq[c], j == je);
      }
      if (k + 2 <= N + 1) ptx::addc(E[k + 2], E[k + 2], 0u);
#pragma unroll
      for (int j = jo; j <= N + 1; j += 2) {
        k = i + j - (N - 1);
        wide_step(O[k], O[k + 1], xs[j], f.wq[c], j == jo);
      }
      if (k + 2 <= N) ptx::addc(O[k + 2], O[k + 2], 0u);
    }
    h[0] = E[0];
    ptx::add_cc(h[1], E[1], O[0]);
#pragma unroll
    for (int k = 2; k <= N; ++k) ptx::addc_cc(h[k], E[k], O[k - 1]);
    ptx::addc(h[N + 1], E[N + 1], O[N]);
  }
  sum_lanes<N + 2>(h);
  uint32_t E[N], O[N], t[N];
#pragma unroll
  for (int j = 0; j < N; ++j) E[j] = O[j] = 0u;
  auto xl = [&](int j) { return xs[j]; };
#pragma unroll
  for (int c = 0; c < N / 4; ++c) low_row<N>(E, O, xl, 4 * c, f.w[c]);
  {
    uint32_t q[N], qs[N];
#pragma unroll
    for (int j = 0; j < N; ++j) q[j] = h[j + 2];
    shift_words<N, N>(qs, q, g);
    auto ql = [&](int j) { return qs[j]; };
#pragma unroll
    for (int c = 0; c < N / 4; ++c) low_row<N>(E, O, ql, 4 * c, neg[c]);
  }
  t[0] = E[0];
  ptx::add_cc(t[1], E[1], O[0]);
#pragma unroll
  for (int j = 2; j < N - 1; ++j) ptx::addc_cc(t[j], E[j], O[j - 1]);
  ptx::addc(t[N - 1], E[N - 1], O[N - 2]);
  sum_lanes<N>(t);
#pragma unroll
  for (int j = 0; j < N; ++j) r.l[j] = t[j];
}

}  // namespace lanes

template <class P>
__global__ void __launch_bounds__(lanes::kMaxBlock) ntt_lanes_kernel(const __grid_constant__ PassArgs A) {
  using namespace lanes;
  constexpr int N = P::N;
  extern __shared__ uint4 gsn_smem[];
  uint32_t* sm = reinterpret_cast<uint32_t*>(gsn_smem);
  const int lr = A.log_r, lj = A.log_j;
  const uint32_t R = 1u << lr, J = 1u << lj;
  const uint32_t g = threadIdx.x & (kLanes - 1), groups = blockDim.x / kLanes;
  const unsigned array = blockIdx.y;
  uint32_t neg[N / 4];
#pragma unroll
  for (int c = 0; c < N / 4; ++c)
    neg[c] = g == 0 ? neg_mod<P>(4 * c) : g == 1 ? neg_mod<P>(4 * c + 1) : g == 2 ? neg_mod<P>(4 * c + 2)
                                                                                 : neg_mod<P>(4 * c + 3);
  chain_wait();
  for (uint64_t tile = blockIdx.x; tile < A.tiles; tile += gridDim.x) {
    const TileGeom G(A, (uint32_t)tile);
    bool in_tile = false;
    // Phases as in field_tile: -1 pre-scale, 0 .. lr-2 stages, lr the last stage with the outputs one per group.
#pragma unroll 1
    for (int ph = A.first && A.pre_table ? -1 : lr >= 2 ? 0 : lr; ph <= lr; ph += ph == lr - 2 ? 2 : 1) {
      const bool stage = ph >= 0 && ph < lr;
      const uint32_t count = stage ? (R >> 1) << lj : R << lj;
      const uint32_t half = stage ? R >> (ph + 1) : 1u, flip = tile_slot<-1>(half, 0, lj);
      if (ph == lr && tile + gridDim.x >= A.tiles) chain_next();
      // whole warps stay together for the shuffles: groups past the end repeat the last element and do not store
#pragma unroll 1
      for (uint32_t b0 = 0; b0 < count; b0 += groups) {
        const uint32_t mine = b0 + threadIdx.x / kLanes;
        if (b0 + (threadIdx.x & ~31u) / kLanes >= count) break;  // the whole warp is past the end
        const bool valid = mine < count;
        const uint32_t b = valid ? mine : count - 1u;
        // A pass in the middle works in place, and with radix 2 no stage has brought its tile into shared memory: the two
        // outputs of a column then go to neighbouring groups, so that one warp has read both rows before it stores either.
        const uint32_t jj = lr == 1 ? b >> 1 : b & (J - 1u), t = lr == 1 ? b & 1u : b >> lj;
        Fe<P> x, y;
        Factor<P> f;
        bool mul_here = true;
        uint32_t su = 0, pos = 0;
        if (ph < 0) {
          pos = G.src(A, t, jj);
          load_factor<P>(f, A.pre_table + tw_offset<P>(pos), g);
          fe_load_cg<P>(x, A.arrays.src[array] + (size_t)pos * N);
          su = tile_slot<-1>(t, jj, lj) ^ flip;  // stored at su ^ flip below
        } else {
          const uint32_t i = t >> ph;
          const uint32_t r = stage ? ((t & ((1u << ph) - 1u)) << (lr - ph)) + i : bitrev_bits(t, lr);
          const uint32_t u = stage ? r : r & ~1u;
          if (stage) {
            load_factor<P>(f, stage_entry<P>(A, i << ph), g);
          } else {
            pos = G.dst<P>(A, t, jj);
            mul_here = !A.last || A.post_table;
            if (mul_here)
              load_factor<P>(f, A.last ? A.post_table + tw_offset<P>(pos) : step_entry<P>(A, G.jbase + jj, t), g);
          }
          su = tile_slot<-1>(u, jj, lj);
          if (in_tile) {
            tile_load<P>(x, tile_at<P>(sm, su));
            if (lr > 0) tile_load<P>(y, tile_at<P>(sm, su ^ flip));
          } else {
            fe_load_cg<P>(x, A.arrays.src[array] + (size_t)G.src(A, u, jj) * N);
            if (lr > 0) fe_load_cg<P>(y, A.arrays.src[array] + (size_t)G.src(A, u + half, jj) * N);
          }
          __syncwarp();  // all four lanes have read what the first one overwrites
          if (stage) {
            Fe<P> s;
            fe_add<P, 2>(s, x, y);
            fe_sub<P, 2>(x, x, y);
            // a group past the end may read what this writes: its results are not used
            if (valid && g == 0) tile_store<P>(tile_at<P>(sm, su), s);
          } else {
            if (lr > 0) {
              if (r & 1u) {
                fe_sub<P, 2>(x, x, y);
              } else {
                fe_add<P, 2>(x, x, y);
              }
            }
            if (A.last && A.div_log) fe_div_pow2<P>(x, x, A.div_log);
          }
        }
        __syncwarp();
        if (mul_here) mul<P>(x, x, f, neg, g);  // uniform over the block
        if (ph < lr) {
          if (valid && g == 0) tile_store<P>(tile_at<P>(sm, su ^ flip), x);
        } else {
          if (A.last) fe_reduce_once<P>(x, x.l);
          if (valid && g == 0) fe_store<P>(A.arrays.dst[array] + (size_t)pos * N, x);
        }
      }
      in_tile = true;
      __syncthreads();
    }
  }
}

template <class P>
struct LanesKernels {
  static cudaError_t load() {
    if constexpr (P::N == 24) {
      cudaFuncAttributes attr;
      return cudaFuncGetAttributes(&attr, ntt_lanes_kernel<P>);
    }
    return cudaSuccess;
  }
  // Built for the 24-limb field only.
  static cudaError_t pass(const PassArgs& A, int arrays, int block, cudaStream_t s) {
    if constexpr (P::N != 24) {
      return cudaErrorInvalidValue;
    } else {
      const size_t smem = tile_words(P::N, (uint64_t)1 << (A.log_r + A.log_j)) * sizeof(uint32_t);
      auto k = ntt_lanes_kernel<P>;
      if (smem > kDefaultSmemOptIn) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
      }
      const uint64_t grid = A.tiles < (1u << 20) ? A.tiles : (1u << 20);
      return launch_chained(k, dim3((unsigned)grid, (unsigned)arrays), (unsigned)std::min(block, lanes::kMaxBlock), smem,
                            s, A);
    }
  }
};

}  // namespace gsn
