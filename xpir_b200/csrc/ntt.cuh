// The reference's lazy DIF NTT (crypto/NFLlib.hpp:450-537) on polynomials held in shared
// memory, shared by the import and the query encryption (forward twiddles) and the
// client-side decryption (inverse twiddles after a bit-reversal, crypto/NFLlib.hpp:548-566).
// All threads of the block take part.  Its layers: log2(N)-2 radix-2 layers (inputs and
// outputs in [0, 2p)), then the last two layers fused per group of four.
//
// What bounds it: the multiplier and the issue slots (a lazy Shoup product is six 32x32+64-bit
// multiply-adds of four issue cycles each and four of two).  So everything around the
// products is kept small: the degree is a template parameter (every stride, twiddle offset
// and shared-memory offset is an immediate), a twiddle and its Shoup factor are one 16-byte
// load, sums are reduced by their sign, and the first pass takes its coefficients from the
// caller's producer.  Against a transform with run-time degree and separate factor tables,
// B200, instructions per coefficient of the whole import kernel 336 -> 222: 16,000 polys of
// 2048 526 -> 352 us, 24,576 of 4096 (74 bits) 2526 -> 1440 us.  Two polynomials per thread
// sharing each twiddle load: 205 instructions but half the warps, 346..393 us.
#pragma once

#include <stdint.h>

#include "modarith.cuh"

namespace xpir {

// Position of coefficient idx in a swizzled shared-memory polynomial: the low 4 bits of
// the word index XORed with bits 7..4, so that the passes of ntt_lazy (and the callers'
// coefficient-order loops) read and write shared memory with few or no bank conflicts; REV:
// with bits 10..7 as well, which also spreads the lanes of a bit-reversed order (their index
// bits are the high ones).  Linear over XOR, so swz(a | b) = swz(a) ^ swz(b) for disjoint bits.
template <bool REV = false>
__host__ __device__ constexpr uint32_t swz(uint32_t idx) {
  return idx ^ ((REV ? (idx >> 4) ^ (idx >> 7) : idx >> 4) & 15u);
}

// x less 2p unless that is negative.  For coefficients that began in [0, 2p) x stays below 4p
// < 2^63 and the sign bit tells; ANY: for words of any size (what a decryption may meet) only
// the comparison has the reference's bits.
template <bool ANY>
__device__ __forceinline__ uint64_t less_2p(uint64_t x, uint64_t p2) {
  const uint64_t d = x - p2;
  if constexpr (ANY) return x >= p2 ? d : x;
  return (int64_t)d < 0 ? x : d;
}

// One radix-2 layer of the lazy DIF butterfly on 8 register-held coefficients whose indices
// are base | (r << LO): the pair differs in bit LO + RB of the
// index, and the twiddle index is the lower index modulo the layer's half-length (the
// twiddles of layer `half` start at tw + N - 2*half).
template <int LOGN, int LO, int RB, bool ANY>
__device__ __forceinline__ void ntt_layer(uint64_t (&x)[8], uint32_t base, const ulonglong2 *__restrict__ tw,
                                          uint64_t np, uint64_t p2) {
  constexpr uint32_t half = 1u << (LO + RB), off = (1u << LOGN) - 2 * half;
  const ulonglong2 *t = tw + off + (base & (half - 1));
#pragma unroll
  for (uint32_t k = 0; k < (1u << RB); k++) {
    const bool one = LO == 0 && k == 0;  // every thread's twiddle is the layer's first power, 1
    const ulonglong2 w = one ? make_ulonglong2(1, 8) : __ldg(t + (k << LO));
#pragma unroll
    for (uint32_t r = k; r < 8; r += 1u << RB) {
      if (r & (1u << RB)) continue;
      const uint64_t u0 = x[r], u1 = x[r | (1u << RB)];
      x[r] = less_2p<ANY>(u0 + u1, p2);
      const uint64_t t1 = u0 - u1 + p2;
      x[r | (1u << RB)] = one ? shoup_lazy_one_np(t1, np) : shoup_lazy_np(t1, w.x, w.y, np);
    }
  }
}

// The passes on index bits TOP .. 3, three at a time: each thread holds 8 coefficients whose
// indices differ in three consecutive bits and runs up to three layers on them before
// exchanging through shared memory.  A short last group also holds the bits below 3, left to
// the last pass.
template <int LOGN, int TOP, bool FIRST, bool ALIAS, bool ANY, class Load>
__device__ __forceinline__ void ntt_passes(uint64_t *s, const ulonglong2 *__restrict__ tw, uint64_t np, uint64_t p2,
                                           Load load) {
  if constexpr (TOP >= 3) {
    constexpr int LO = TOP - 2;
    constexpr uint32_t N = 1u << LOGN;
    if constexpr (!FIRST) __syncthreads();
    for (uint32_t g = threadIdx.x; g < N / 8; g += blockDim.x) {
      const uint32_t base = ((g >> LO) << (LO + 3)) | (g & ((1u << LO) - 1));
      const uint32_t at = swz<ANY>(base);
      uint64_t x[8];
      if constexpr (FIRST) {
#pragma unroll
        for (uint32_t r = 0; r < 8; r++) x[r] = load(base | (r << LO));
      } else {
#pragma unroll
        for (uint32_t r = 0; r < 8; r++) x[r] = s[at ^ swz<ANY>(r << LO)];
      }
      ntt_layer<LOGN, LO, 2, ANY>(x, base, tw, np, p2);
      if constexpr (LO + 1 >= 3) ntt_layer<LOGN, LO, 1, ANY>(x, base, tw, np, p2);
      if constexpr (LO >= 3) ntt_layer<LOGN, LO, 0, ANY>(x, base, tw, np, p2);
      if constexpr (FIRST && ALIAS) __syncthreads();
#pragma unroll
      for (uint32_t r = 0; r < 8; r++) s[at ^ swz<ANY>(r << LO)] = x[r];
    }
    ntt_passes<LOGN, TOP - 3, false, ALIAS, ANY>(s, tw, np, p2, load);
  }
}

// The reference's butterflies with its lazy reductions, so its output bits.  The first pass
// takes its inputs from load(idx), coefficient idx, in [0, 2p) unless ANY; the output is left
// in s[swz<ANY>(idx)] (after a barrier).
// 512 <= N <= 8192; any block size, but N/8 threads with ALIAS: load reads memory that s
// overlaps, so no thread writes s before all have loaded.
template <int LOGN, bool ALIAS, bool ANY = false, class Load>
__device__ __forceinline__ void ntt_lazy(uint64_t *s, const ulonglong2 *__restrict__ tw, uint64_t p, Load load) {
  constexpr uint32_t N = 1u << LOGN;
  const uint64_t p2 = p << 1, np = 0 - p;
  ntt_passes<LOGN, LOGN - 1, true, ALIAS, ANY>(s, tw, np, p2, load);
  __syncthreads();
  // Bits 2..0 on 8 consecutive coefficients: one layer, then the fused last two.
  const ulonglong2 w1 = __ldg(tw + N - 4 + 1);
  for (uint32_t g = threadIdx.x; g < N / 8; g += blockDim.x) {
    const uint32_t base = g * 8, at = swz<ANY>(base);
    uint64_t x[8];
#pragma unroll
    for (uint32_t r = 0; r < 8; r++) x[r] = s[at ^ r];
    ntt_layer<LOGN, 0, 2, ANY>(x, 0, tw, np, p2);
#pragma unroll
    for (uint32_t r = 0; r < 8; r += 4) {
      const uint64_t u0 = x[r], u1 = x[r + 1], u2 = x[r + 2], u3 = x[r + 3];
      const uint64_t v0 = less_2p<ANY>(u0 + u2, p2), v1 = less_2p<ANY>(u1 + u3, p2);
      uint64_t v2 = u0 - u2;
      v2 = ((int64_t)v2 < 0) ? v2 + p2 : v2;
      const uint64_t v3 = shoup_lazy_np(u1 - u3 + p2, w1.x, w1.y, np);
      const uint64_t z1 = v0 - v1, z3 = v2 - v3;
      s[at ^ r] = less_2p<ANY>(v0 + v1, p2);
      s[at ^ (r + 1)] = ((int64_t)z1 < 0) ? z1 + p2 : z1;
      s[at ^ (r + 2)] = less_2p<ANY>(v2 + v3, p2);
      s[at ^ (r + 3)] = ((int64_t)z3 < 0) ? z3 + p2 : z3;
    }
  }
  __syncthreads();
}

// Threads of a block that transforms polynomials of degree N: a group of 8 coefficients each,
// at most 512.
inline uint32_t ntt_threads(uint32_t N) { return N / 8 < 512 ? N / 8 : 512; }

// Runs f.template operator()<LOGN>() for a supported degree.
#define XPIR_BY_DEGREE(log_n, F)  \
  switch (log_n) {                \
    case 9: F(9); break;          \
    case 10: F(10); break;        \
    case 11: F(11); break;        \
    case 12: F(12); break;        \
    default: F(13); break;        \
  }

}  // namespace xpir
