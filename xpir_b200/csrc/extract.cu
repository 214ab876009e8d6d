// Client-side reply extraction on the GPU: NFLLWE decryption of every reply ciphertext
// and the recursion back to the element (crypto/NFLLWE.cpp:375-475, 515-551;
// pir/replyExtraction/PIRReplyExtraction_internal.cpp:41-106).
//
// Per level, two kernels:
//   decrypt_poly_kernel  one CTA per (ciphertext, modulus): m = b - a*s (lazy Shoup MAC
//                        then submod, crypto/NFLlib.hpp:255-267, 303-321), bit reversal,
//                        the lazy NTT with the inverse twiddles, bit reversal back, and
//                        the N^-1 phi^-i scaling (crypto/NFLlib.hpp:548-566, 613-626);
//   lift_pack_kernel     one thread per (ciphertext, coefficient): the CRT lift to
//                        [0, P) by mixed radix (the unique value NFLlib::poly2mpz also
//                        computes, crypto/NFLlib.cpp:504-532), centred (x - P when
//                        2x > P), its low b bits appended LSB-first to the ciphertext's
//                        plaintext bytes (the bit order of NFLlib::serializeData32/64,
//                        crypto/NFLlib.cpp:412-495).
// The level's plaintext bytes are the next level's ciphertexts; the innermost level's
// are the aggregated element.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "handles.h"
#include "kernels.h"
#include "modarith.cuh"
#include "ntt.cuh"
#include "params.h"
#include "residue_sum.cuh"
#include "xpir_b200.h"

namespace xpir {
namespace {

constexpr uint32_t kMaxLiftModuli = 4;  // b < 128 bits per coefficient
constexpr int kLimbs = kMaxLiftModuli + 1;
constexpr int kExtractThreads = 256;  // of the decrypting kernels
// Ciphertexts from which one CTA per ciphertext fills the GPU, and the shared memory it may
// take (two CTAs per SM; larger parameter sets keep the two kernels).
constexpr uint64_t kFusedCiphertexts = 296;
constexpr size_t kFusedSmem = 112 * 1024;

// Mixed-radix constants: x = v0 + v1*M1 + ... with M_c = p_0*...*p_{c-1}.
struct LiftConsts {
  uint64_t P[kLimbs];              // product of the moduli
  uint64_t M[kMaxLiftModuli][kLimbs];
  uint64_t inv[kMaxLiftModuli];    // M_c^-1 mod p_c
  uint64_t inv_shoup[kMaxLiftModuli];  // floor(inv * 2^64 / p_c)
};

// Exact reductions modulo one of XPIR's moduli (mod_word, mod_two_words) give the unique
// residue the reference's GMP lift computes.
//
// x (its low NL little-endian limbs) mod p, from the top limb down.
template <int NL>
__device__ __forceinline__ uint64_t limbs_mod_fast(const uint64_t *x, uint64_t p, uint64_t np, uint32_t delta) {
  uint64_t r = mod_word(x[NL - 1], p, np);
#pragma unroll
  for (int l = NL - 2; l >= 0; l--) r = mod_two_words(r, x[l], p, np, delta);
  return r;
}

// b - a*s of one ciphertext and modulus, transformed back: coefficient k (before the N^-1
// phi^-k scaling) is left in poly[swz<true>(brev(k))].
template <int LOGN>
__device__ __forceinline__ void decrypt_poly(uint64_t *poly, const uint64_t *__restrict__ a,
                                             const uint64_t *__restrict__ b, const uint64_t *__restrict__ s,
                                             const uint64_t *__restrict__ ss, const uint64_t *__restrict__ tab,
                                             uint64_t p) {
  constexpr uint32_t N = 1u << LOGN, shift = 32 - LOGN;
  // Unrolled: eight rows of loads in flight (the 4,764 ciphertexts 348 us, four rows 360).
#pragma unroll 8
  for (uint32_t i = threadIdx.x; i < N; i += kExtractThreads) {
    const uint64_t temp = shoup_mac(0, a[i], s[i], ss[i], p);  // in [0, p)
    const uint64_t y = (temp < p) ? p - temp : p - temp % p;
    uint64_t z = b[i] + y;
    z -= (z >= p) ? p : 0;
    poly[swz<true>(__brev(i) >> shift)] = z;
  }
  __syncthreads();
  ntt_lazy<LOGN, false, true>(poly, reinterpret_cast<const ulonglong2 *>(tab + kInvOmega * N), p,
                              [&](uint32_t k) { return poly[swz<true>(k)]; });
}

template <int LOGN>
__global__ void __launch_bounds__(kExtractThreads, 4) decrypt_poly_kernel(const uint64_t *__restrict__ ct,
                                                              const uint64_t *__restrict__ sk,
                                                              const uint64_t *__restrict__ sks,
                                                              const uint64_t *__restrict__ tables, uint32_t m,
                                                              const DevModuli dm, uint64_t *__restrict__ res) {
  constexpr uint32_t N = 1u << LOGN, shift = 32 - LOGN;
  extern __shared__ __align__(16) uint64_t poly[];
  const uint32_t c = blockIdx.y;
  const uint64_t j = blockIdx.x, p = dm.p[c];
  const uint64_t *tab = tables + (uint64_t)c * kTableSlots * N;
  decrypt_poly<LOGN>(poly, ct + (j * 2 * m + c) * N, ct + (j * 2 * m + m + c) * N, sk + (uint64_t)c * N,
                     sks + (uint64_t)c * N, tab, p);
  const ulonglong2 *iphi = reinterpret_cast<const ulonglong2 *>(tab + kInvPhi * N);
  uint64_t *o = res + (j * m + c) * N;
  // In output order (coalesced global loads and stores); the bit reversal is its own
  // inverse, so output k reads transform slot brev(k).
  for (uint32_t k = threadIdx.x; k < N; k += blockDim.x) {
    const ulonglong2 f = __ldg(iphi + k);
    o[k] = shoup_mul(poly[swz<true>(__brev(k) >> shift)], f.x, f.y, p);
  }
}

// One more modulus of the mixed radix: x += M_C * v with v in [0, p_C) such that x = residue
// mod p_C.  Before it x < p_0*...*p_{C-1} < 2^(61C) has C limbs (as M_C), after it C + 1.
template <int C, int M>
__device__ __forceinline__ void lift_step(uint64_t (&x)[M], uint64_t residue, const LiftConsts &lc, const DevModuli &dm) {
  const uint64_t p = dm.p[C], np = 0 - p;
  const uint64_t r = mod_word(residue, p, np);
  if constexpr (C == 0) {
    x[0] = r;
  } else {
    uint64_t t = r + p - limbs_mod_fast<C>(x, p, np, (uint32_t)dm.shoup_delta[C]);
    t = t >= p ? t - p : t;
    const uint64_t v = shoup_mul(t, lc.inv[C], lc.inv_shoup[C], p);
    unsigned __int128 carry = 0;
#pragma unroll
    for (int l = 0; l < C; l++) {
      const unsigned __int128 s = (unsigned __int128)lc.M[C][l] * v + x[l] + carry;
      x[l] = (uint64_t)s;
      carry = s >> 64;
    }
    x[C] = (uint64_t)carry;
  }
}

// The plaintext value of one coefficient from its M residues (residue(c), any 64-bit words):
// mixed radix, centred, cut to `bits` bits.
template <int M, class Residue>
__device__ __forceinline__ unsigned __int128 lift(uint32_t bits, const LiftConsts &lc, const DevModuli &dm,
                                                  Residue residue) {
  uint64_t x[M];
  lift_step<0>(x, residue(0), lc, dm);
  if constexpr (M > 1) lift_step<1>(x, residue(1), lc, dm);
  if constexpr (M > 2) lift_step<2>(x, residue(2), lc, dm);
  if constexpr (M > 3) lift_step<3>(x, residue(3), lc, dm);
  // centred: x - P when 2x > P
  int cmp = 0;  // sign of 2x - P (x < P < 2^(61M): 2x fits the limbs)
#pragma unroll
  for (int l = M - 1; l >= 0; l--) {
    const uint64_t x2 = (x[l] << 1) | (l ? x[l > 0 ? l - 1 : 0] >> 63 : 0);
    if (cmp == 0 && x2 != lc.P[l]) cmp = x2 > lc.P[l] ? 1 : -1;
  }
  unsigned __int128 v = x[0], top = lc.P[0];
  if constexpr (M > 1) {
    v |= (unsigned __int128)x[1] << 64;
    top |= (unsigned __int128)lc.P[1] << 64;
  }
  if (cmp > 0) v -= top;  // below 2^128: for one modulus the difference's high word is all ones
  return v & ((((unsigned __int128)1) << bits) - 1);
}

// lift() for a modulus count known at run time (1..kMaxLiftModuli).
template <class Residue>
__device__ __forceinline__ unsigned __int128 lift_any(uint32_t m, uint32_t bits, const LiftConsts &lc,
                                                      const DevModuli &dm, Residue residue) {
  switch (m) {
    case 1: return lift<1>(bits, lc, dm, residue);
    case 2: return lift<2>(bits, lc, dm, residue);
    case 3: return lift<3>(bits, lc, dm, residue);
    default: return lift<4>(bits, lc, dm, residue);
  }
}

__global__ void __launch_bounds__(256) lift_pack_kernel(const uint64_t *__restrict__ res, uint64_t nct, uint32_t N,
                                                        uint32_t m, uint32_t bits, const LiftConsts lc,
                                                        const DevModuli dm, unsigned long long *__restrict__ out) {
  const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (t >= nct * N) return;
  const uint64_t j = t / N, i = t % N;
  const unsigned __int128 v = lift_any(m, bits, lc, dm, [&](uint32_t c) { return res[(j * m + c) * N + i]; });
  // append at bit offset i*bits of ciphertext j's plaintext (bits*N/64 words per ciphertext)
  const uint64_t pos = (uint64_t)i * bits, words = (uint64_t)bits * N / 64;
  unsigned long long *w = out + j * words + (pos >> 6);
  const uint32_t sh = (uint32_t)(pos & 63);
  const unsigned __int128 lo = v << sh;  // bits [sh, sh+bits) of a 192-bit window
  const uint64_t w0 = (uint64_t)lo, w1 = (uint64_t)(lo >> 64);
  const uint64_t w2 = sh ? (uint64_t)(v >> (128 - sh)) : 0;
  if (w0) atomicOr(w, (unsigned long long)w0);
  if (w1) atomicOr(w + 1, (unsigned long long)w1);
  if (w2) atomicOr(w + 2, (unsigned long long)w2);
}

// Decryption, lift and packing of one ciphertext per CTA: the moduli one after another, their
// residues kept in shared memory (the last one's in registers), then each thread packs whole
// words of the plaintext.  For many ciphertexts: the residues never reach HBM and no word is
// written twice (decrypt_poly_kernel and lift_pack_kernel move 2 * m * N words more per
// ciphertext, zero the output first and update it atomically).  Rows of `keep`: m - 1, and as
// many as a value has words.  The output is `limit` bytes long.
template <int LOGN>
__global__ void __launch_bounds__(kExtractThreads, 4) extract_kernel(const uint64_t *__restrict__ ct,
                                                         const uint64_t *__restrict__ sk,
                                                         const uint64_t *__restrict__ sks,
                                                         const uint64_t *__restrict__ tables, uint32_t m, uint32_t bits,
                                                         const LiftConsts lc, const DevModuli dm,
                                                         uint64_t *__restrict__ out, uint64_t limit) {
  constexpr uint32_t N = 1u << LOGN, shift = 32 - LOGN;
  extern __shared__ __align__(16) uint64_t poly[];
  uint64_t *keep = poly + N;
  const uint64_t j = blockIdx.x;
  for (uint32_t c = 0; c < m; c++) {
    const uint64_t p = dm.p[c];
    if (c + 1 < m) {  // the next modulus' rows on their way to L2
      for (uint32_t i = threadIdx.x * 16; i < N; i += kExtractThreads * 16) {
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(ct + (j * 2 * m + c + 1) * N + i));
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(ct + (j * 2 * m + m + c + 1) * N + i));
      }
    }
    decrypt_poly<LOGN>(poly, ct + (j * 2 * m + c) * N, ct + (j * 2 * m + m + c) * N, sk + (uint64_t)c * N,
                       sks + (uint64_t)c * N, tables + (uint64_t)c * kTableSlots * N, p);
    const ulonglong2 *iphi = reinterpret_cast<const ulonglong2 *>(tables + ((uint64_t)c * kTableSlots + kInvPhi) * N);
    for (uint32_t k = threadIdx.x; k < N; k += blockDim.x) {
      const ulonglong2 f = __ldg(iphi + k);
      const uint64_t r = shoup_mul(poly[swz<true>(__brev(k) >> shift)], f.x, f.y, p);
      if (c + 1 < m) {
        keep[c * N + k] = r;
        continue;
      }
      const unsigned __int128 v = lift_any(m, bits, lc, dm, [&](uint32_t i) { return i + 1 < m ? keep[i * N + k] : r; });
      keep[k] = (uint64_t)v;
      if (bits > 64) keep[N + k] = (uint64_t)(v >> 64);
    }
    __syncthreads();
  }
  // Word w of the plaintext: bits 64w .. of the values, `bits` each.
  const uint32_t words = bits * N / 64;
  for (uint32_t w = threadIdx.x; w < words; w += blockDim.x) {
    const uint32_t from = w * 64;
    uint32_t i = from / bits;
    int at = (int)(i * bits) - (int)from;  // position of value i in the word
    uint64_t v = 0;
    for (; at < 64; i++, at += (int)bits) {
      const uint64_t lo = keep[i], hi = bits > 64 ? keep[N + i] : 0;
      if (at >= 0) v |= lo << at;
      else if (at > -64) v |= lo >> -at | hi << (64 + at);
      else v |= hi >> (-at - 64);
    }
    const uint64_t byte = (j * words + w) * 8;
    if (byte + 8 <= limit) {
      out[j * words + w] = v;
    } else {
      for (uint32_t k = 0; k < 8; k++)
        if (byte + k < limit) reinterpret_cast<uint8_t *>(out)[byte + k] = (uint8_t)(v >> (8 * k));
    }
  }
}

// Limb helpers on the host.
void limbs_mul_small(uint64_t *M, uint64_t v) {
  unsigned __int128 carry = 0;
  for (int i = 0; i < kLimbs; i++) {
    const unsigned __int128 t = (unsigned __int128)M[i] * v + carry;
    M[i] = (uint64_t)t;
    carry = t >> 64;
  }
}

uint64_t limbs_mod_host(const uint64_t *x, uint64_t p) {
  unsigned __int128 r = 0;
  for (int i = kLimbs - 1; i >= 0; i--) r = ((r << 64) | x[i]) % p;
  return (uint64_t)r;
}

uint64_t powmod_host(uint64_t a, uint64_t e, uint64_t p) {
  uint64_t r = 1;
  a %= p;
  while (e) {
    if (e & 1) r = (uint64_t)(((unsigned __int128)r * a) % p);
    a = (uint64_t)(((unsigned __int128)a * a) % p);
    e >>= 1;
  }
  return r;
}

// Ciphertexts decrypted at level lvl: PIRReplyExtraction_internal::extractReply's float
// arithmetic (…_internal.cpp:50-58).
uint64_t extract_count(uint64_t agg_bytes, uint32_t lvl, uint32_t bits, uint32_t N, uint32_t m) {
  const float abs_bytes = (float)((uint64_t)bits * N / 8), ct_bytes = (float)(16ull * m * N);
  uint64_t nbr = (uint64_t)std::ceil((float)agg_bytes / abs_bytes);
  for (uint32_t i = 1; i < lvl; i++) {
    const float t = (float)nbr * ct_bytes;
    nbr = (uint64_t)std::ceil(t / abs_bytes);
  }
  return nbr;
}

int status_of(cudaError_t e) {
  if (e == cudaSuccess) return XPIR_B200_OK;
  (void)cudaGetLastError();
  if (e == cudaErrorMemoryAllocation) return XPIR_B200_ERR_NOMEM;
  return XPIR_B200_ERR_CUDA;
}

}  // namespace
}  // namespace xpir

using namespace xpir;

extern "C" uint64_t xpir_b200_extract_count(uint64_t aggregated_bytes, uint32_t level, uint32_t bits_per_coeff,
                                            uint32_t poly_degree, uint32_t nb_moduli) {
  if (level == 0 || bits_per_coeff == 0 || poly_degree == 0 || nb_moduli == 0) return 0;
  return extract_count(aggregated_bytes, level, bits_per_coeff, poly_degree, nb_moduli);
}

extern "C" int xpir_b200_extract(xpir_b200_ctx *ctx, const uint64_t *secret_key, uint32_t d, uint32_t bits_per_coeff,
                                 uint64_t aggregated_bytes, const void *replies, uint64_t nb_replies,
                                 int replies_on_device, void *plaintext, uint64_t capacity_bytes, int out_on_device) {
  if (!ctx || !secret_key || !replies || !plaintext || d == 0 || d > XPIR_B200_MAX_LEVELS || aggregated_bytes == 0)
    return XPIR_B200_ERR_ARG;
  const ParamSet &ps = ctx->ps;
  const uint32_t N = ps.N, m = ps.m, bits = bits_per_coeff;
  if (m > kMaxLiftModuli || bits == 0 || bits >= 128 || bits >= 61 * m || (uint64_t)bits * N % 64 != 0)
    return XPIR_B200_ERR_ARG;
  if (capacity_bytes < aggregated_bytes) return XPIR_B200_ERR_ARG;
  for (uint32_t c = 0; c < m; c++) {  // the lift's reductions (mod_word, mod_two_words) assume these
    const uint64_t p = ps.mod[c].p;
    if (p <= (1ull << 60) || p >= (1ull << 61) || (1ull << 61) - p >= (1ull << 57) || !shoup_factor_ok(p))
      return XPIR_B200_ERR_ARG;
  }
  const uint64_t top = extract_count(aggregated_bytes, d, bits, N, m);
  if (nb_replies < top) return XPIR_B200_ERR_ARG;
  const uint64_t mN = (uint64_t)m * N, ct_words = 2 * mN, abs_words = (uint64_t)bits * N / 64;

  // Host constants of the mixed-radix lift (the key's Shoup factors are computed on the device).
  LiftConsts lc;
  memset(&lc, 0, sizeof(lc));
  lc.P[0] = 1;
  for (uint32_t c = 0; c < m; c++) {
    const uint64_t p = ps.mod[c].p;
    memcpy(lc.M[c], lc.P, sizeof(lc.P));
    lc.inv[c] = c ? powmod_host(limbs_mod_host(lc.P, p), p - 2, p) : 1;
    lc.inv_shoup[c] = (uint64_t)(((unsigned __int128)lc.inv[c] << 64) / p);
    limbs_mul_small(lc.P, p);
  }
  const DevModuli dm = make_dev_moduli(ps);

  std::lock_guard<std::mutex> lock(ctx->mu);
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return status_of(e);
  cudaStream_t st = ctx->stream;
  uint64_t *d_sk = nullptr, *d_sks = nullptr, *d_in = nullptr, *d_res = nullptr, *d_out = nullptr;
  auto cleanup = [&]() {
    cudaFreeAsync(d_sk, st);
    cudaFreeAsync(d_sks, st);
    cudaFreeAsync(d_in, st);
    cudaFreeAsync(d_res, st);
    cudaFreeAsync(d_out, st);
  };
  e = pool_allocate(ctx, (void **)&d_sk, mN * 8);
  if (e == cudaSuccess) e = pool_allocate(ctx, (void **)&d_sks, mN * 8);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_sk, secret_key, mN * 8, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) {
    e = launch_key_shoup(d_sk, d_sks, N, m, dm, st);
    ctx->launches++;
  }
  const uint64_t *level_in = (const uint64_t *)replies;
  if (e == cudaSuccess && !replies_on_device) {
    e = pool_allocate(ctx, (void **)&d_in, top * ct_words * 8);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(d_in, replies, top * ct_words * 8, cudaMemcpyHostToDevice, st);
    level_in = d_in;
  }
  bool delivered = false;  // the last level's kernel wrote the caller's buffer itself
  for (uint32_t lvl = d; lvl >= 1 && e == cudaSuccess; lvl--) {
    const uint64_t nbr = extract_count(aggregated_bytes, lvl, bits, N, m);
    uint64_t *res = nullptr, *out = nullptr;
    // The plaintext (plus slack for the last value's straddling word) is read by the next
    // level as its ciphertexts, or copied to the caller: size it for both.  The count's float
    // arithmetic can fall a few bytes short of a long element; those bytes are zero.
    const uint64_t used_words = lvl > 1 ? extract_count(aggregated_bytes, lvl - 1, bits, N, m) * ct_words
                                        : (aggregated_bytes + 7) / 8;
    const uint64_t out_words = std::max<uint64_t>(nbr * abs_words + 3, used_words);
    if (nbr > 0x7fffffffull) e = cudaErrorInvalidValue;
    const uint32_t rows = std::max(m - 1, bits > 64 ? 2u : 1u);
    const size_t fused_smem = (size_t)(1 + rows) * N * 8;
    if (nbr >= kFusedCiphertexts && fused_smem <= kFusedSmem) {
      // Only the words past the plaintext need zeroing, and the last level's plaintext can go
      // straight to an aligned device buffer, unless that overlaps the ciphertexts other CTAs
      // may still be reading (extraction in place).
      delivered = lvl == 1 && out_on_device && ((uintptr_t)plaintext & 7) == 0 &&
                  !overlap(level_in, nbr * ct_words * 8, plaintext, aggregated_bytes);
      uint64_t *dst = (uint64_t *)plaintext, limit = aggregated_bytes;
      if (!delivered) {
        if (e == cudaSuccess) e = pool_allocate(ctx, (void **)&out, out_words * 8);
        if (e == cudaSuccess) e = cudaMemsetAsync(out + nbr * abs_words, 0, (out_words - nbr * abs_words) * 8, st);
        dst = out;
        limit = out_words * 8;
      }
      if (e == cudaSuccess) {
#define XPIR_EXTRACT(L)                                                                                            \
  {                                                                                                                \
    e = allow_max_dynamic_smem((const void *)extract_kernel<L>);                                                   \
    if (e == cudaSuccess) {                                                                                        \
      extract_kernel<L><<<(unsigned)nbr, kExtractThreads, fused_smem, st>>>(level_in, d_sk, d_sks, ctx->d_tables, m, bits, lc, \
                                                              dm, dst, limit);                                     \
      e = cudaGetLastError();                                                                                      \
    }                                                                                                              \
  }
        XPIR_BY_DEGREE(ps.log_n, XPIR_EXTRACT)
        ctx->launches++;
      }
      const uint64_t held = nbr * abs_words * 8;
      if (e == cudaSuccess && delivered && held < aggregated_bytes)
        e = cudaMemsetAsync((char *)plaintext + held, 0, aggregated_bytes - held, st);
    } else {
      if (e == cudaSuccess) e = pool_allocate(ctx, (void **)&res, nbr * mN * 8);
      if (e == cudaSuccess) e = pool_allocate(ctx, (void **)&out, out_words * 8);
      if (e == cudaSuccess) e = cudaMemsetAsync(out, 0, out_words * 8, st);
      if (e == cudaSuccess) {
#define XPIR_DECRYPT(L)                                                                                           \
  {                                                                                                               \
    e = allow_max_dynamic_smem((const void *)decrypt_poly_kernel<L>);                                             \
    if (e == cudaSuccess) {                                                                                       \
      decrypt_poly_kernel<L><<<dim3((unsigned)nbr, m), kExtractThreads, N * 8, st>>>(level_in, d_sk, d_sks, ctx->d_tables, m, \
                                                                        dm, res);                                \
      e = cudaGetLastError();                                                                                     \
    }                                                                                                             \
  }
        XPIR_BY_DEGREE(ps.log_n, XPIR_DECRYPT)
      }
      if (e == cudaSuccess) {
        const uint64_t threads = nbr * N;
        lift_pack_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(res, nbr, N, m, bits, lc, dm,
                                                                             (unsigned long long *)out);
        e = cudaGetLastError();
        ctx->launches += 2;
      }
      cudaFreeAsync(res, st);
    }
    // This level's plaintext is the next level's ciphertexts.
    if (d_out) cudaFreeAsync(d_out, st);
    d_out = out;
    level_in = out;
  }
  if (e == cudaSuccess && !delivered)
    e = cudaMemcpyAsync(plaintext, d_out, aggregated_bytes,
                        out_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, st);
  cleanup();
  const cudaError_t se = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = se;
  return status_of(e);
}
