// Database import on the GPU: aggregation, bit split, CRT, phi-twist and the lazy
// decimation-in-frequency NTT, fused in one kernel per (aggregated element, poly, modulus).
//
// Reference path (crypto/NFLlib.cpp:375-401, 672-916; crypto/NFLlib.hpp:450-537, 597-608;
// pir/replyGenerator/PIRReplyGeneratorNFL_internal.cpp:79-158).  The same kernel performs
// the re-import of level replies between recursion levels (…NFL_internal.cpp:599-626):
// the P reply ciphertexts of an element are one contiguous little-endian bit stream.
//
// HBM layout of the output: [element][poly][modulus][coefficient] u64, values in [0, 2p).
#include <cuda_runtime.h>
#include <algorithm>
#include <stdint.h>

#include "kernels.h"
#include "modarith.cuh"
#include "ntt.cuh"

namespace xpir {

DevModuli make_dev_moduli(const ParamSet &ps) {
  DevModuli d{};
  for (uint32_t c = 0; c < ps.m; c++) {
    d.p[c] = ps.mod[c].p;
    d.shoup_k[c] = ps.mod[c].shoup_k;
    d.shoup_delta[c] = ps.mod[c].shoup_delta;
    for (int t = 0; t < 4; t++) {
      d.crt[c][t] = ps.mod[c].crt[t];
      d.crt_shoup[c][t] = ps.mod[c].crt_shoup[t];
    }
  }
  return d;
}

namespace {

struct ImportShape {
  uint32_t N, m, b, nsub;
  uint32_t P, active;    // element s of CTA poly (u, j): (u / active) * per_row + u % active
  uint64_t per_row;
  uint64_t polys;        // polys to import: rows * active * P
  uint64_t total_bytes;  // bytes of one aggregated element (alpha * element_bytes)
  uint32_t stage_words;  // u64 words of staged input per poly (even)
};

// Byte i of aggregated element s, following the reference's reused import buffer: a
// short last group (r < alpha real elements) reads its last real slot r-1 and slots up
// to alpha-2 as zeros, and slot alpha-1 as the previous group's last element (zeros for
// the first group).  See oracle xo_aggregate and pir/dbhandlers/DBHandler.cpp:3-26.
__device__ __forceinline__ uint8_t agg_byte(const AggSource &src, uint64_t s, uint64_t i, uint64_t real) {
  const uint64_t slot = i / src.element_bytes, off = i - slot * src.element_bytes;
  const uint64_t first = s * src.alpha;
  uint64_t elem;
  if (real == src.alpha) {
    elem = first + slot;
  } else if (slot + 1 < real) {
    elem = first + slot;
  } else if (slot + 1 == src.alpha) {
    if (s == 0) return 0;
    elem = first - 1;
  } else {
    return 0;
  }
  return src.base[elem * src.element_stride + off];
}


// Bits pos .. of the staged little-endian words, cut by the masks of the two result halves.
__device__ __forceinline__ uint64_t staged_bits(const uint32_t *st, uint32_t pos, uint32_t mask_lo, uint32_t mask_hi) {
  const uint32_t *w = st + (pos >> 5);
  const uint32_t w0 = w[0], w1 = w[1], w2 = w[2];
  return (uint64_t)(__funnelshift_r(w1, w2, pos) & mask_hi) << 32 | (__funnelshift_r(w0, w1, pos) & mask_lo);
}
__device__ __forceinline__ uint32_t low_mask(int bits) { return bits >= 32 ? ~0u : bits <= 0 ? 0u : (1u << bits) - 1; }

// Eight bytes of a contiguous element from byte `at` on; bytes past `bytes` are zero.
__device__ __forceinline__ uint64_t flat_word(const uint8_t *base, uint64_t at, uint64_t bytes) {
  const uint8_t *p = base + at;
  const uint32_t off = (uint32_t)(uintptr_t)p & 7;
  const uint64_t *w = (const uint64_t *)(p - off);
  if (off == 0 && at + 8 <= bytes) return w[0];
  // Between two aligned words that both lie in the element.
  if (off && at >= off && at - off + 16 <= bytes) return w[0] >> (8 * off) | w[1] << (64 - 8 * off);
  uint64_t v = 0;
  for (uint32_t q = 0; q < 8; q++)
    if (at + q < bytes) v |= (uint64_t)p[q] << (8 * q);
  return v;
}

// One CTA imports one poly of one modulus: grid: x = poly, y = modulus; T threads.  ALIAS: one group of coefficients per thread
// (T = N/8), so that the transform's buffer can take the place of the staged input once
// every thread holds its coefficients.  Dynamic smem: the staged words and the polys.
template <int LOGN, int T, bool ALIAS, int MINB>
__global__ void __launch_bounds__(T, MINB) import_kernel(const AggSource src, const ImportShape sh, const DevModuli dm,
                                                         const uint64_t *__restrict__ tables,
                                                         uint64_t *__restrict__ out) {
  constexpr uint32_t N = 1u << LOGN;
  static_assert(!ALIAS || T == (int)N / 8, "aliasing needs one group per thread");
  extern __shared__ __align__(16) uint64_t smem[];
  uint64_t *stage = smem;
  uint64_t *poly = ALIAS ? smem : smem + sh.stage_words;
  const uint32_t c = blockIdx.y;
  const uint64_t p = dm.p[c];
  const uint32_t u = blockIdx.x / sh.P, j = blockIdx.x - u * sh.P, row = u / sh.active;
  const uint64_t s = row * sh.per_row + (u - row * sh.active);
  // Stage the bytes of this poly's bit range, from an 8-byte aligned start.
  const uint64_t bit0 = (uint64_t)j * N * sh.b, byte0 = (bit0 >> 3) & ~7ull;
  const uint64_t first = s * src.alpha;
  const uint64_t real = (first + src.alpha <= src.nb_elements) ? src.alpha : src.nb_elements - first;
  const bool flat = (real == src.alpha) && (src.alpha == 1 || src.element_stride == src.element_bytes);
  const uint8_t *base = src.base + first * src.element_stride;
  uint64_t any = 0;
  for (uint32_t w = threadIdx.x; w < sh.stage_words; w += T) {
    const uint64_t at = byte0 + 8ull * w;
    uint64_t v = 0;
    if (at < sh.total_bytes) {
      if (flat) {
        v = flat_word(base, at, sh.total_bytes);
      } else {
        for (uint32_t k = 0; k < 8; k++)
          if (at + k < sh.total_bytes) v |= (uint64_t)agg_byte(src, s, at + k, real) << (8 * k);
      }
    }
    stage[w] = v;
    any |= v;
  }
  if (!__syncthreads_or(any != 0) && threadIdx.x == 0 && c == 0 && real == src.alpha && src.zero_seen &&
      atomicAdd(src.zero_seen, 1) + 1 == kZeroPolys)
    *(volatile int *)src.zero_hint = 1;

  // Coefficient k, twisted by phi^k: b <= 56 one chunk per coefficient; b > 56 sub-chunks
  // of 56 bits combined per modulus as sum_t mulmod(s_t, 2^(56t)) without a final reduction
  // (the first is below p and stays as it is).
  const uint64_t *tab = tables + (uint64_t)c * kTableSlots * N;
  const ulonglong2 *phi = reinterpret_cast<const ulonglong2 *>(tab + kPhi * N);
  const uint32_t *st = reinterpret_cast<const uint32_t *>(stage);
  const uint32_t b = sh.b, nsub = sh.nsub, rel0 = (uint32_t)(bit0 - 8 * byte0);
  const int first_bits = nsub == 1 ? (int)b : 56, last_bits = (int)b - 56 * (int)(nsub - 1);
  const uint32_t mask_lo = low_mask(first_bits), mask_hi = low_mask(first_bits - 32);
  auto coefficient = [&](uint32_t k) -> uint64_t {
    const ulonglong2 f = __ldg(phi + k);
    const uint32_t pos = rel0 + k * b;
    uint64_t x = staged_bits(st, pos, mask_lo, mask_hi);
    if (nsub == 1 && b <= 32) return shoup_mul_small((uint32_t)x, f.x, f.y, p);
    for (uint32_t t = 1; t < nsub; t++) {
      const int bits = t + 1 < nsub ? 56 : last_bits;
      const uint64_t sub = staged_bits(st, pos + 56 * t, low_mask(bits), low_mask(bits - 32));
      x += bits <= 32 ? shoup_mul_small((uint32_t)sub, dm.crt[c][t], dm.crt_shoup[c][t], p)
                      : shoup_mul(sub, dm.crt[c][t], dm.crt_shoup[c][t], p);
    }
    return shoup_mul(x, f.x, f.y, p);
  };
  ntt_lazy<LOGN, ALIAS>(poly, reinterpret_cast<const ulonglong2 *>(tab + kOmega * N), p, coefficient);

  // Coalesced 16-byte stores; swz(2t+1) == swz(2t) ^ 1.
  ulonglong2 *o = reinterpret_cast<ulonglong2 *>(out + ((s * sh.P + j) * sh.m + c) * (uint64_t)N);
  for (uint32_t t = threadIdx.x; t < N / 2; t += T) {
    const uint32_t at = swz(2 * t);
    o[t] = make_ulonglong2(poly[at], poly[at ^ 1]);
  }
}

// The import of an all-zero bit stream, broadcast: every coefficient chunk is 0, so the
// twisted coefficients are 0 and the lazy NTT leaves one fixed poly per modulus (values
// 0 and p).  Each CTA computes it for modulus blockIdx.y in shared memory, then writes it
// to its share of the `count` known-zero polys t (element row * per_row + active +
// (t / P) % (per_row - active) of row t / (P * (per_row - active)), poly t % P).
template <int LOGN>
__global__ void __launch_bounds__(512) import_zero_fill_kernel(const ImportShape sh, const DevModuli dm,
                                                               const uint64_t *__restrict__ tables,
                                                               uint64_t *__restrict__ out, uint64_t count) {
  constexpr uint32_t N = 1u << LOGN;
  extern __shared__ __align__(16) uint64_t smem[];
  const uint32_t c = blockIdx.y;
  const uint64_t p = dm.p[c];
  const uint64_t *tab = tables + (uint64_t)c * kTableSlots * N;
  const ulonglong2 *phi = reinterpret_cast<const ulonglong2 *>(tab + kPhi * N);
  auto coefficient = [&](uint32_t k) -> uint64_t {
    const ulonglong2 f = __ldg(phi + k);
    return shoup_mul(0, f.x, f.y, p);
  };
  ntt_lazy<LOGN, false>(smem, reinterpret_cast<const ulonglong2 *>(tab + kOmega * N), p, coefficient);
  const uint64_t zeros = sh.per_row - sh.active;
  for (uint64_t t = blockIdx.x; t < count; t += gridDim.x) {
    const uint64_t u = t / sh.P, j = t - u * sh.P;
    const uint64_t row = u / zeros, s = row * sh.per_row + sh.active + (u - row * zeros);
    ulonglong2 *o = reinterpret_cast<ulonglong2 *>(out + ((s * sh.P + j) * sh.m + c) * (uint64_t)N);
    for (uint32_t i = threadIdx.x; i < N / 2; i += blockDim.x) {
      const uint32_t at = swz(2 * i);
      o[i] = make_ulonglong2(smem[at], smem[at ^ 1]);
    }
  }
}

template <int LOGN, int T, bool ALIAS, int MINB>
cudaError_t launch_import_n(const AggSource &src, const ImportShape &sh, const DevModuli &dm, const uint64_t *tables,
                            uint64_t *out, cudaStream_t stream) {
  auto kern = import_kernel<LOGN, T, ALIAS, MINB>;
  const size_t words = ALIAS ? std::max(sh.stage_words, sh.N) : sh.stage_words + sh.N;
  kern<<<dim3((unsigned)sh.polys, sh.m), T, words * 8, stream>>>(src, sh, dm, tables, out);
  return cudaGetLastError();
}

typedef cudaError_t (*ImportFn)(const AggSource &, const ImportShape &, const DevModuli &, const uint64_t *, uint64_t *,
                                cudaStream_t);
struct ImportEntry {
  ImportFn import;
  const void *kernels[2];
};
#define XPIR_IMPORT(LOGN, T, ALIAS, MINB)                                                       \
  {                                                                                             \
    &launch_import_n<LOGN, T, ALIAS, MINB>, {                                                   \
      (const void *)import_kernel<LOGN, T, ALIAS, MINB>, (const void *)import_zero_fill_kernel<LOGN> \
    }                                                                                           \
  }
// By degree 512..8192; 64 registers and 32 warps per SM (16,000 polys of 2048: 348 us, with 80
// registers and 24 warps 369).  At 8192 a thread has two groups of coefficients.
const ImportEntry kImports[] = {
    XPIR_IMPORT(9, 64, true, 16),  XPIR_IMPORT(10, 128, true, 8),   XPIR_IMPORT(11, 256, true, 4),
    XPIR_IMPORT(12, 512, true, 2), XPIR_IMPORT(13, 512, false, 2),
};

template <int LOGN>
cudaError_t launch_zero_fill(const ImportShape &sh, const DevModuli &dm, const uint64_t *tables, uint64_t *out,
                             uint64_t count, unsigned blocks, cudaStream_t stream) {
  auto kern = import_zero_fill_kernel<LOGN>;
  kern<<<dim3(blocks, sh.m), ntt_threads(sh.N), (size_t)sh.N * 8, stream>>>(sh, dm, tables, out, count);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_import(const AggSource &src, uint64_t groups, uint64_t P, const ParamSet &ps,
                          const DevModuli &dm, const uint64_t *tables, uint64_t *out, cudaStream_t stream,
                          const ImportRows *rows, uint32_t *launches) {
  if (groups == 0 || P == 0) return cudaSuccess;
  const ImportRows r = rows ? *rows : ImportRows{1, groups, groups};
  if (r.rows == 0 || r.per_row == 0 || r.rows * r.per_row != groups || r.active > r.per_row)
    return cudaErrorInvalidValue;
  const uint64_t computed = r.rows * r.active, zero_polys = r.rows * (r.per_row - r.active) * P;
  if (computed * P > 0x7fffffffull || P > 0x7fffffffull) return cudaErrorInvalidValue;
  ImportShape sh;
  sh.N = ps.N;
  sh.m = ps.m;
  sh.b = ps.b;
  sh.nsub = (ps.b + 55) / 56;
  sh.P = (uint32_t)P;
  sh.per_row = r.per_row;
  sh.active = (uint32_t)r.active;
  sh.polys = computed * P;
  sh.total_bytes = (uint64_t)src.alpha * src.element_bytes;
  // bits of one poly plus the in-word offset, rounded up, plus spare words for the
  // three-half-word reads of staged_bits; even, so that the polys stay 16-byte aligned
  sh.stage_words = (uint32_t)(((64 + (uint64_t)ps.N * ps.b + 63) / 64 + 3) & ~1ull);
  if (computed > 0) {
    const cudaError_t e = kImports[ps.log_n - 9].import(src, sh, dm, tables, out, stream);
    if (e != cudaSuccess) return e;
    if (launches) (*launches)++;
  }
  if (zero_polys > 0 && r.fill) {
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    // About four CTAs per SM over all moduli: each computes the constant poly once.
    const uint64_t per_mod = std::max<uint64_t>(1, 4ull * (uint64_t)sms / ps.m);
    const unsigned blocks = (unsigned)std::min<uint64_t>(zero_polys, per_mod);
#define XPIR_FILL(L) e = launch_zero_fill<L>(sh, dm, tables, out, zero_polys, blocks, stream)
    XPIR_BY_DEGREE(ps.log_n, XPIR_FILL)
    if (e != cudaSuccess) return e;
    if (launches) (*launches)++;
  }
  return cudaSuccess;
}

cudaError_t launch_zero_poly(const ParamSet &ps, const DevModuli &dm, const uint64_t *tables, uint64_t *out,
                             cudaStream_t stream) {
  ImportShape sh{};
  sh.N = ps.N;
  sh.m = ps.m;
  sh.P = 1;
  sh.per_row = 1;  // one element, known zero
  cudaError_t e = cudaSuccess;
#define XPIR_ZERO(L) e = launch_zero_fill<L>(sh, dm, tables, out, 1, 1, stream)
  XPIR_BY_DEGREE(ps.log_n, XPIR_ZERO)
  return e;
}

// Loads the import kernels on the current device (lazy module loading would otherwise do
// it, and reserve their device memory, at their first launch) and lets them take any amount
// of shared memory.
cudaError_t preload_import_kernels() {
  for (const ImportEntry &entry : kImports)
    for (const void *k : entry.kernels) {
      const cudaError_t e = allow_max_dynamic_smem(k);
      if (e != cudaSuccess) return e;
    }
  return cudaSuccess;
}

}  // namespace xpir
