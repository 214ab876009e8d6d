// Host-side check of the short forms of the lazy Shoup product (xpir_b200/csrc/modarith.cuh):
// x below 2^32, and factor 1, against the general form for every modulus.
#include <stdio.h>

#include <random>

#include "../../xpir_b200/csrc/modarith.cuh"
#include "../../xpir_b200/csrc/params.h"

int main() {
  std::mt19937_64 rng(99);
  for (unsigned c = 0; c < xpir::kMaxModuli; c++) {
    const uint64_t p = xpir::kModuli[c], np = 0 - p;
    const uint64_t ys[] = {0, 1, 2, p - 1, p - 2, 1ull << 56, 1ull << 60, (1ull << 32) - 1, 1ull << 32};
    const uint64_t xs[] = {0, 1, 2, 0x7fffffff, 0x80000000, 0xfffffffe, 0xffffffff};
    for (int i = 0; i < 200000; i++) {
      const uint64_t y = i < 9 * 7 ? ys[i / 7] : rng() % p, w = rng();
      const uint32_t x = (uint32_t)(i < 9 * 7 ? xs[i % 7] : w);
      const uint64_t f = (uint64_t)(((unsigned __int128)y << 64) / p);
      const uint64_t one = (uint64_t)(((unsigned __int128)1 << 64) / p);
      if (xpir::shoup_lazy_small_np(x, y, f, np) != xpir::shoup_lazy(x, y, f, p) ||
          xpir::shoup_mul_small(x, y, f, p) != xpir::shoup_mul(x, y, f, p) ||
          xpir::shoup_lazy_one_np(w, np) != xpir::shoup_lazy(w, 1, one, p)) {
        printf("mismatch p=%llu x=%u y=%llu w=%llu\n", (unsigned long long)p, x, (unsigned long long)y,
               (unsigned long long)w);
        return 1;
      }
    }
  }
  printf("ok\n");
  return 0;
}
