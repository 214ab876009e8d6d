// Host-side check of the residue sums with an exact tail (xpir_b200/csrc/residue_sum.cuh),
// compiled with g++: whenever the sums vouch for a chain, it must equal the slot-by-slot
// chain of lazy Shoup multiply-accumulates; for words as queries and databases have them
// they must vouch for it, and for chains that pass 2^64 they must not.  Every split into
// runs that the kernels use (multiples of four slots) is tried on the same words.
#include <stdio.h>
#include <stdlib.h>

#include <random>
#include <vector>

#include "../../xpir_b200/csrc/params.h"
#include "../../xpir_b200/csrc/residue_sum.cuh"

using namespace xpir;
typedef std::vector<uint64_t> Words;

static uint64_t shoup_of(uint64_t y, uint64_t p) { return (uint64_t)(((unsigned __int128)y << 64) / p); }

// The chain slot by slot; *wrapped: a sum passed 2^64.
static uint64_t by_slot(const Words &x, const Words &y, uint64_t p, bool *wrapped) {
  uint64_t rop = 0;
  *wrapped = false;
  for (size_t i = 0; i < x.size(); i++) {
    const uint64_t t = shoup_lazy(x[i], y[i], shoup_of(y[i], p), p), w = rop + t;
    if (w < rop) *wrapped = true;
    rop = w >= p ? w - p : w;
  }
  return rop;
}

static long again = 0;

// The same chain as the kernels evaluate it; false: not vouched for.
static bool by_sums(const Words &x, const Words &y, uint64_t p, size_t runs, size_t step, uint64_t *out) {
  const ShoupConst sc = make_shoup_const(p);
  const uint32_t delta = (uint32_t)sc.delta, d64 = delta * 8;
  const uint64_t np = 0 - p;
  const size_t n = x.size();
  if (n < kTailSlots) return false;
  const size_t prefix = (n - kTailSlots) / step * step, len = (prefix / step + runs - 1) / runs * step;
  uint64_t r = 0;
  uint32_t above = 0;
  bool ok = true;
  for (size_t s0 = 0; s0 < prefix; s0 += len) {
    const size_t end = s0 + len < prefix ? s0 + len : prefix;
    SumAcc a;
    sum_clear(a, runs == 1 ? 0 : kBoundStart);
    for (size_t i = s0; i < end; i += 4) {
      uint32_t xs = 0, v[4];
      for (int k = 0; k < 4; k++) {
        ok &= y[i + k] < p;
        xs += (uint32_t)(x[i + k] >> 32);
        v[k] = sum_slot(a, x[i + k], sum_word(y[i + k], d64));
      }
      a.bound = sum_bound(a.bound + sum_block(xs), v);
      ok &= a.bound <= kBoundMax;
    }
    ok &= a.bound <= kBoundStart;
    r = (r + sum_residue(a, p, np, delta)) % p;
    above = sum_above(a.bound);
  }
  auto term = [&](size_t i) { return shoup_lazy(x[i], y[i], shoup_of(y[i], p), p); };
  ExactTail t{r, above, 0};
  for (size_t i = prefix; i < n; i++) {
    ok &= y[i] < p;
    tail_step(t, term(i), p);
  }
  ok &= !prefix || tail_in_range(t, kRunAbove);
  if (t.above) {
    const size_t from = prefix > kBackSlots ? prefix - kBackSlots : 0;
    t = ExactTail{0, 0, 0};
    if (from) {
      t = ExactTail{r, kMaxAbove, 0};
      for (size_t i = from; i < prefix; i++) t.rop = residue_before(t.rop, term(i), p);
    }
    for (size_t i = from; i < n; i++) tail_step(t, term(i), p);
    ok &= t.above == 0 && (!from || tail_in_range(t, kMaxAbove));
    again++;
  }
  *out = t.rop;
  return ok;
}

static long vouched = 0, refused = 0;

// must: +1 every split must vouch for it, -1 none may, 0 either.
static void check(const Words &x, const Words &y, uint64_t p, int must, const char *what) {
  bool wrapped;
  const uint64_t want = by_slot(x, y, p, &wrapped);
  for (size_t step : {4u, 8u})
    for (size_t runs : {1u, 2u, 3u, 7u}) {
      if (runs > 1 && x.size() / runs < kMinRunSlots + kTailSlots) continue;
      uint64_t got = 0;
      const bool ok = by_sums(x, y, p, runs, step, &got);
      (ok ? vouched : refused)++;
      if ((ok && (got != want || wrapped)) || (must > 0 && !ok) || (must < 0 && ok)) {
        printf("%s: p %llu, %zu slots, %zu runs: %s, got %llu want %llu%s\n", what, (unsigned long long)p, x.size(),
               runs, ok ? "vouched for" : "refused", (unsigned long long)got, (unsigned long long)want,
               wrapped ? " (wrapped)" : "");
        exit(1);
      }
    }
}

int main() {
  std::mt19937_64 rng(20250);
  for (unsigned c = 0; c < kMaxModuli; c++) {
    const uint64_t p = kModuli[c], d = (1ull << 61) - p;
    if (d >= (1ull << 23) || (p >> 32) != 0x1fffffffu) return 1;  // what the header assumes
    auto rx = [&] { return rng() % (2 * p); };
    auto ry = [&] { return rng() % p; };
    // a query word whose factor's fraction is just below one, and a database word near 2p,
    // so that every term they give lies above p
    uint64_t hy = 0, hx = 0;
    for (;;) {
      hy = ry();
      const unsigned __int128 z = (unsigned __int128)hy << 64;
      if ((uint64_t)(z % p) < p / 10 * 9) continue;
      bool found = false;
      for (int k = 0; k < 2000 && !found; k++) {
        hx = 2 * p - 1 - rng() % (p / 64);
        const uint64_t t = shoup_lazy(hx, hy, shoup_of(hy, p), p);
        found = t > p + p / 8;
      }
      if (found) break;
    }
    for (size_t n : {12u, 13u, 15u, 16u, 19u, 20u, 24u, 31u, 44u, 60u, 64u, 96u, 100u, 257u, 1000u, 4099u}) {
      for (int rep = 0; rep < (n > 1000 ? 4 : 40); rep++) {
        Words x(n), y(n);
        for (size_t i = 0; i < n; i++) x[i] = rx(), y[i] = ry();
        check(x, y, p, 1, "uniform words");
        Words a = x, b = y;
        for (size_t i = n / 2; i < n; i++) a[i] = 0;  // padding slots
        check(a, b, p, 1, "zero words at the end");
        a = x;
        for (size_t i = 0; i < n; i++)
          if (rng() % 2) a[i] = rng() % 2 ? p : 0;  // imports of zero bits scattered in the database
        check(a, b, p, 0, "words 0 and p");
        a = x;
        for (size_t i = 0; i + 60 < n; i++) a[i] = i % 2 ? p : a[i];
        check(a, b, p, 0, "every other word p up to the tail");
        a = x;
        for (size_t i = n / 4; i + 60 < n; i++) a[i] = p;
        check(a, b, p, 0, "a stretch of words p up to the tail");
        a.assign(n, p);
        check(a, b, p, 0, "all words p");
        a = x;
        for (size_t i = n - (n < 64 ? n / 2 : 40); i < n; i++) a[i] = p;
        check(a, b, p, 0, "words p in the tail");
        a = x;
        const uint64_t edge[] = {0, 1, 2, p - 1, p - 2, p / 2, 8, hy};
        const uint64_t edge_x[] = {0, 1, p - 1, p, p + 1, 2 * p - 1, 2 * p - 2, hx};
        for (size_t i = 0; i < n; i++) {
          if (rng() % 3 == 0) b[i] = edge[rng() % 8];
          if (rng() % 3 == 0) a[i] = edge_x[rng() % 8];
        }
        check(a, b, p, 0, "edge words");
        b = y;
        b[rng() % n] = p + rng() % 8;
        check(x, b, p, -1, "one word not below p");
        b = y;
        b[rng() % n] = rng() | (1ull << 61);
        check(x, b, p, -1, "one unreduced word");
        // a stretch of terms above p anywhere: its length decides whether a sum passes 2^64
        for (size_t len : {8u, 20u, 30u, 60u, 120u}) {
          if (len > n) continue;
          a = x, b = y;
          const size_t at = rng() % (n - len + 1);
          for (size_t i = at; i < at + len; i++) a[i] = hx, b[i] = hy;
          check(a, b, p, 0, "a stretch of terms above p");
        }
        a.assign(n, hx), b.assign(n, hy);
        check(a, b, p, n >= 100 ? -1 : 0, "only terms above p");
        a.assign(n, rx()), b.assign(n, ry());
        check(a, b, p, 0, "constant words");
      }
    }
  }
  printf("ok: %ld chains vouched for, %ld refused, %ld went back\n", vouched, refused, again);
  return 0;
}
