// The reply chain of one output coefficient, evaluated without running it slot by slot.
//
// The chain (crypto/NFLlib.hpp:303-321) is, for words x < 2p of the database and y of the
// query,   rop = rop + t;  rop -= (rop >= p) ? p : 0   (mod 2^64),
// with t = x*y - hi(x*y')*p and y' = floor(y*2^64/p).  For y < p the term t is x*y mod p,
// plus p when the high product fell one short, and 0 <= t < p*(1 + x/2^64) < 1.25 p.  As
// long as no sum reaches 2^64 (just above 8p), three facts hold:
//
//   1. rop is (the sum of all x*y) mod p, plus j*p.  The residue can be summed in any order
//      and over any split of the slots.
//   2. j only grows while terms above p dominate:  with u(k) = t(k)/p - 1, a chain that was
//      below p before slot i satisfies rop < p*(1 + max over windows ending here of sum u).
//      So when every window's sum stays at or below 5.75 no sum reaches 2^64.
//   3. Two chains over the same terms that start a multiple of p apart come together:  the
//      difference loses one p at every slot where the lower one does not subtract.  Once
//      that happened as often as the difference at the start, both are equal.
//
// So the residue of all slots but the last kTailSlots comes from plain products (SumAcc),
// with a running upper bound of the windows' sums (fact 2), and only the last slots are run
// as the exact chain, from the residue and with the count of fact 3.  Whatever cannot be
// shown this way (a query word not below p, a bound that is exceeded, chains still apart at
// the end) is reported, and the caller runs the slot-by-slot kernel instead.
//
// The bound.  Write 2^64 = 8p + delta, D = 2^61 - p = delta/8 < 2^23, and halves
// x = x1*2^32 + x0, y = y1*2^32 + y0.  ys = 8y + q0 with q0 = floor(y1*64D / 2^32) is at
// most y' and at least y*2^64/p - 1.125.  With z = x*ys/2^64:  t/p = xy/p - hi(x*y') <=
// frac(z) + 1.125*x/2^64.  frac(z)'s top 32 bits are (8*w + x1*q0) mod 2^32, w the second
// 32-bit word of x*y, short by less than 2^-6 for the dropped x0*q0 and less than 2^-28 for
// the bits below.
#pragma once

#include <stdint.h>

#include "modarith.cuh"

namespace xpir {

// Slots of the exact tail, at least.  The lower chain has to fail to subtract once or twice
// in it, which about 7 of 16 terms make it do: 12 uniform terms miss that with probability
// near 1e-6.  A chain that does starts again kBackSlots earlier (about 1e-17 then).
constexpr uint32_t kTailSlots = 12;
constexpr uint32_t kBackSlots = 32;

// Units of the bound: 2^28 is p.  Every run of slots starts from kBoundStart, assumes at
// most kBoundStart from the slots before it, and must end at or below it; inside it may
// not pass kBoundMax.  The bound is only looked at every kBoundBlock slots, so a window can
// exceed it by the growth of two partial blocks, 2 * 3 * 0.25 p:  4.2 + 1.5 < 5.75.
constexpr int32_t kBoundOne = 1 << 28;
constexpr int32_t kBoundStart = (int32_t)(2.1 * (1 << 28));
constexpr int32_t kBoundMax = (int32_t)(4.2 * (1 << 28));
constexpr uint32_t kBoundBlock = 4;
// Slots per run below which a run need not return below kBoundStart.
constexpr uint32_t kMinRunSlots = 64;

// A 64-bit word mod p for XPIR's moduli (2^60 < p < 2^61, 2^61 - p < 2^57): q0 = w >> 61 and
// w - q0*p = (w mod 2^61) + q0*D < 2p.
XPIR_HD uint64_t mod_word(uint64_t w, uint64_t p, uint64_t np) {
  const uint64_t r = w + (w >> 61) * np;
  return r >= p ? r - p : r;
}

// h*2^64 + l mod p for h < p: h*2^64 mod p = h*2^64 - f*p with f = floor(h*2^64/p) (the
// Shoup factor of h), whose low word is f*(2^64 - p).
XPIR_HD uint64_t mod_two_words(uint64_t h, uint64_t l, uint64_t p, uint64_t np, uint32_t delta) {
  const uint64_t s = shoup_factor8_np(h, p, np, delta) * np + mod_word(l, p, np);  // < 2p
  return s >= p ? s - p : s;
}

// Sum of x*(8y) of one coefficient (one database column, one ciphertext half) and the bound
// of fact 2.  With 8y = e1*2^32 + e0 (below 2^64: the bound's fraction then needs no shift)
// the products x0*e0 and x1*e1 go to the words a (160 bits), the cross products to the words
// m (96 bits, from 2^32 on): the two sets keep every 32x32+64-bit multiply-add on one pair
// of words, with one carry chain each.
struct SumAcc {
  uint32_t a0, a1, a2, a3, a4, m0, m1, m2;
  uint32_t last;  // a1 + m0 after the previous slot
  int32_t bound;
};

XPIR_HD void sum_clear(SumAcc &a, int32_t bound) {
  a = SumAcc{};
  a.bound = bound;
}

// What the sums need of a query word.
struct SumWord {
  uint32_t e0, e1;  // 8y
  uint32_t q0;
};

XPIR_HD SumWord sum_word(uint64_t y, uint32_t d64) {
  SumWord w;
  const uint64_t e = y << 3;
  const uint32_t y1 = (uint32_t)(y >> 32);
  w.e0 = (uint32_t)e;
  w.e1 = (uint32_t)(e >> 32);
#if defined(__CUDA_ARCH__)
  w.q0 = __umulhi(y1, d64);
#else
  w.q0 = (uint32_t)(((uint64_t)y1 * d64) >> 32);
#endif
  return w;
}

// One slot's product; returns the top word of frac(z).  That word's w part is the change of
// a1 + m0 (the carry out of a0 may add one unit of 2^-32).
XPIR_HD uint32_t sum_slot(SumAcc &a, uint64_t x, const SumWord &w) {
  const uint32_t x0 = (uint32_t)x, x1 = (uint32_t)(x >> 32);
#if defined(__CUDA_ARCH__)
  asm("mad.lo.cc.u32 %0, %8, %10, %0;\n madc.hi.cc.u32 %1, %8, %10, %1;\n"
      "madc.lo.cc.u32 %2, %9, %11, %2;\n madc.hi.cc.u32 %3, %9, %11, %3;\n addc.u32 %4, %4, 0;\n"
      "mad.lo.cc.u32 %5, %8, %11, %5;\n madc.hi.cc.u32 %6, %8, %11, %6;\n addc.u32 %7, %7, 0;\n"
      "mad.lo.cc.u32 %5, %9, %10, %5;\n madc.hi.cc.u32 %6, %9, %10, %6;\n addc.u32 %7, %7, 0;\n"
      : "+r"(a.a0), "+r"(a.a1), "+r"(a.a2), "+r"(a.a3), "+r"(a.a4), "+r"(a.m0), "+r"(a.m1), "+r"(a.m2)
      : "r"(x0), "r"(x1), "r"(w.e0), "r"(w.e1));
#else
  // v*2^64 + carry-in added to the words r0, r1; returns the carry out
  auto add = [](uint32_t &r0, uint32_t &r1, uint64_t v, uint32_t carry) {
    const unsigned __int128 s = ((unsigned __int128)((uint64_t)r1 << 32 | r0)) + v + carry;
    r0 = (uint32_t)s;
    r1 = (uint32_t)(s >> 32);
    return (uint32_t)(s >> 64);
  };
  const uint32_t c = add(a.a0, a.a1, (uint64_t)x0 * w.e0, 0);
  a.a4 += add(a.a2, a.a3, (uint64_t)x1 * w.e1, c);
  a.m2 += add(a.m0, a.m1, (uint64_t)x0 * w.e1, 0);
  a.m2 += add(a.m0, a.m1, (uint64_t)x1 * w.e0, 0);
#endif
  const uint32_t now = a.a1 + a.m0;
  const uint32_t v = x1 * w.q0 + (now - a.last);
  a.last = now;
  return v;
}

// The bound's change over a block of kBoundBlock slots without the fractions: xs is the sum
// of the slots' x1 (each below 2^30).  Per slot 1.125*x1/2^32 - 1 and the slack of 2^-6 and
// 2^-20, in 2^-28.
XPIR_HD int32_t sum_block(uint32_t xs) {
  return (int32_t)((xs >> 4) + (xs >> 7)) +
         (int32_t)(kBoundBlock * ((1 << 22) + (1 << 8)) - kBoundBlock * (uint32_t)kBoundOne);
}

// The bound after a block, from the bound before it plus sum_block, and the block's fractions.
XPIR_HD int32_t sum_bound(int32_t before, const uint32_t v[kBoundBlock]) {
  const uint64_t sum = ((uint64_t)v[0] + v[1]) + ((uint64_t)v[2] + v[3]);
  const int32_t g = before + (int32_t)(uint32_t)(sum >> 4);
  return g > 0 ? g : 0;
}

// The residue of everything summed (p = 1 mod 8, so that an eighth of r mod p is the exact
// eighth of r + k*p for k = -r mod 8).
XPIR_HD uint64_t sum_residue(const SumAcc &a, uint64_t p, uint64_t np, uint32_t delta) {
  const uint64_t lo = (uint64_t)a.a1 << 32 | a.a0, hi = (uint64_t)a.a3 << 32 | a.a2;
  const uint64_t w0 = lo + ((uint64_t)a.m0 << 32);
  const uint64_t mid = ((uint64_t)a.m2 << 32 | a.m1) + (w0 < lo ? 1 : 0);  // m2 counts slots: no carry
  const uint64_t w1 = mid + hi;
  const uint64_t w2 = (uint64_t)a.a4 + (w1 < mid ? 1 : 0);
  const uint64_t r = mod_two_words(mod_two_words(w2, w1, p, np, delta), w0, p, np, delta);
  return (r + (uint64_t)((0u - (uint32_t)r) & 7u) * p) >> 3;
}

// Multiples of p that the chain may stand above its residue after a run that ended with
// this bound (fact 2, one partial block added).
XPIR_HD uint32_t sum_above(int32_t bound) { return (uint32_t)(kBoundOne + kBoundOne / 4 * 3 + bound) >> 28; }

// The exact chain: the lower of the candidate chains, and how many multiples of p the
// highest candidate still stands above it.
struct ExactTail {
  uint64_t rop;
  uint32_t above;
  uint32_t top;  // largest high word of rop seen
};

XPIR_HD void tail_step(ExactTail &s, uint64_t t, uint64_t p) {
  const uint64_t w = s.rop + t;
  const bool sub = w >= p;
  s.rop = sub ? w - p : w;
  if (!sub && s.above) s.above--;
  const uint32_t hi = (uint32_t)(s.rop >> 32);
  s.top = hi > s.top ? hi : s.top;
}

// Multiples of p that a chain can stand above its residue at the end of a run (kBoundStart)
// and inside one (kBoundMax), each with one partial block and the p below the window.
constexpr uint32_t kRunAbove = 3, kMaxAbove = 5;

// Whether no candidate can have reached 2^64 (just above 8p): the highest stands at most
// `most` * p above the lowest, a term is below 1.25 p, and the lowest stayed below 3p (3 + 3
// + 1.25) or 1.5 p (1.5 + 5 + 1.25).
XPIR_HD bool tail_in_range(const ExactTail &s, uint32_t most) {
  return s.top < (most <= kRunAbove ? 0x5fffffffu : 0x2fffffffu);
}

// A residue taken back by one slot's product.
XPIR_HD uint64_t residue_before(uint64_t r, uint64_t t, uint64_t p) {
  const uint64_t u = t >= p ? t - p : t;  // t < 1.25 p
  return r >= u ? r - u : r + p - u;
}

// `steps` slots whose database word is 0 (t = 0): each subtracts p while rop >= p.
XPIR_HD uint64_t zero_steps(uint64_t rop, uint64_t steps, uint64_t p) {
  while (steps && rop >= p) {
    rop -= p;
    steps--;
  }
  return rop;
}

}  // namespace xpir
