// shoup.cuh -- products by fixed factors (twiddles, scale factors) with a
// precomputed quotient, and the lazy ranges the butterflies keep.
//
// A product by a factor w known beforehand needs no Montgomery reduction:
// with q = floor(w 2^256 / p) stored beside w, the quotient of x w by p is
// floor(x q / 2^256), one or two too small at most, and the result is
// x w - quotient p, whose low 256 bits are all of it (Shoup's method; V. Shoup's
// NTL, and D. Harvey, "Faster arithmetic for number-theoretic transforms",
// 2014).  x w and quotient p are needed in their low halves only and x q in its
// high half, so the three cost 28 + 28 + 36 full 32x32->64 products, 16 low ones and
// four dot products of halves and bytes where a Montgomery product costs 136 full
// ones: 204 multiply-pipe slots of a 32-bit multiply-add against 272 (176 for
// BLS12-381-Fr, below).  The transforms are bound by that pipe.
//
// Which x: any value below 2^256 / 1.03 (lazy fields; below 2p for the others).  The
// quotient estimate drops the columns of x q below 6, worth less than 2^227, and
// takes column 6's products x_i q_(6-i) from the 16 top bits of x_i and the 8 top
// bits of q_(6-i), each low by less than (2^24 + 2^16) 2^224: in all less than
// 0.0275 2^256 (seven of them are 0.02745), so with q > w 2^256 / p - 1 it is above
// x w / p - x / 2^256 - 1 - 0.0275 and
//   0 <= result < (1.0275 + x / 2^256) p.
//
// The factor is the plain value w, not its Montgomery form: x in Montgomery
// form times w is the product in Montgomery form.  Both parts come out of one
// Montgomery reduction of the table entry t = w 2^256 mod p: its row
// multipliers are t (-p^-1) mod 2^256, which is (w 2^256 - t) / p = q, and its
// result is w.
#pragma once

#include "field.cuh"

namespace zntt {

// A fixed factor: the plain value and its quotient.
struct fe_pair {
  fe w, q;
};

// Chains of N full products b_k * m added to 2N words: madN leaves the top
// word's carry (none occurs), madNc puts it into a new word, madNl goes on
// into one more word with the low half of a last product.
__device__ __forceinline__ void mad1(uint32_t& a0, uint32_t& a1, uint32_t b0, uint32_t m) {
  asm("mad.lo.cc.u32  %0, %2, %3, %0;\n\t"
      "madc.hi.u32    %1, %2, %3, %1;"
      : "+r"(a0), "+r"(a1)
      : "r"(b0), "r"(m));
}
__device__ __forceinline__ void mad2(uint32_t& a0, uint32_t& a1, uint32_t& a2, uint32_t& a3, uint32_t b0, uint32_t b1, uint32_t m) {
  asm("mad.lo.cc.u32  %0, %4, %6, %0;\n\t"
      "madc.hi.cc.u32 %1, %4, %6, %1;\n\t"
      "madc.lo.cc.u32 %2, %5, %6, %2;\n\t"
      "madc.hi.u32    %3, %5, %6, %3;"
      : "+r"(a0), "+r"(a1), "+r"(a2), "+r"(a3)
      : "r"(b0), "r"(b1), "r"(m));
}
__device__ __forceinline__ void mad3(uint32_t& a0, uint32_t& a1, uint32_t& a2, uint32_t& a3, uint32_t& a4, uint32_t& a5, uint32_t b0, uint32_t b1, uint32_t b2, uint32_t m) {
  asm("mad.lo.cc.u32  %0, %6, %9, %0;\n\t"
      "madc.hi.cc.u32 %1, %6, %9, %1;\n\t"
      "madc.lo.cc.u32 %2, %7, %9, %2;\n\t"
      "madc.hi.cc.u32 %3, %7, %9, %3;\n\t"
      "madc.lo.cc.u32 %4, %8, %9, %4;\n\t"
      "madc.hi.u32    %5, %8, %9, %5;"
      : "+r"(a0), "+r"(a1), "+r"(a2), "+r"(a3), "+r"(a4), "+r"(a5)
      : "r"(b0), "r"(b1), "r"(b2), "r"(m));
}
__device__ __forceinline__ void mad4(uint32_t& a0, uint32_t& a1, uint32_t& a2, uint32_t& a3, uint32_t& a4, uint32_t& a5, uint32_t& a6, uint32_t& a7, uint32_t b0, uint32_t b1, uint32_t b2, uint32_t b3, uint32_t m) {
  asm("mad.lo.cc.u32  %0, %8, %12, %0;\n\t"
      "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
      "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
      "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
      "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
      "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
      "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
      "madc.hi.u32    %7, %11, %12, %7;"
      : "+r"(a0), "+r"(a1), "+r"(a2), "+r"(a3), "+r"(a4), "+r"(a5), "+r"(a6), "+r"(a7)
      : "r"(b0), "r"(b1), "r"(b2), "r"(b3), "r"(m));
}
__device__ __forceinline__ void mad1c(uint32_t& a0, uint32_t& a1, uint32_t& a2, uint32_t b0, uint32_t m) {
  asm("mad.lo.cc.u32  %0, %3, %4, %0;\n\t"
      "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
      "addc.u32       %2, 0, 0;"
      : "+r"(a0), "+r"(a1), "=r"(a2)
      : "r"(b0), "r"(m));
}
__device__ __forceinline__ void mad2c(uint32_t& a0, uint32_t& a1, uint32_t& a2, uint32_t& a3, uint32_t& a4, uint32_t b0, uint32_t b1, uint32_t m) {
  asm("mad.lo.cc.u32  %0, %5, %7, %0;\n\t"
      "madc.hi.cc.u32 %1, %5, %7, %1;\n\t"
      "madc.lo.cc.u32 %2, %6, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %6, %7, %3;\n\t"
      "addc.u32       %4, 0, 0;"
      : "+r"(a0), "+r"(a1), "+r"(a2), "+r"(a3), "=r"(a4)
      : "r"(b0), "r"(b1), "r"(m));
}
__device__ __forceinline__ void mad3c(uint32_t& a0, uint32_t& a1, uint32_t& a2, uint32_t& a3, uint32_t& a4, uint32_t& a5, uint32_t& a6, uint32_t b0, uint32_t b1, uint32_t b2, uint32_t m) {
  asm("mad.lo.cc.u32  %0, %7, %10, %0;\n\t"
      "madc.hi.cc.u32 %1, %7, %10, %1;\n\t"
      "madc.lo.cc.u32 %2, %8, %10, %2;\n\t"
      "madc.hi.cc.u32 %3, %8, %10, %3;\n\t"
      "madc.lo.cc.u32 %4, %9, %10, %4;\n\t"
      "madc.hi.cc.u32 %5, %9, %10, %5;\n\t"
      "addc.u32       %6, 0, 0;"
      : "+r"(a0), "+r"(a1), "+r"(a2), "+r"(a3), "+r"(a4), "+r"(a5), "=r"(a6)
      : "r"(b0), "r"(b1), "r"(b2), "r"(m));
}
__device__ __forceinline__ void mad4c(uint32_t& a0, uint32_t& a1, uint32_t& a2, uint32_t& a3, uint32_t& a4, uint32_t& a5, uint32_t& a6, uint32_t& a7, uint32_t& a8, uint32_t b0, uint32_t b1, uint32_t b2, uint32_t b3, uint32_t m) {
  asm("mad.lo.cc.u32  %0, %9, %13, %0;\n\t"
      "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
      "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
      "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
      "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
      "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
      "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
      "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
      "addc.u32       %8, 0, 0;"
      : "+r"(a0), "+r"(a1), "+r"(a2), "+r"(a3), "+r"(a4), "+r"(a5), "+r"(a6), "+r"(a7), "=r"(a8)
      : "r"(b0), "r"(b1), "r"(b2), "r"(b3), "r"(m));
}
__device__ __forceinline__ void mad1l(uint32_t& a0, uint32_t& a1, uint32_t& a2, uint32_t b0, uint32_t b1, uint32_t m) {
  asm("mad.lo.cc.u32  %0, %3, %5, %0;\n\t"
      "madc.hi.cc.u32 %1, %3, %5, %1;\n\t"
      "madc.lo.u32    %2, %4, %5, %2;"
      : "+r"(a0), "+r"(a1), "+r"(a2)
      : "r"(b0), "r"(b1), "r"(m));
}
__device__ __forceinline__ void mad2l(uint32_t& a0, uint32_t& a1, uint32_t& a2, uint32_t& a3, uint32_t& a4, uint32_t b0, uint32_t b1, uint32_t b2, uint32_t m) {
  asm("mad.lo.cc.u32  %0, %5, %8, %0;\n\t"
      "madc.hi.cc.u32 %1, %5, %8, %1;\n\t"
      "madc.lo.cc.u32 %2, %6, %8, %2;\n\t"
      "madc.hi.cc.u32 %3, %6, %8, %3;\n\t"
      "madc.lo.u32    %4, %7, %8, %4;"
      : "+r"(a0), "+r"(a1), "+r"(a2), "+r"(a3), "+r"(a4)
      : "r"(b0), "r"(b1), "r"(b2), "r"(m));
}
__device__ __forceinline__ void mad3l(uint32_t& a0, uint32_t& a1, uint32_t& a2, uint32_t& a3, uint32_t& a4, uint32_t& a5, uint32_t& a6, uint32_t b0, uint32_t b1, uint32_t b2, uint32_t b3, uint32_t m) {
  asm("mad.lo.cc.u32  %0, %7, %11, %0;\n\t"
      "madc.hi.cc.u32 %1, %7, %11, %1;\n\t"
      "madc.lo.cc.u32 %2, %8, %11, %2;\n\t"
      "madc.hi.cc.u32 %3, %8, %11, %3;\n\t"
      "madc.lo.cc.u32 %4, %9, %11, %4;\n\t"
      "madc.hi.cc.u32 %5, %9, %11, %5;\n\t"
      "madc.lo.u32    %6, %10, %11, %6;"
      : "+r"(a0), "+r"(a1), "+r"(a2), "+r"(a3), "+r"(a4), "+r"(a5), "+r"(a6)
      : "r"(b0), "r"(b1), "r"(b2), "r"(b3), "r"(m));
}


__device__ __forceinline__ fe fe_sub_raw(const fe& a, const fe& b) {
  fe r;
  asm("sub.cc.u32  %0, %8, %16;\n\t"
      "subc.cc.u32 %1, %9, %17;\n\t"
      "subc.cc.u32 %2, %10, %18;\n\t"
      "subc.cc.u32 %3, %11, %19;\n\t"
      "subc.cc.u32 %4, %12, %20;\n\t"
      "subc.cc.u32 %5, %13, %21;\n\t"
      "subc.cc.u32 %6, %14, %22;\n\t"
      "subc.u32    %7, %15, %23;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
        "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
  return r;
}
__device__ __forceinline__ fe fe_add_raw(const fe& a, const fe& b) {
  fe r;
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
        "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
  return r;
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
// c + the products of a's two 16-bit halves with b's two low (high) bytes.
__device__ __forceinline__ uint32_t dp2a_lo(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("dp2a.lo.u32.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}
__device__ __forceinline__ uint32_t dp2a_hi(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("dp2a.hi.u32.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}

// Words 8..15 of x * b, from the columns 7..14 of the product and an estimate of
// column 6 (above).  Even columns accumulate in e (word 8 on), odd ones in o (word
// 7 on).  The estimate, 35 bits at word 7, starts them, one word each: the first
// product of a column takes a word more without a carry, but not two.
__device__ __forceinline__ fe mul_high(const fe& x, const fe& b) {
  // Column 6: the 16 top bits of x_i times the 8 top bits of b_(6-i).
  const uint32_t x01 = prmt(x.v[0], x.v[1], 0x7632), x23 = prmt(x.v[2], x.v[3], 0x7632),
                 x45 = prmt(x.v[4], x.v[5], 0x7632), x6 = x.v[6] >> 16;
  const uint32_t b6543 = prmt(prmt(b.v[6], b.v[5], 0x0073), prmt(b.v[4], b.v[3], 0x0073), 0x5410),
                 b210 = prmt(prmt(b.v[2], b.v[1], 0x0073), b.v[0], 0x0710);
  uint32_t c6 = dp2a_lo(x01, b6543, 0);
  c6 = dp2a_hi(x23, b6543, c6);
  c6 = dp2a_lo(x45, b210, c6);
  c6 = dp2a_hi(x6, b210, c6);
  uint32_t e8 = c6 >> 24, e9 = 0, e10 = 0, e11 = 0, e12, e13 = 0, e14, e15 = 0;
  uint32_t o7 = c6 << 8, o8 = 0, o9, o10 = 0, o11, o12 = 0, o13, o14 = 0, o15;
  mad1(o7, o8, b.v[7], x.v[0]);
  mad1(e8, e9, b.v[7], x.v[1]);
  mad1c(o7, o8, o9, b.v[6], x.v[1]);
  mad1c(e8, e9, e10, b.v[6], x.v[2]);
  mad2(o7, o8, o9, o10, b.v[5], b.v[7], x.v[2]);
  mad2(e8, e9, e10, e11, b.v[5], b.v[7], x.v[3]);
  mad2c(o7, o8, o9, o10, o11, b.v[4], b.v[6], x.v[3]);
  mad2c(e8, e9, e10, e11, e12, b.v[4], b.v[6], x.v[4]);
  mad3(o7, o8, o9, o10, o11, o12, b.v[3], b.v[5], b.v[7], x.v[4]);
  mad3(e8, e9, e10, e11, e12, e13, b.v[3], b.v[5], b.v[7], x.v[5]);
  mad3c(o7, o8, o9, o10, o11, o12, o13, b.v[2], b.v[4], b.v[6], x.v[5]);
  mad3c(e8, e9, e10, e11, e12, e13, e14, b.v[2], b.v[4], b.v[6], x.v[6]);
  mad4(o7, o8, o9, o10, o11, o12, o13, o14, b.v[1], b.v[3], b.v[5], b.v[7], x.v[6]);
  mad4(e8, e9, e10, e11, e12, e13, e14, e15, b.v[1], b.v[3], b.v[5], b.v[7], x.v[7]);
  mad4c(o7, o8, o9, o10, o11, o12, o13, o14, o15, b.v[0], b.v[2], b.v[4], b.v[6], x.v[7]);
  fe r;
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
        "=r"(r.v[7])
      : "r"(e8), "r"(e9), "r"(e10), "r"(e11), "r"(e12), "r"(e13), "r"(e14), "r"(e15), "r"(o8),
        "r"(o9), "r"(o10), "r"(o11), "r"(o12), "r"(o13), "r"(o14), "r"(o15));
  return r;
}

// The low 256 bits of a running sum of products: even columns in e, odd ones
// in o (o[1..7]; its word 7 takes low halves only).
struct low_acc {
  uint32_t e[8], o[8];
};

// acc += x * b mod 2^256.
__device__ __forceinline__ void mul_low_add(low_acc& s, const fe& x, const fe& b) {
  mad4(s.e[0], s.e[1], s.e[2], s.e[3], s.e[4], s.e[5], s.e[6], s.e[7], b.v[0], b.v[2], b.v[4], b.v[6], x.v[0]);
  mad3l(s.o[1], s.o[2], s.o[3], s.o[4], s.o[5], s.o[6], s.o[7], b.v[1], b.v[3], b.v[5], b.v[7], x.v[0]);
  mad3(s.e[2], s.e[3], s.e[4], s.e[5], s.e[6], s.e[7], b.v[1], b.v[3], b.v[5], x.v[1]);
  mad3l(s.o[1], s.o[2], s.o[3], s.o[4], s.o[5], s.o[6], s.o[7], b.v[0], b.v[2], b.v[4], b.v[6], x.v[1]);
  mad3(s.e[2], s.e[3], s.e[4], s.e[5], s.e[6], s.e[7], b.v[0], b.v[2], b.v[4], x.v[2]);
  mad2l(s.o[3], s.o[4], s.o[5], s.o[6], s.o[7], b.v[1], b.v[3], b.v[5], x.v[2]);
  mad2(s.e[4], s.e[5], s.e[6], s.e[7], b.v[1], b.v[3], x.v[3]);
  mad2l(s.o[3], s.o[4], s.o[5], s.o[6], s.o[7], b.v[0], b.v[2], b.v[4], x.v[3]);
  mad2(s.e[4], s.e[5], s.e[6], s.e[7], b.v[0], b.v[2], x.v[4]);
  mad1l(s.o[5], s.o[6], s.o[7], b.v[1], b.v[3], x.v[4]);
  mad1(s.e[6], s.e[7], b.v[1], x.v[5]);
  mad1l(s.o[5], s.o[6], s.o[7], b.v[0], b.v[2], x.v[5]);
  mad1(s.e[6], s.e[7], b.v[0], x.v[6]);
  s.o[7] += b.v[1] * x.v[6];
  s.o[7] += b.v[0] * x.v[7];
}

__device__ __forceinline__ fe low_merge(const low_acc& s) {
  fe r;
  r.v[0] = s.e[0];
  asm("add.cc.u32  %0, %7, %14;\n\t"
      "addc.cc.u32 %1, %8, %15;\n\t"
      "addc.cc.u32 %2, %9, %16;\n\t"
      "addc.cc.u32 %3, %10, %17;\n\t"
      "addc.cc.u32 %4, %11, %18;\n\t"
      "addc.cc.u32 %5, %12, %19;\n\t"
      "addc.u32    %6, %13, %20;"
      : "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
      : "r"(s.e[1]), "r"(s.e[2]), "r"(s.e[3]), "r"(s.e[4]), "r"(s.e[5]), "r"(s.e[6]), "r"(s.e[7]), "r"(s.o[1]),
        "r"(s.o[2]), "r"(s.o[3]), "r"(s.o[4]), "r"(s.o[5]), "r"(s.o[6]), "r"(s.o[7]));
  return r;
}

// 2^256 - p: adding quotient * (2^256 - p) subtracts quotient * p mod 2^256.
template <class F>
__device__ __forceinline__ fe fe_neg_p() {
  fe r;
  r.v[0] = ~F::P0 + 1u;  // p is odd: the borrow reaches every higher word
  r.v[1] = ~F::P1; r.v[2] = ~F::P2; r.v[3] = ~F::P3;
  r.v[4] = ~F::P4; r.v[5] = ~F::P5; r.v[6] = ~F::P6; r.v[7] = ~F::P7;
  return r;
}

// acc += x * b * 2^64 mod 2^256 for b of six words.
__device__ __forceinline__ void mul_low_add_hi6(low_acc& s, const fe& x, const fe& b) {
  mad3(s.e[2], s.e[3], s.e[4], s.e[5], s.e[6], s.e[7], b.v[0], b.v[2], b.v[4], x.v[0]);
  mad2l(s.o[3], s.o[4], s.o[5], s.o[6], s.o[7], b.v[1], b.v[3], b.v[5], x.v[0]);
  mad2l(s.o[3], s.o[4], s.o[5], s.o[6], s.o[7], b.v[0], b.v[2], b.v[4], x.v[1]);
  mad2(s.e[4], s.e[5], s.e[6], s.e[7], b.v[1], b.v[3], x.v[1]);
  mad2(s.e[4], s.e[5], s.e[6], s.e[7], b.v[0], b.v[2], x.v[2]);
  mad1l(s.o[5], s.o[6], s.o[7], b.v[1], b.v[3], x.v[2]);
  mad1l(s.o[5], s.o[6], s.o[7], b.v[0], b.v[2], x.v[3]);
  mad1(s.e[6], s.e[7], b.v[1], x.v[3]);
  mad1(s.e[6], s.e[7], b.v[0], x.v[4]);
  s.o[7] += b.v[1] * x.v[4];
  s.o[7] += b.v[0] * x.v[5];
}

// x * w mod p up to a multiple of p, below (1.0275 + x / 2^256) p, for the fixed
// factor (w, q).
//
// BLS12-381-Fr's low limbs make 28 of the 64 slots of quotient * p shifts and
// adds: p = h 2^64 + 2^64 - 2^32 + 1 with h = floor(p / 2^64), so -t p is
// t (2^192 - 1 - h) 2^64 + t 2^32 - t mod 2^256.  The pass kernel gained 4.4%
// from it (2^24 forward 2.892 -> 2.764 ms, B200).  BN254-Fr's p0 = 2^32 -
// 2^28 + 1 would save 15 slots for 24 adds and shifts: 2.707 -> 2.752 ms, not used.
template <class F>
__device__ __forceinline__ fe fe_mul_fixed(const fe& x, const fe& w, const fe& q) {
  const fe t = mul_high(x, q);
  low_acc s;
#pragma unroll
  for (int k = 0; k < 8; k++) s.e[k] = s.o[k] = 0;
  mul_low_add(s, w, x);
  if constexpr (F::kLow64) {
    fe nh, sh;
    nh.v[0] = ~F::P2; nh.v[1] = ~F::P3; nh.v[2] = ~F::P4; nh.v[3] = ~F::P5; nh.v[4] = ~F::P6; nh.v[5] = ~F::P7;
    nh.v[6] = nh.v[7] = 0;
    mul_low_add_hi6(s, t, nh);
    sh.v[0] = 0;
#pragma unroll
    for (int k = 1; k < 8; k++) sh.v[k] = t.v[k - 1];
    return fe_sub_raw(fe_add_raw(low_merge(s), sh), t);
  } else {
    mul_low_add(s, fe_neg_p<F>(), t);
    return low_merge(s);
  }
}

// A fixed factor in memory: 64 bytes, the value and then the quotient, each
// one 32-byte load.
__device__ __forceinline__ fe ld_fe32(const uint4* p) {
  fe r;
  asm("ld.global.nc.v8.u32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
      : "l"(p));
  return r;
}
__device__ __forceinline__ void pair_store(uint4* p, const fe_pair& f) {
  fe_store(p, f.w);
  fe_store(p + 2, f.q);
}

// The fixed factor of a table entry t = w 2^256 mod p (t < p).
template <class F>
__device__ __forceinline__ fe_pair pair_of(const fe& t) {
  fe_pair f;
  f.w = fe_from_mont<F>(t, &f.q);
  return f;
}
// ... and the table entry of a fixed factor: t = w 2^256 - q p = q (-p) mod 2^256.
template <class F>
__device__ __forceinline__ fe pair_entry(const fe& q) {
  low_acc s;
#pragma unroll
  for (int k = 0; k < 8; k++) s.e[k] = s.o[k] = 0;
  mul_low_add(s, fe_neg_p<F>(), q);
  return low_merge(s);
}

// x / 2 mod p for x in [0, p): x or x + p, whichever is even, shifted down.
template <class F>
__device__ __forceinline__ fe fe_half(const fe& x) {
  const uint32_t odd = 0u - (x.v[0] & 1u);
  fe p;
  p.v[0] = F::P0 & odd; p.v[1] = F::P1 & odd; p.v[2] = F::P2 & odd; p.v[3] = F::P3 & odd;
  p.v[4] = F::P4 & odd; p.v[5] = F::P5 & odd; p.v[6] = F::P6 & odd; p.v[7] = F::P7 & odd;
  const fe s = fe_add_raw(x, p);  // below 2p < 2^256
  fe r;
#pragma unroll
  for (int k = 0; k < 7; k++) r.v[k] = __funnelshift_r(s.v[k], s.v[k + 1], 1);
  r.v[7] = s.v[7] >> 1;
  return r;
}

// k * p for k = 0..5, as two planes of 16-byte halves.
struct Multiples {
  uint32_t h[2][6][4];
};
template <class F>
constexpr Multiples make_multiples() {
  Multiples m{};
  const uint32_t p[8] = {F::P0, F::P1, F::P2, F::P3, F::P4, F::P5, F::P6, F::P7};
  for (uint32_t k = 0; k < 6; k++) {
    uint64_t c = 0;
    for (int i = 0; i < 8; i++) {
      c += (uint64_t)k * p[i];
      m.h[i / 4][k][i % 4] = (uint32_t)c;
      c >>= 32;
    }
  }
  return m;
}
static __device__ const __align__(16) Multiples kBnMultiples = make_multiples<Bn254Fr>();

// The ranges of the butterflies, u, v -> u + t, u - t with t = w v.
//
// Lazy fields (BN254-Fr: 2^256 = 5.29 p).  v may be any value below 5.07 p, for
// which t stays below 1.986 p, so only u needs a bound, and two stages in a row
// need it once: from u < 1.07 p the first stage's results are below 3.07 p and,
// as u of the second stage, lead to results below 5.07 p < 2^256.  fe_weak brings a
// stored value (or a v whose factor is one) below 1.07 p: k = its top byte times
// 84 / 4096 rounded down (p is 48.39 units of that byte, 4096 / 84 is 48.76) is at
// most x / p and above x / p - 1.07.
// Other fields (BLS12-381-Fr: 2^256 = 2.21 p) keep values below 2 p, for which t is
// below 1.934 p: u and t are reduced to [0, p) before each butterfly.
template <class F>
__device__ __forceinline__ fe fe_weak(const fe& x) {
  if constexpr (F::kLazy) {
    const uint32_t k = ((x.v[7] >> 24) * 84u) >> 12;
    const uint4* m = reinterpret_cast<const uint4*>(&kBnMultiples) + k;
    const uint4 lo = __ldg(m), hi = __ldg(m + 6);
    fe y;
    y.v[0] = lo.x; y.v[1] = lo.y; y.v[2] = lo.z; y.v[3] = lo.w;
    y.v[4] = hi.x; y.v[5] = hi.y; y.v[6] = hi.z; y.v[7] = hi.w;
    return fe_sub_raw(x, y);
  } else {
    return fe_reduce<F>(x);
  }
}

// Any butterfly result -> [0, p).
template <class F>
__device__ __forceinline__ fe fe_canonical(const fe& x) {
  if constexpr (F::kLazy) return fe_reduce<F>(fe_weak<F>(x));
  else return fe_reduce<F>(x);
}

// sum = u + t, diff = u - t up to a multiple of p, in the ranges above.
template <class F>
__device__ __forceinline__ void fe_butterfly(const fe& u, const fe& t, fe& sum, fe& diff) {
  fe off;
  if constexpr (F::kLazy) {
    off.v[0] = F::Q0; off.v[1] = F::Q1; off.v[2] = F::Q2; off.v[3] = F::Q3;
    off.v[4] = F::Q4; off.v[5] = F::Q5; off.v[6] = F::Q6; off.v[7] = F::Q7;
  } else {
    off.v[0] = F::P0; off.v[1] = F::P1; off.v[2] = F::P2; off.v[3] = F::P3;
    off.v[4] = F::P4; off.v[5] = F::P5; off.v[6] = F::P6; off.v[7] = F::P7;
  }
  sum = fe_add_raw(u, t);
  diff = fe_sub_raw(fe_add_raw(u, off), t);
}

// One FRI fold: (a + b) / 2 + alpha (a - b) / (2 x) for canonical a and b, with the
// fixed factors 1 / (2 x) (entry j of a table; NARROW: an element) and alpha.
template <class F, bool NARROW = false>
__device__ __forceinline__ fe fe_fold(const fe& a, const fe& b, const uint4* table, uint64_t j, const fe_pair& alpha) {
  const fe even = fe_half<F>(fe_add<F>(a, b));
  fe p;
  p.v[0] = F::P0; p.v[1] = F::P1; p.v[2] = F::P2; p.v[3] = F::P3;
  p.v[4] = F::P4; p.v[5] = F::P5; p.v[6] = F::P6; p.v[7] = F::P7;
  const fe d = fe_sub_raw(fe_add_raw(a, p), b);  // (0, 2p)
  const uint4* f = table + (NARROW ? 2 : 4) * j;
  fe t;
  if constexpr (NARROW) t = fe_mul<F>(fe_load_nc(f), d);
  else t = fe_mul_fixed<F>(d, ld_fe32(f), ld_fe32(f + 2));
  const fe odd = fe_mul_fixed<F>(t, alpha.w, alpha.q);  // below 2p
  if constexpr (F::kLazy) return fe_canonical<F>(fe_add_raw(even, odd));
  else return fe_add<F>(even, fe_reduce<F>(odd));
}

}  // namespace zntt
