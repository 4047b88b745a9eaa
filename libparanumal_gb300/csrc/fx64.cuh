// Block fixed-point arithmetic for FP64-accurate contractions on the integer pipe.
//
// A line of FP64 values shares the exponent of its largest magnitude: value = F * 2^(eL -
// 1075 - S) with an integer |F| < 2^(53 + S), and eL the biased FP64 exponent of the line's
// largest entry. A value keeps all 53 bits of its significand down to 2^-S of the largest
// entry; below that it is cut at 2^-(52 + S) of it. Matrix rows are held the same way
// (exponent eR of the row's largest entry).
//
// F is used as signed halves, F = h * 2^31 + l with |l| <= 2^30, and a product F * D takes
// three 32 x 32 + 64 multiply-adds: the two middle quarters and the high one. The low x low
// quarter is dropped; a sum holds F * D / 2^62, with the largest possible product of one
// line entry and one row entry at 2^55 or more and at most a quarter of a unit lost per
// product. The sums are exact apart from that and one rounding, where FP64 rounds after
// every term (N = 7, smooth field: error of the operator 1.0e-14 against 1.9e-14).
//
// GB300 issues 64 multiply-adds (32 x 32 + 64) per clock and SM against 2 FP64 operations
// (61 and 1.9 measured), so the three take a tenth of the time of the FP64 FMA they replace.
//
// Lines whose largest entry is not in [2^-895, 2^897) (Inf, NaN, subnormals, zero) are left
// to the caller (fx_ordinary), and so should be those where one entry outweighs all others
// together: a sum of which that entry is no part is exact to the unit of the line only, not to
// that of its own terms.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace lpg {

// magnitude key of a double: the high word without its sign; its top 11 bits are the
// biased exponent
__device__ __forceinline__ unsigned fx_key(double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; }
__device__ __forceinline__ bool fx_ordinary(int eL) { return (unsigned)(eL - 128) < 1792u; }

// 2 F of v for S = SH - 1 on a line of biased exponent eL >= 128 (entries so small against
// the line's largest that nothing is left, zeros and subnormals among them, shift to 0: the
// PTX shift clamps its amount). Negative values are complemented, not negated: one unit of
// 2 F, the size of the cut.
// mag: the high word of the magnitude of 2 F (in [2^(20 + SH), 2^(21 + SH)) for the largest).
template <int SH>
__device__ __forceinline__ int64_t fx_from_double(double v, int eL, unsigned& mag) {
  const int hi = __double2hiint(v), lo = __double2loint(v);
  const int n = eL - (int)(fx_key(v) >> 20);
  const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
  int64_t F;
  asm("{\n"
      ".reg .u32 h, l;\n"
      ".reg .s32 s;\n"
      ".reg .u64 m;\n"
      "shf.l.wrap.b32 h, %3, %2, %6;\n"
      "shl.b32 l, %3, %6;\n"
      "mov.b64 m, {l, h};\n"
      "shr.u64 m, m, %4;\n"
      "shr.s32 s, %5, 31;\n"
      "mov.b64 {l, h}, m;\n"
      "mov.u32 %1, h;\n"
      "xor.b32 l, l, s;\n"
      "xor.b32 h, h, s;\n"
      "mov.b64 %0, {l, h};\n"
      "}\n"
      : "=l"(F), "=r"(mag)
      : "r"(mh), "r"(lo), "r"(n), "r"(hi), "n"(SH));
  return F;
}
template <int SH>
__device__ __forceinline__ int64_t fx_from_double(double v, int eL) {
  unsigned mag;
  return fx_from_double<SH>(v, eL, mag);
}

// base word of fx_to_double for R * 2^(E - 1086): a normal result for 64 <= E <= 2047 (a line's
// exponent reaches 1919, a row's 1086: E <= 1990 in the operators and transfers)
__device__ __forceinline__ int fx_base(int E) { return (E - 1) << 20; }

// R * 2^(E - 1086), |R| < 2^63, rounded to nearest: |R| is shifted so that its leading bit
// becomes the implicit one, which the sum then adds to the exponent field of base; the
// carry of the rounding may pass into it, as it should
__device__ __forceinline__ double fx_to_double(int64_t R, int base) {
  double v;
  asm("{\n"
      ".reg .u32 h, l, n, t, s, x, y;\n"
      ".reg .s64 a;\n"
      ".reg .pred p, z;\n"
      "mov.b64 {x, s}, %1;\n"
      "setp.lt.s32 p, s, 0;\n"
      "mov.b64 a, %1;\n"
      "@p neg.s64 a, a;\n"
      "mov.b64 {l, h}, a;\n"
      "bfind.shiftamt.u32 n, h;\n"          // leading zeros; -1 for 0
      "bfind.shiftamt.u32 t, l;\n"
      "add.s32 t, t, 32;\n"
      "setp.eq.u32 p, h, 0;\n"
      "selp.b32 n, t, n, p;\n"
      "setp.eq.and.u32 z, n, 31, p;\n"     // only 0 has a leading -1 + 32 in its low word
      "shl.b64 a, a, n;\n"
      "mov.b64 {l, h}, a;\n"
      "shf.r.wrap.b32 x, l, h, 11;\n"
      "shr.u32 y, h, 11;\n"
      "shl.b32 t, l, 21;\n"
      "add.cc.u32 t, t, t;\n"               // carry = the bit below the significand
      "addc.cc.u32 x, x, 0;\n"
      "addc.u32 y, y, %2;\n"
      "mad.lo.s32 y, n, -1048576, y;\n"
      "lop3.b32 y, s, -2147483648, y, 0xea;\n"   // (s & sign) | y
      "selp.b32 y, 0, y, z;\n"
      "mov.b64 %0, {x, y};\n"
      "}\n"
      : "=d"(v)
      : "l"(R), "r"(base));
  return v;
}

// R >> n, n >= 0 (the PTX shift clamps n: the sign remains)
__device__ __forceinline__ int64_t fx_shr(int64_t R, int n) {
  asm("shr.s64 %0, %0, %1;" : "+l"(R) : "r"(n));
  return R;
}

struct fx_half {
  int h, l;
};
// halves of F from 2 F: the word boundary of 2 F is the 31-bit boundary of F
__device__ __forceinline__ fx_half fx_split(int64_t F2) { return {(int)((F2 + 0x80000000ll) >> 32), (int)F2 >> 1}; }

// c + a * b with a 64-bit sum. As PTX: from C++ the halves of a 64-bit value are multiplied
// as 64-bit integers, three instructions for one.
__device__ __forceinline__ int64_t fx_mad(int a, int b, int64_t c) {
  int64_t r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}

// a * b with a 64-bit product
__device__ __forceinline__ int64_t fx_mul(int a, int b) {
  int64_t r;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
  return r;
}

// sum of products of split integers, in units of 2^62: the middle quarters (started with the
// first product's), then the high ones on top of them, shifted. The shift rounds down;
// starting from 2^30 it rounds to nearest.
struct fx_acc {
  int64_t v;
  __device__ __forceinline__ fx_acc(fx_half a, fx_half b) { v = fx_mad(a.l, b.h, fx_mul(a.h, b.l)); }
  __device__ __forceinline__ explicit fx_acc(int64_t v0) : v(v0) {}
  __device__ __forceinline__ void cross(fx_half a, fx_half b) { v = fx_mad(a.l, b.h, fx_mad(a.h, b.l, v)); }
  __device__ __forceinline__ void fold() { v >>= 31; }
  __device__ __forceinline__ void high(fx_half a, fx_half b) { v = fx_mad(a.h, b.h, v); }
};

}  // namespace lpg
