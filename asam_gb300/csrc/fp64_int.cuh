// Correctly rounded FP64 multiplication and division on the integer units.
//
// GB300 executes one FP64 warp instruction in 64 cycles per SM sub-partition,
// dependent or not (19 per SM with all four busy; 1.06 TFLOP/s for the GPU),
// so a kernel that multiplies and divides in FP64 is bound by that unit while
// the integer units idle.  The functions below compute the IEEE
// round-to-nearest-even result with 32-bit integer multiplies: a product in
// about 35 integer instructions (14 cycles per SM and warp at full occupancy
// against 19 for DMUL, and both units run side by side), a quotient by a
// known divisor in about 30 and a general quotient in about 75, where FP64
// takes three and about ten instructions.  Operands with an exponent outside
// [-480, 480] (zero apart), infinities and NaN take the FP64 instruction, so
// the result is that of the hardware bit for bit for every operand.
//
// Quotients: R = 2^127/D for the divisor's left-justified significand D, by
// Newton's iteration in fixed point from a single-precision seed; the 64-bit
// product of the dividend's significand and R carries ten or eleven bits beyond
// the result's 53, and when those lie within the error of the rounding point
// the exact remainder of the midpoint decides (a quotient of two 53-bit
// significands is never a midpoint itself).
#pragma once
#include <cuda_runtime.h>

namespace fpi {

typedef unsigned long long u64;

// exponent field in [543, 1503]: products and quotients of two such numbers
// are normal
__device__ __forceinline__ bool in_range(unsigned hi) { return (hi & 0x7fffffffu) - (543u << 20) < (961u << 20); }

__device__ __forceinline__ bool finite(unsigned hi) { return (hi & 0x7ff00000u) != 0x7ff00000u; }

// significand with the leading one at bit 63
__device__ __forceinline__ u64 left_sig(unsigned hi, unsigned lo) {
  const unsigned h = __funnelshift_l(lo, (hi & 0xfffffu) | 0x100000u, 11);
  return ((u64)h << 32) | (lo << 11);
}

static __device__ __noinline__ double mul_special(double a, double b) { return __dmul_rn(a, b); }
static __device__ __noinline__ double div_special(double a, double b) { return __ddiv_rn(a, b); }

// RN(a*b)
__device__ __forceinline__ double mul_rn(double a, double b) {
  const unsigned ah = __double2hiint(a), al = __double2loint(a), bh = __double2hiint(b), bl = __double2loint(b);
  const unsigned sign = (ah ^ bh) & 0x80000000u;
  if (!(in_range(ah) && in_range(bh))) {
    if ((((ah << 1) | al) == 0 || ((bh << 1) | bl) == 0) && finite(ah) && finite(bh)) return __hiloint2double(sign, 0);
    return mul_special(a, b);
  }
  const unsigned A1 = __funnelshift_l(al, (ah & 0xfffffu) | 0x100000u, 11), A0 = al << 11;
  const unsigned B1 = (bh & 0xfffffu) | 0x100000u, B0 = bl;
  const u64 p00 = (u64)A0 * B0;
  const u64 t1 = (u64)A1 * B0 + (unsigned)(p00 >> 32);
  const u64 t2 = (u64)A0 * B1 + (unsigned)t1;
  const u64 h = (u64)A1 * B1 + (unsigned)(t1 >> 32) + (unsigned)(t2 >> 32);
  const unsigned l0 = (unsigned)p00, l1 = (unsigned)t2, h0 = (unsigned)h, h1 = (unsigned)(h >> 32);
  // the product's leading one is at bit 116 or 115 of 128; shift it to 116
  const unsigned s = (h1 >> 20) ^ 1u;
  const unsigned H1 = __funnelshift_l(h0, h1, s), H0 = __funnelshift_l(l1, h0, s), L1 = __funnelshift_l(l0, l1, s);
  const unsigned r = L1 | min(l0, 1u);  // the bits below the last place, the lowest one sticky
  // exponent less one: the leading one of H adds it
  const unsigned top = ((((ah >> 20) & 0x7ffu) + ((bh >> 20) & 0x7ffu) - 1023u - s) << 20) | sign;
  unsigned x0, x1;
  // carry of r + 0x7fffffff + odd: round to nearest, ties to even
  asm("{.reg .u32 t;\n add.cc.u32 t,%2,%3;\n addc.cc.u32 %0,%4,0;\n addc.u32 %1,%5,%6;}"
      : "=r"(x0), "=r"(x1)
      : "r"(r), "r"(0x7fffffffu + (H0 & 1u)), "r"(H0), "r"(H1), "r"(top));
  return __hiloint2double(x1, x0);
}

// 2^127/D to within 4 for D in [2^63, 2^64) (2^64 itself comes out just below)
__device__ __forceinline__ u64 recip_sig(u64 D) {
  const unsigned Dh = (unsigned)(D >> 32), Dl = (unsigned)D;
  float f;
  asm("rcp.approx.ftz.f32 %0,%1;" : "=f"(f) : "f"(__uint_as_float(0x3f000000u | ((Dh >> 8) & 0x7fffffu))));
  // f in [1, 2] with a relative error below 2^-21; r1 = f*2^31, kept below 1/d
  const unsigned r1 = __float2uint_rz(f * 2147483648.0f * (1.0f - 5.0e-7f));
  // e1 = 2^63*(1 - r1*d) >= 0, below 2^43
  const u64 e1 = 0x8000000000000000ull - ((u64)r1 * Dh + (unsigned)(((u64)r1 * Dl) >> 32));
  const u64 r2 = ((u64)r1 << 32) + (((u64)r1 * (unsigned)(e1 >> 12)) >> 19);
  // e2 = 2^63*(1 - r2*d), a few 2^22
  const long long e2 = (long long)(0x8000000000000000ull - __umul64hi(r2, D));
  const long long c = ((long long)(unsigned)(r2 >> 32) * (int)e2) >> 31;
  const u64 r3 = r2 + (u64)c;
  return r3 < 0x8000000000000000ull ? 0xffffffffffffffffull : r3;  // D = 2^63: 2^64 does not fit
}
// The reciprocal of a divisor for several quotients: floor(2^127/D), 2^64 - 1
// for a power of two, 0 (no quotient on the integer units) when d is out of
// range.
__device__ __forceinline__ u64 recip(double d) {
  const unsigned dh = (unsigned)__double2hiint(d);
  if (!in_range(dh)) return 0;
  const u64 D = left_sig(dh, (unsigned)__double2loint(d));
  u64 r = recip_sig(D);
  // 2^127 - r*D, a few D either way
  u64 lo = 0 - r * D;
  long long hi = (long long)(0x8000000000000000ull - __umul64hi(r, D) - (lo != 0));
  while (hi < 0) {
    --r;
    lo += D;
    hi += lo < D;
  }
  while ((hi > 0 || lo >= D) && r != 0xffffffffffffffffull) {
    ++r;
    hi -= lo < D;
    lo -= D;
  }
  return r;
}

// The quotients that quot_chain leaves: special operands, and the 53-bit
// candidates m and m + 1 around the midpoint, of which the exact remainder takes
// one (s: the significands' quotient is below 1).
static __device__ __noinline__ double quot_rest(double x, double d, u64 R, u64 m, unsigned s) {
  const unsigned xh = __double2hiint(x), xl = __double2loint(x), dh = __double2hiint(d);
  const unsigned sign = (xh ^ dh) & 0x80000000u;
  if (R == 0 || !in_range(xh)) return __ddiv_rn(x, d);
  const u64 xm = ((u64)((xh & 0xfffffu) | 0x100000u) << 32) | xl;
  const u64 dm = ((u64)((dh & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(d);
  const u64 v = m + ((long long)((xm << (53 + s)) - (2 * m + 1) * dm) > 0);
  const unsigned top = ((xh & 0x7ff00000u) - (dh & 0x7ff00000u) + (1022u << 20) - (s << 20)) | sign;
  return __hiloint2double((unsigned)(v >> 32) + top, (unsigned)v);
}

// RN(x/d), R = recip(d), for a chain of quotients.  The product M*R/2^64 of the dividend's significand,
// without its lowest partial product and with the partial sums cut, is less than
// three units low and R costs less than another one: the quotient lies in
// [q, q + 4), with its leading one at bit 63 or 62; both roundings are formed
// and one is taken.  When the midpoint lies in that interval (one case in 300
// to 700), or for special operands, quot_rest decides; nothing but that one
// test is in the way of the result, 142 cycles after x (three FP64 instructions
// take 192, quot_rn 190); where many warps share the units quot_rn is ahead,
// 17 cycles per SM and warp against 18.
__device__ __forceinline__ double quot_chain(double x, double d, u64 R) {
  const unsigned xh = __double2hiint(x), xl = __double2loint(x), dh = __double2hiint(d);
  const unsigned M1 = __funnelshift_l(xl, xh, 11) | 0x80000000u, M0 = xl << 11;
  const unsigned R1 = (unsigned)(R >> 32), R0 = (unsigned)R;
  const u64 q = (u64)M1 * R1 + (((u64)M1 * R0 >> 32) + ((u64)M0 * R1 >> 32));
  const u64 qa = q + 0x400u, qb = q + 0x200u;
  const unsigned e = (xh & 0x7ff00000u) - (dh & 0x7ff00000u) + (1022u << 20), sign = (xh ^ dh) & 0x80000000u;
  const bool ge1 = (long long)q < 0;  // the significands' quotient is at least 1
  const unsigned v1 = ge1 ? ((unsigned)(qa >> 32) >> 11) + (e | sign) : ((unsigned)(qb >> 32) >> 10) + ((e - (1u << 20)) | sign);
  double v = __hiloint2double(v1, ge1 ? (unsigned)(qa >> 11) : (unsigned)(qb >> 10));
  const unsigned near = ge1 ? ((unsigned)qa + 4u) & 0x7ffu : ((unsigned)qb + 4u) & 0x3ffu;
  if (near < 4u || R == 0 || !in_range(xh)) {
    if (((xh << 1) | xl) == 0 && R != 0)  // the dead cells of a cut-cell column
      v = __hiloint2double(sign, 0);
    else
      v = quot_rest(x, d, R, ge1 ? ((qa + 4) >> 11) - 1 : ((qb + 4) >> 10) - 1, ge1 ? 0u : 1u);
  }
  return v;
}

// RN(x/d) from a reciprocal within 4 (or recip): the midpoint is near in one
// case of 60 to 30, and what decides it stays in line.  recip_quick takes any d;
// the reciprocal of one out of range is not used.
__device__ __forceinline__ u64 recip_quick(double d) {
  return recip_sig(left_sig((unsigned)__double2hiint(d), (unsigned)__double2loint(d)));
}
__device__ __forceinline__ double quot_rn(double x, double d, u64 R) {
  const unsigned xh = __double2hiint(x), xl = __double2loint(x), dh = __double2hiint(d);
  const unsigned sign = (xh ^ dh) & 0x80000000u;
  if (!(in_range(xh) && in_range(dh))) {
    if (((xh << 1) | xl) == 0 && in_range(dh)) return __hiloint2double(sign, 0);
    return div_special(x, d);
  }
  u64 q = __umul64hi(left_sig(xh, xl), R);
  const unsigned s = (unsigned)(q >> 63) ^ 1u;
  q <<= s;
  const unsigned extra = (unsigned)q & 0x7ffu;
  u64 v = q >> 11;
  unsigned up = extra >> 10;
  if (extra - 0x3f0u <= 0x20u) {  // within 16 of the midpoint
    const u64 xm = ((u64)((xh & 0xfffffu) | 0x100000u) << 32) | xl;
    const u64 dm = ((u64)((dh & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(d);
    up = (long long)((xm << (53 + s)) - (2 * v + 1) * dm) > 0;
  }
  v += up;
  const unsigned top = ((((xh >> 20) & 0x7ffu) - ((dh >> 20) & 0x7ffu) + 1022u - s) << 20) | sign;
  return __hiloint2double((unsigned)(v >> 32) + top, (unsigned)v);
}
__device__ __forceinline__ double div_rn(double x, double d) { return quot_rn(x, d, recip_quick(d)); }

// A double whose products and quotients run on the integer units and whose
// sums on the FP64 unit, for expressions that are written out as the reference
// writes them.
struct Num {
  double v;
  __device__ __forceinline__ Num(double x) : v(x) {}
  friend __device__ __forceinline__ Num operator*(Num a, Num b) { return mul_rn(a.v, b.v); }
  friend __device__ __forceinline__ Num operator/(Num a, Num b) { return div_rn(a.v, b.v); }
  friend __device__ __forceinline__ Num operator+(Num a, Num b) { return __dadd_rn(a.v, b.v); }
  friend __device__ __forceinline__ Num operator-(Num a, Num b) { return __dsub_rn(a.v, b.v); }
};

// FP32 to FP64 and back, rounded to nearest even.  A conversion is an FP64
// instruction as well (64 cycles of a sub-partition per warp), so the conversions
// of normal numbers and their products run on the integer units.
__device__ __forceinline__ double widen(float x) {
  const unsigned b = __float_as_uint(x), a = b & 0x7fffffffu;
  if (a - 0x00800000u >= 0x7f000000u && a != 0) return (double)x;  // subnormal, infinite, NaN
  const unsigned hi = a == 0 ? b : ((a >> 3) + (896u << 20)) | (b & 0x80000000u);
  return __hiloint2double((int)hi, (int)(b << 29));
}
__device__ __forceinline__ float narrow(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned a = hi & 0x7fffffffu;
  if (a - (897u << 20) >= (254u << 20)) {  // the result is not a normal number
    if ((a | lo) == 0) return __uint_as_float(hi);
    return (float)x;
  }
  const unsigned m = ((a - (896u << 20)) << 3) | (lo >> 29), rest = lo << 3;
  const unsigned up = rest > 0x80000000u || (rest == 0x80000000u && (m & 1u));
  return __uint_as_float((m + up) | (hi & 0x80000000u));  // a carry out of the largest exponent gives infinity
}

}  // namespace fpi
