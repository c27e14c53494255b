// 64-bit fixed point on the integer pipes, for products and sums that FP64
// would hold to 53 bits.
//
// On this part an FP64 instruction takes an SM's pipe 19 clocks per warp, a
// 32 x 32 -> 64 bit multiply-add 1.2 and a 64-bit add 0.5 (measured), so a sum
// of products of numbers that share a scale is cheaper in integers. A quantity is
// S 2^x: S a signed 64-bit integer, x an exponent shared by the quantities that
// are added.
//
// A factor has up to 62 bits and is held as two signed 32-bit limbs; a product
// keeps the limbs' high and middle partial products, S = (f g) / 2^64 to
// within a unit, with |S| <= 2^60 for 62-bit factors. So a sum is off by a few
// units of 2^-59 of the largest product that the exponents of its factors admit.
// That is less than FP64's error only where its largest term is within some 2^-5
// of that bound, and says nothing about an entry far below the largest that
// shares its exponent: the caller looks at both (k_elem_fix).
#pragma once

#include "common.cuh"

namespace goal {

#ifdef __CUDACC__

constexpr int kFxMinExp = 64;       // least biased exponent of a scale: smaller numbers count as zero
constexpr int kFxFloat = 0x7fff;    // in place of an exponent: the entries are FP64

// Largest difference of the exponents of an element's gradients in x, y and z.
// The entries of a block differ by its square, and one of 2^-10 of the largest
// is held to some 49 bits, as good as in FP64 after its few roundings.
constexpr int kFxSpread = 5;

struct Fx {
  int hi, lo;  // value hi 2^32 + lo
};

// Biased exponent of |v| (0x7ff: infinite or not a number), in the running
// maximum of the high words of a group.
__device__ __forceinline__ int fx_high(double v) { return __double2hiint(v) & 0x7fffffff; }
__device__ __forceinline__ int fx_spread(const int (&x)[3]) {
  return max(x[0], max(x[1], x[2])) - min(x[0], min(x[1], x[2]));
}
__device__ __forceinline__ int fx_exp(int high) { return max(high >> 20, kFxMinExp); }

// v / 2^x, rounded, for |v| < 2^(x + 62)
__device__ __forceinline__ long long fx_at(double v, int x) {
  const int h = __double2hiint(v), l = __double2loint(v);
  const int e = (h >> 20) & 0x7ff;
  const unsigned long long m =
      ((unsigned long long)(unsigned)((h & 0xfffff) | (e ? 0x100000 : 0)) << 42) | ((unsigned long long)(unsigned)l << 10);
  const int k = min(max(1085 + x - e, 0), 63);
  const long long r = (long long)((m + ((1ull << k) >> 1)) >> k), s = h >> 31;
  return (r ^ s) - s;
}
__device__ __forceinline__ Fx fx_split(long long r) {
  Fx f;
  f.lo = (int)r;
  f.hi = (int)((r + 0x80000000ll) >> 32);
  return f;
}
// a factor below 2^(be - 1022) as 60 bits: value = Fx x 2^(be - 1082), or as 62
__device__ __forceinline__ Fx fx_factor(double v, int be) { return fx_split(fx_at(v, be - 1082)); }
__device__ __forceinline__ Fx fx_factor62(double v, int be) { return fx_split(fx_at(v, be - 1084)); }

// a b + c in one instruction (written out, the compiler took three)
__device__ __forceinline__ long long fx_mad(int a, int b, long long c) {
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}

// f g / 2^64, rounded; for factors of up to 62 bits
__device__ __forceinline__ long long fx_mul(const Fx& f, const Fx& g) {
  const long long m = fx_mad(f.lo, g.hi, fx_mad(f.hi, g.lo, 0x80000000ll));
  return fx_mad(f.hi, g.hi, m >> 32);
}
// f g / 2^63
__device__ __forceinline__ long long fx_mul1(const Fx& f, const Fx& g) {
  const long long m = fx_mad(f.lo, g.hi, fx_mad(f.hi, g.lo, 0x40000000ll));
  return (fx_mad(f.hi, g.hi, 0) << 1) + (m >> 31);
}

// Sums of up to three products of 60-bit factors, with five bits more:
// sum / 2^59. High parts in s, middle parts in m (at 2^32).
struct FxSum {
  long long s = 0, m = 0;
  __device__ __forceinline__ void add(const Fx& a, const Fx& b) {
    s = fx_mad(a.hi, b.hi, s);
    m = fx_mad(a.hi, b.lo, m);
    m = fx_mad(a.lo, b.hi, m);
  }
  template <int B>
  __device__ __forceinline__ long long value() const { return (s << B) + (m >> (32 - B)); }  // sum / 2^(64 - B)
  // with the product of the low limbs, where a difference of two large numbers follows
  __device__ __forceinline__ void add_low(const Fx& a, const Fx& b) { m += fx_mad(a.lo, b.lo, 0x80000000ll) >> 32; }
};

// v 2^d
__device__ __forceinline__ long long fx_scale(long long v, int d) {
  return (v << min(max(d, 0), 63)) >> min(max(-d, 0), 63);
}
// bits of |v|
__device__ __forceinline__ unsigned long long fx_abs(long long v) { return (unsigned long long)(v ^ (v >> 63)); }
__device__ __forceinline__ int fx_bits(unsigned long long a) { return 64 - __clzll((long long)a); }

__device__ __forceinline__ int fx_shift(int d) { return min(max(d, 0), 63); }

// acc 2^xa += v 2^xv, at the larger exponent
__device__ __forceinline__ void fx_acc(long long& acc, int xa, long long v, int xv) {
  acc = (acc >> fx_shift(xv - xa)) + (v >> fx_shift(xa - xv));
}

// S 2^x in FP64, correctly rounded while it is a normal number
__device__ __forceinline__ double fx_double(long long s, int x) {
  const double d = (double)s;
  if (abs(x) > 900) return scalbn(d, x);
  return __hiloint2double(__double2hiint(d) + (s ? x << 20 : 0), __double2loint(d));
}

#endif

}  // namespace goal
