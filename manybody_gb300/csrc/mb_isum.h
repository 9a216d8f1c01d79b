// Sums of +-doubles on the integer pipes (device code).
//
// This GPU's FP64 pipe takes one warp instruction in about 17 cycles of an SM
// (measured 0.05-0.06 a cycle), its ALU and FMA pipes two each a cycle.  A
// complex hop is two FP64 adds, 34 cycles; as integers it is about 10 cycles
// (6 where the term was decoded once for many uses).
//
// A sum keeps a 64-bit integer in units of the largest term so far: a term of
// biased exponent e contributes its 53-bit significand, placed so that the
// largest possible term is below 2^(64 - base), shifted right by E - e with E
// the largest exponent met (when E grows the sum so far is shifted too, by a
// spare bit more, which also keeps 2^(base - 1) floored terms of either sign in
// 64 bits: the first ones are below half).  base = 1 + ceil(log2(terms)), at
// least 7 with decoded terms and 6 without (isum_base), leaves room for every
// term's carry; at 64 terms (4x4) it is 7, and 3 or 4 bits stay below a double's
// last place of the largest term (at 512 terms one or none).  What is cut off is
// below one such unit a term, towards zero, or of a decoded term downwards: a
// sum is off by less than 2^-55 (base 7) of its largest term for every term,
// where FP64 adds round by up to 2^-53 of the partial sum.  The bound is
// against the largest term: where large terms cancel, a term below the unit is
// lost that FP64 adds could have kept (1 - 1 + 2^-70 gives 0).  A sum that holds an
// infinity or NaN, or starts with terms below 2^-511 that are not zeros, is
// reported (odd) and left to FP64 by the caller.  Zeros are not: the imaginary
// parts of a real vector, or a neighbourhood outside a sparse vector, are sums
// like any other.
//
// Signs are multiplied in: four terms' high and low parts (29 bits each) times
// +-1 meet in two 32-bit integers, on the FMA pipe, and go to the 64-bit sum
// together.  Conditional complements and carries would run on the ALU pipe,
// which the decoding and shifting already fill: 9.7 ALU and 8.8 FMA
// instructions a term against 14.6 and 3.5, 5.5 against 7.5 cycles of an SM.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstddef>
#include <type_traits>

namespace mb {

// PTX shifts: an amount above 63 gives 0 (or the sign), unlike C++'s
__device__ __forceinline__ unsigned long long shr_clamp(unsigned long long v, uint32_t s) {
  unsigned long long r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
  return r;
}
__device__ __forceinline__ long long sar_clamp(long long v, uint32_t s) {
  long long r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
  return r;
}

constexpr int kISumLeast = 512;  // terms above zero up to this biased exponent are odd
constexpr int kISumOdd = 0x7FF;  // the exponent of an odd sum, and of infinity and NaN

// A sum's constants.  The factors are kept from the compiler, which would
// turn the products into shifts on the ALU pipe.
struct ISumForm {
  int base;
  int unit;             // exponent of the unit less the largest biased exponent
  uint32_t by11;        // 2^11
  int by29, by0;        // 2^29, 1
  __device__ __forceinline__ explicit ISumForm(int b) : base(b), unit(b - 1023 - 63) {
    asm("mov.u32 %0, 2048;" : "=r"(by11));
    asm("mov.u32 %0, 0x20000000;" : "=r"(by29));
    asm("mov.u32 %0, 1;" : "=r"(by0));
  }
};

// A double decoded once for many sums: its signed significand in the top 54
// bits, its biased exponent less 512 in the low 10 (0: zero).  Exponents
// outside 513..1535 do not fit: *out is set for them (not for zeros).
__device__ __forceinline__ long long isum_pack(double v, bool* out) {
  const uint32_t h = (uint32_t)__double2hiint(v), l = (uint32_t)__double2loint(v);
  const uint32_t ex = (h >> 20) & 0x7FFu;
  if (ex <= (uint32_t)kISumLeast || ex > (uint32_t)kISumLeast + 1023u) {
    if ((h + h) | l) *out = true;
    return 0;
  }
  const unsigned long long m =
      ((unsigned long long)((h & 0xFFFFFu) | 0x100000u) << 32 | l) << 10;
  return (long long)((int)h < 0 ? 0ull - m : m) | (long long)(ex - kISumLeast);
}

// One component's sum.
struct ISum {
  long long a = 0;
  int e = kISumLeast;  // at least the largest biased exponent met

  // room for a term that needs `least` (below 0) bits more, and a spare bit, so
  // that most sums grow once
  __device__ __forceinline__ void grow(int least) {
    if (least < 0) {
      a = sar_clamp(a, (uint32_t)(1 - least));
      e += 1 - least;
    }
  }
  // the parts of four terms at most, summed with their signs
  __device__ __forceinline__ void take(const ISumForm& f, int hi, int lo) {
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(a) : "r"(hi), "r"(f.by29));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(a) : "r"(lo), "r"(f.by0));
  }
  // a word of the terms' bits where the sum is still below kISumLeast
  __device__ __forceinline__ void see(uint32_t bits) {
    if (e <= kISumLeast && bits) e = kISumOdd;
  }
  __device__ __forceinline__ bool odd() const { return e >= kISumOdd; }
  // a and the exponent of its unit, for scaled_by
  __device__ __forceinline__ double count() const { return __ll2double_rn(a); }
  __device__ __forceinline__ int exponent(const ISumForm& f) const { return e + f.unit; }
  // a * 2^(e + unit): the conversion rounds, the product is exact.  e > 512 and
  // base < 64 keep the factor a normal number.
  __device__ __forceinline__ double value(const ISumForm& f) const {
    return __ll2double_rn(a) * __hiloint2double((e + f.unit + 1023) << 20, 0);
  }
};

// a * c = (a * 2^k) * c0 exactly, with the power of two in c where that stays a
// normal number (no FP64 instruction), else in a; k of ISum::exponent, or 0.
__device__ __forceinline__ void scaled_by(int k, double c0, double& a, double& c) {
  const int h = __double2hiint(c0), ex = (h >> 20) & 0x7FF;
  c = c0;
  if (ex != 0 && (unsigned)(ex + k - 1) < 2046u && ex != 0x7FF)
    c = __hiloint2double(h + k * (1 << 20), __double2loint(c0));
  else
    a *= __hiloint2double((k + 1023) << 20, 0);
}

// hi += sign * (r >> 32), lo += sign * (bits 3..31 of r)
__device__ __forceinline__ void isum_parts(unsigned long long r, int sign, int& hi, int& lo) {
  hi += (int)(r >> 32) * sign;
  lo += (int)((uint32_t)r >> 3) * sign;
}

// A complex sum.
struct ISum2 {
  ISum re, im;

  // N <= 4 terms; bit 31 of neg[k] turns term k's sign
  template <int N>
  __device__ __forceinline__ void add(const ISumForm& f, const double2 (&v)[N],
                                      const uint32_t (&neg)[N]) {
    int sr[N], si[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      sr[k] = exponent((uint32_t)__double2hiint(v[k].x));
      si[k] = exponent((uint32_t)__double2hiint(v[k].y));
    }
    auto look = [&] {
      uint32_t br = 0, bi = 0;
#pragma unroll
      for (int k = 0; k < N; ++k) {
        br |= bits(v[k].x);
        bi |= bits(v[k].y);
      }
      re.see(br);
      im.see(bi);
    };
    shifts<N>(sr, si, look);
    int rh = 0, rl = 0, ih = 0, il = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int s = 2 * ((int)neg[k] >> 31) + 1;
      part(f, v[k].x, sr[k], s, rh, rl);
      part(f, v[k].y, si[k], s, ih, il);
    }
    re.take(f, rh, rl);
    im.take(f, ih, il);
  }

  // the same of decoded terms (isum_pack)
  template <int N>
  __device__ __forceinline__ void add_packed(const ISumForm& f, const longlong2 (&v)[N],
                                             const uint32_t (&neg)[N]) {
    int sr[N], si[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      sr[k] = (int)((uint32_t)v[k].x & 1023u) + kISumLeast;
      si[k] = (int)((uint32_t)v[k].y & 1023u) + kISumLeast;
    }
    shifts<N>(sr, si, nullptr);
    int rh = 0, rl = 0, ih = 0, il = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int s = 2 * ((int)neg[k] >> 31) + 1;
      isum_parts((unsigned long long)sar_clamp(v[k].x & ~1023ll, (uint32_t)(sr[k] + f.base - 4)), s,
                 rh, rl);
      isum_parts((unsigned long long)sar_clamp(v[k].y & ~1023ll, (uint32_t)(si[k] + f.base - 4)), s,
                 ih, il);
    }
    re.take(f, rh, rl);
    im.take(f, ih, il);
  }

  __device__ __forceinline__ bool odd() const { return re.odd() || im.odd(); }
  __device__ __forceinline__ double2 value(const ISumForm& f) const {
    return make_double2(re.value(f), im.value(f));
  }

 private:
  static __device__ __forceinline__ int exponent(uint32_t h) { return (int)((h + h) >> 21); }

  // zero for +-0 alone
  static __device__ __forceinline__ uint32_t bits(double v) {
    const uint32_t h = (uint32_t)__double2hiint(v);
    return (h + h) | (uint32_t)__double2loint(v);
  }

  // Exponents -> right shifts, the sums brought to larger exponents first.  look
  // (undecoded terms) runs while a sum holds only zeros: rare, but for real or
  // sparse vectors, whose sums went to FP64 without it (4x4 6+6 real 11.0 ms, now
  // 4.14, 99 % zeros 4.38).  It shares the branch that grows the sums: one of its
  // own cost every vector 1.2 % (3.96 -> 4.01 ms, now 3.94), a loop of its own for
  // the warps that need it spilled (4.07).
  template <int N, typename Look>
  __device__ __forceinline__ void shifts(int (&sr)[N], int (&si)[N], Look look) {
    constexpr bool kLook = !std::is_same<Look, std::nullptr_t>::value;
    int any = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      sr[k] = re.e - sr[k];
      si[k] = im.e - si[k];
      any |= sr[k] | si[k];
    }
    if ((kLook ? any | (min(re.e, im.e) - (kISumLeast + 1)) : any) < 0) {  // rare after the first terms
      if (!kLook || any < 0) {
        const int er = re.e, ei = im.e;
        int lr = sr[0], li = si[0];
#pragma unroll
        for (int k = 1; k < N; ++k) {
          lr = min(lr, sr[k]);
          li = min(li, si[k]);
        }
        re.grow(lr);
        im.grow(li);
#pragma unroll
        for (int k = 0; k < N; ++k) {
          sr[k] += re.e - er;
          si[k] += im.e - ei;
        }
      }
      if constexpr (kLook) {
        if (min(re.e, im.e) <= kISumLeast) look();
      }
    }
  }

  static __device__ __forceinline__ void part(const ISumForm& f, double v, int s, int hop, int& hi,
                                              int& lo) {
    const uint32_t h = (uint32_t)__double2hiint(v), l = (uint32_t)__double2loint(v);
    const uint32_t th = __funnelshift_l(l, h, 11) | 0x80000000u;
    const unsigned long long r =
        shr_clamp(((unsigned long long)th << 32) | (l * f.by11), (uint32_t)(s + f.base - 3));
    isum_parts(r, ((int)h >> 31) * (2 * hop) + hop, hi, lo);
  }
};

}  // namespace mb
