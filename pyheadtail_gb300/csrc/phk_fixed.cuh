// FP64 work on the integer pipes.  GB300 starts one FP64 addition,
// multiplication or multiply-add of a warp every 19 cycles per SM and a
// conversion every 16 (measured), an integer instruction every half cycle, so
// whatever a plain-form kernel can evaluate exactly, or to more than 53 bits,
// in 64-bit integers is cheaper there, and runs beside the FP64 pipe.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace phk {

typedef unsigned long long u64;

// The significand of a normal double, left-aligned in 64 bits: with its
// biased exponent e, |v| = mant64 * 2^(e - 1086).
__device__ __forceinline__ u64 mant64(int hi, int lo) {
    const unsigned h = __funnelshift_l((unsigned)lo, (unsigned)hi, 11) | 0x80000000u;
    return ((u64)h << 32) | ((unsigned)lo << 11);
}
__device__ __forceinline__ int biased_exp(int hi) { return (hi >> 20) & 0x7ff; }

// v >> r for any r >= 0 (0 from 64 on; the PTX shift clamps its amount)
__device__ __forceinline__ u64 shr_clamp(u64 v, int r) {
    u64 o;
    asm("shr.u64 %0, %1, %2;" : "=l"(o) : "l"(v), "r"(r));
    return o;
}

// -------------------------------------------------------------------
// FP64 product on the integer pipes, correctly rounded (to nearest, ties to
// even): the same bits as __dmul_rn for normal operands and a normal result.
// A factor is its left-aligned significand and its sign and exponent bits.
// About 26 integer instructions.
// -------------------------------------------------------------------
struct Factor {
    unsigned hi, lo;    // significand, top bit set
    int e;              // sign and exponent bits of the high word
};
__host__ __device__ inline Factor factor_bits(unsigned hi, unsigned lo) {
    return Factor{0x80000000u | (hi << 11) | (lo >> 21), lo << 11,
                  (int)(hi & 0xfff00000u)};
}
__device__ __forceinline__ Factor factor_of(double v) {
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    return Factor{__funnelshift_l(lo, hi, 11) | 0x80000000u, lo << 11,
                  (int)(hi & 0xfff00000u)};
}
// magnitude outside [2^-256, 2^256) (zeros, subnormals, infinities and NaN
// among them): one of the top three bits of the result
__device__ __forceinline__ unsigned off_centre(double v) {
    return ((unsigned)__double2hiint(v) & 0x7fffffffu) - (767u << 20);
}
constexpr unsigned kOffCentre = 0xe0000000u;
// magnitude in [2^-511, 2^512): bit 30 of the result (zeros, subnormals,
// infinities and NaN clear it)
__device__ __forceinline__ unsigned mid_range(double v) {
    return (unsigned)__double2hiint(v) + 0x20000000u;
}

__device__ __forceinline__ double mul_int(const Factor& a, const Factor& b) {
    const u64 p0 = (u64)a.lo * b.lo;
    const u64 p1 = (u64)a.hi * b.lo + (p0 >> 32);
    const u64 p2 = (u64)a.lo * b.hi + (unsigned)p1;
    const u64 p3 = (u64)a.hi * b.hi + (p1 >> 32) + (p2 >> 32);
    const unsigned h = (unsigned)(p3 >> 32), l = (unsigned)p3;
    // 53 bits of the product, the rest and whether anything is below it
    const int top = (int)(h >> 31), s = 10 + top;
    unsigned ml = __funnelshift_r(l, h, s), mh = h >> s;
    const unsigned rest = (l << (32 - s)) | (((unsigned)p0 | (unsigned)p2) != 0u ? 1u : 0u);
    const unsigned up = rest + (ml & 1u) > 0x80000000u ? 1u : 0u;
    ml += up;
    mh += ml < up ? 1u : 0u;
    return __hiloint2double((int)mh + a.e + b.e + (top << 20) - (1024 << 20), (int)ml);
}

// the product as a factor again, 63 bits and more of it (truncated)
__device__ __forceinline__ Factor mul_factor(const Factor& a, const Factor& b) {
    u64 p = __umul64hi(((u64)a.hi << 32) | a.lo, ((u64)b.hi << 32) | b.lo);
    const int top = (int)(p >> 63);
    p <<= 1 - top;
    return Factor{(unsigned)(p >> 32), (unsigned)p,
                  a.e + b.e + (top << 20) - (1023 << 20)};
}

// -------------------------------------------------------------------
// Exact sums of doubles as fixed-point integers.
//
// A value u = w 2^(e - 1075) (w: its signed 53-bit significand, e: its biased
// exponent) is the integer w 2^(e - base) of at most 74 bits and a sign, where
// base <= e <= base + 21; it is split into three unsigned 19-bit digits and the
// signed rest, added to 32-bit counters.  Nothing is rounded, so the sum of such
// values is exact and does not depend on their order.  Every other value (far
// from the typical value that sets the base, subnormal, infinite, NaN) is left
// to the caller, who adds it in FP64: a sum is never less accurate than a
// floating-point loop's.  (A 64-bit number that truncates what lies below its
// unit took 5 cycles less of a warp's 41 per particle, but lost slices whose
// values are all small.  Digits with the sign, by multiplication, are 2 cycles
// shorter but hold half as many values, and the pass's multiply pipe is busier
// than its logic pipe.)
// -------------------------------------------------------------------
constexpr int kDigitBits = 19;
constexpr unsigned kDigitMask = (1u << kDigitBits) - 1u;
constexpr int kWindow = 21;
constexpr int kDigitValues = 8190;      // at most, between two carries
constexpr int kNoBase = 1 << 16;        // no value is representable

// base for a typical magnitude, given as the high word of the double (sign
// cleared; 0: none seen): down to 2^-low of it
__device__ __forceinline__ int digit_base(unsigned mhi, int low) {
    if (mhi == 0u) return kNoBase;
    const int e = (int)(mhi >> 20);
    return (e < 100 ? 100 : (e > 2000 ? 2000 : e)) - low;
}

// adds u to the four digits at d (shared memory); false if it is not
// representable
__device__ __forceinline__ bool add_digits(int* d, int base, double u) {
    const int hi = __double2hiint(u);
    const unsigned wl = (unsigned)__double2loint(u);
    const int s = biased_exp(hi) - base;
    if ((unsigned)s > (unsigned)kWindow) return false;
    const int sign = hi >> 31;
    const long long w = ((((long long)((hi & 0xfffff) | 0x100000)) << 32 | wl) ^ sign) - sign;
    const unsigned w0 = (unsigned)w;
    const int w1 = (int)(w >> 32);
    const unsigned v0 = w0 << s, v1 = __funnelshift_l(w0, (unsigned)w1, s);
    const int v2 = (w1 >> (32 - kWindow)) >> (kWindow - s);
    atomicAdd(d, (int)(v0 & kDigitMask));
    atomicAdd(d + 1, (int)(__funnelshift_r(v0, v1, 19) & kDigitMask));
    atomicAdd(d + 2, (int)((v1 >> 6) & kDigitMask));
    atomicAdd(d + 3, (int)__funnelshift_r(v1, (unsigned)v2, 25));
    return true;
}

// carries the digits at d upwards, at least every kDigitValues values; a top
// digit that might overflow before the next carry is taken out and returned
// (in units of 2^57)
__device__ __forceinline__ int carry_digits(int* d) {
    u64 c = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        c += (unsigned)d[i];
        d[i] = (int)((unsigned)c & kDigitMask);
        c >>= kDigitBits;
    }
    const int top = d[3] + (int)c;
    const int out = top >= (1 << 29) || top <= -(1 << 29) ? top : 0;
    d[3] = top - out;
    return out;
}

// the FP64 value of the digits at d and of a top digit that was taken out
__device__ __forceinline__ double digit_unit(int base) {
    return __hiloint2double(((base == kNoBase ? 1023 : base) - 52) << 20, 0);
}
__device__ __forceinline__ double digits_value(const int* d, int base) {
    const long long h = (long long)d[3] * (1 << kDigitBits) + (unsigned)d[2];
    const long long l = ((long long)(unsigned)d[1] << kDigitBits) + (unsigned)d[0];
    return fma((double)h, 0x1p38, (double)l) * digit_unit(base);
}
__device__ __forceinline__ double top_value(int top, int base) {
    return (double)top * 0x1p57 * digit_unit(base);
}

// -------------------------------------------------------------------
// FixHist64: per-slice counts and sums of x and y of one CTA in shared memory,
// as the digits above; values outside the window go to the CTA's (cluster's)
// partial column in global memory, FP64 atomics.
//
// What it replaces: warp-private FP64 histograms, whose lanes were
// serialised by bids in shared memory, two FP64 additions for each round
// whatever the number of lanes left (19 cycles of the FP64 pipe each, 2 to
// 5 rounds at 500 to 50 slices).
// -------------------------------------------------------------------
constexpr int kFix64Words = 9;   // per slice: count, 4 digits of x, 4 of y

struct Spill64 {
    double* sum[2];       // of x and y in the partial column
    int64_t stride;       // between slices
};
static __device__ __noinline__ void spill64(const Spill64* sp, int q, int s, double u) {
    if (u != 0.0) atomicAdd(sp->sum[q] + s * sp->stride, u);
}

struct FixHist64 {
    int* w;               // [S][kFix64Words]
    const Spill64* sp;    // in shared memory
    int base[2];          // windows of x and y (digit_base)

    __device__ __forceinline__ void add_q(int q, int s, double u) const {
        if (!add_digits(w + s * kFix64Words + 1 + 4 * q, base[q], u)) spill64(sp, q, s, u);
    }
    __device__ __forceinline__ void add(int s, double x, double y) const {
        atomicAdd(w + s * kFix64Words, 1);
        add_q(0, s, x);
        add_q(1, s, y);
    }
};

// -------------------------------------------------------------------
// The typical magnitude that sets a CTA's window.
// -------------------------------------------------------------------

// Particle of this thread in a sample of those that the CTA works on, the
// tiles blockIdx.x, blockIdx.x + gridDim.x, ... of TILE particles; -1 if it has
// none.  Every warp looks into another tile, spread over all of them: in a
// bunch that is ordered by a coordinate, the first tile is no sample.  (A warp's
// 32 from as many tiles cost 6 us of a pass over 1e7 particles.)
template <int THREADS, int TILE>
__device__ __forceinline__ int64_t own_sample(int tid, int64_t n) {
    const int64_t tiles = (n + TILE - 1) / TILE;
    if ((int64_t)blockIdx.x >= tiles) return -1;
    const int64_t own = (tiles - 1 - blockIdx.x) / gridDim.x + 1;
    const int64_t it = (tid >> 5) * own / (THREADS / 32);
    const int64_t i = (blockIdx.x + it * gridDim.x) * TILE + tid;
    return i < n ? i : -1;
}

// the high word of |u|; 0 for zero, infinity and NaN
__device__ __forceinline__ unsigned finite_high(double u) {
    const unsigned b = (unsigned)__double2hiint(u) & 0x7fffffffu;
    return b < 0x7ff00000u ? b : 0u;
}

// The median of what the warps saw at most, of those that saw something: a few
// stray values, or warps that hold none, do not set it.  most: WARPS entries in
// shared memory; all lanes of a warp call it.
template <int WARPS>
__device__ __forceinline__ unsigned typical_of(const unsigned* most) {
    const int lane = threadIdx.x & 31;
    const unsigned v = lane < WARPS ? most[lane] : 0u;
    int rank = 0;
    for (int j = 0; j < WARPS; ++j) {
        const unsigned o = __shfl_sync(0xffffffffu, v, j);
        rank += o > v || (o == v && j < lane);
    }
    const int seen = __popc(__ballot_sync(0xffffffffu, v != 0u));
    const unsigned at = __ballot_sync(0xffffffffu, lane < WARPS && rank == (seen - 1) / 2);
    return seen ? __shfl_sync(0xffffffffu, v, __ffs(at) - 1) : 0u;
}

// -------------------------------------------------------------------
// Sine and cosine of 2 pi F 2^-64, F an unsigned 64-bit fraction of a turn
// (the integer turns drop out by themselves), in units of 2^-62.
//
// The quarter wave is tabulated at 1025 points (shared memory, 8 KB); the
// remainder theta < 2 pi / 4096 enters through angle addition,
//   S cos(theta) + C sin(theta) = S + C sin(theta) - S (1 - cos(theta)),
// with the Maclaurin series sin(theta) = theta - theta^3/6 + theta^5/120 and
// 1 - cos(theta) = theta^2/2 - theta^4/24 (next terms 4e-24 and 2e-20).
// Fixed point throughout: the absolute error is below 2^-61 (4e-19), the
// table's rounding and one truncation per product; a double near 1 resolves
// 1.1e-16.  Measured per warp: 42 cycles for the sine, 54 for sine and cosine
// with their conversions; the library's sin takes 21 FP64 multiply-adds
// (about 400 cycles).
// -------------------------------------------------------------------
constexpr int kSineEntries = 1025;
__device__ static const u64 kSineQuarter[kSineEntries] = {
#include "phk_sine_table.inc"
};

// copies the table to shared memory (all threads; a barrier must follow)
__device__ __forceinline__ void stage_sine(u64* tab, int tid, int nthreads) {
    for (int i = tid; i < kSineEntries; i += nthreads) tab[i] = kSineQuarter[i];
}

struct SineParts {
    u64 s, c;       // table values of the quarter wave at j and 1024 - j
    u64 th;         // sin(theta), units of 2^-73
    u64 q;          // 1 - cos(theta), units of 2^-82
};

// u: a quarter turn or less, units of 2^-64 turn
__device__ __forceinline__ SineParts sine_parts(const u64* tab, u64 u) {
    SineParts p;
    const int j = (int)(u >> 52);
    p.s = tab[j];
    p.c = tab[(kSineEntries - 1) - j];
    // theta = 2 pi (u mod 2^52) 2^-64 in units of 2^-73: 2 pi 2^61 = 0xc90f...
    const u64 th = __umul64hi(u << 12, 0xc90fdaa22168c235ull);
    const u64 t2 = __umul64hi(th, th);                  // theta^2, 2^-82
    const unsigned t2h = (unsigned)(t2 >> 32);          // 2^-50
    const unsigned t4 = __umulhi(t2h, t2h);             // theta^4, 2^-68
    // theta^2/6 - theta^4/120 in units of 2^-52 (4/6 = 0xaaaaaaab 2^-32,
    // 2^-16/120 = 546 2^-32)
    const unsigned e = __umulhi(t2h, 0xaaaaaaabu) - (((t4 >> 16) * 546u) >> 16);
    const u64 x3 = (u64)(unsigned)(th >> 32) * e;       // 2^-93
    p.th = th - (x3 >> 20);
    // theta^4/24: 2^14/24 = 44739243 2^-16
    p.q = (t2 >> 1) - (((u64)t4 * 44739243u) >> 16);
    return p;
}

// m 2^-62 with the given sign bit as a double, rounded to nearest (integer
// work: a conversion takes the FP64 pipe 16 cycles); 0 for m = 0
__device__ __forceinline__ double unit_double(u64 m, unsigned sign) {
    const int lz = __clzll((long long)m);
    const u64 f = m << lz;                       // top bit set
    const u64 r = (f >> 11) + ((f >> 10) & 1ull);
    const unsigned e = (unsigned)(1023 - lz) << 20;   // the top bit of r adds one
    const double v = __hiloint2double((int)((unsigned)(r >> 32) + e | sign), (int)r);
    return m ? v : 0.0;
}

// the same as a factor with 64 significant bits (m = 0: as 2^-62)
__device__ __forceinline__ Factor unit_factor(u64 m, unsigned sign) {
    m = m ? m : 1ull;
    const int lz = __clzll((long long)m);
    const u64 f = m << lz;
    return Factor{(unsigned)(f >> 32), (unsigned)f, (int)(((1024 - lz) << 20) | sign)};
}

// sine, times 2^62, as magnitude and sign bit
__device__ __forceinline__ u64 sine_turn(const u64* tab, u64 F, unsigned* sign) {
    // the second and third quarters mirror about a quarter turn
    const unsigned fh = (unsigned)(F >> 32);
    if ((fh ^ (fh << 1)) & 0x80000000u) F = 0x8000000000000000ull - F;
    const bool neg = (long long)F < 0;
    const SineParts p = sine_parts(tab, neg ? 0ull - F : F);
    const long long d = (long long)(__umul64hi(p.c, p.th) -
                                    (__umul64hi(p.s, p.q) >> 9));   // 2^-71
    const long long r = (long long)p.s + ((d + 256) >> 9);
    *sign = neg ? 0x80000000u : 0u;
    return (u64)(r < 0 ? 0 : r);
}

// sine and cosine, times 2^62, as magnitudes and sign bits
struct SinCos {
    u64 s, c;
    unsigned ns, nc;
};
__device__ __forceinline__ SinCos sincos_turn(const u64* tab, u64 F) {
    const SineParts p = sine_parts(tab, F & 0x3fffffffffffffffull);
    const long long d1 = (long long)(__umul64hi(p.c, p.th) -
                                     (__umul64hi(p.s, p.q) >> 9));   // 2^-71
    const long long d2 = (long long)(__umul64hi(p.s, p.th) +
                                     (__umul64hi(p.c, p.q) >> 9));
    const long long a = (long long)p.s + ((d1 + 256) >> 9);
    const long long b = (long long)p.c - ((d2 + 256) >> 9);
    const u64 sn = (u64)(a < 0 ? 0 : a), cs = (u64)(b < 0 ? 0 : b);
    // quadrants: (sn, cs), (cs, -sn), (-sn, -cs), (-cs, sn)
    const unsigned k = (unsigned)(F >> 62);
    return SinCos{(k & 1u) ? cs : sn, (k & 1u) ? sn : cs, (k & 2u) << 30,
                  ((k + 1u) & 2u) << 30};
}

// t turns (|t| < 2^31) as a fraction of a turn, truncated toward zero
__device__ __forceinline__ u64 turn_fraction(double t) {
    const int hi = __double2hiint(t), lo = __double2loint(t);
    const int r = 1022 - biased_exp(hi);
    const u64 m = mant64(hi, lo);
    u64 F = r >= 0 ? shr_clamp(m, r) : m << -r;
    if (hi < 0) F = 0ull - F;
    return F;
}

// A constant of the phase for turn_product: K = mant 2^-exp
struct TurnFactor {
    u64 mant;
    int32_t exp;
    int32_t reserved;
};

// num / den as 64 significant bits: the quotient and, from its exact
// remainder, what its rounding dropped (1 part in 2^64 against 2^53)
__host__ __device__ inline bool turn_factor(double num, double den, TurnFactor* k) {
    const double q = num / den;
    const double lo = fma(-q, den, num) / den;
    if (!(q > 1e-200 && q < 1e200)) return false;
    int e = 0;
    const double m = frexp(q, &e);            // q = m 2^e, m in [1/2, 1)
    k->mant = ((u64)(m * 9007199254740992.0) << 11) +
              (u64)(long long)rint(ldexp(lo, 64 - e));
    k->exp = 64 - e;
    k->reserved = 0;
    return true;
}

// an angle in radians as a fraction of a turn (1 / 2 pi in two doubles)
__host__ __device__ inline u64 angle_fraction(double rad) {
    const double inv = 0.15915494309189535, inv_lo = -9.839338337591243e-18;
    const double h = rad * inv;
    const double l = fma(rad, inv_lo, fma(rad, inv, -h));
    const double t = h - rint(h);             // exact, |t| <= 1/2
    return ((u64)(long long)rint(t * 9223372036854775807.0) << 1) +
           (u64)(long long)rint(l * 18446744073709551616.0);
}

// z K turns as a fraction of a turn, for a constant K = kmant 2^-kexp
// (kmant left-aligned) and |z K| < 2^31: the product of the significands
// keeps 62 bits and more, rounding nothing to 53
__device__ __forceinline__ u64 turn_product(double z, u64 kmant, int kexp) {
    const int hi = __double2hiint(z), lo = __double2loint(z);
    const u64 m = __umul64hi(mant64(hi, lo), kmant);
    const int r = 958 + kexp - biased_exp(hi);
    u64 F = r >= 0 ? shr_clamp(m, r) : m << -r;
    if (hi < 0) F = 0ull - F;
    return F;
}

}  // namespace phk
