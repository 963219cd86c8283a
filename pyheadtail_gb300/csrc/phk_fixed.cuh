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

// What add_digits leaves: of a value below the window, the bits above the unit go
// to the digits and the rest is returned, too small to cost the sum that it is
// added to a rounding of its own; other values are returned whole.
static __device__ __noinline__ double add_outside(int* d, int base, double u) {
    const int hi = __double2hiint(u);
    const int drop = base - biased_exp(hi);          // bits below the unit
    if (drop < 1 || drop > 52 || base == kNoBase) return u;
    const u64 w = ((u64)((hi & 0xfffff) | 0x100000) << 32) | (unsigned)__double2loint(u);
    const long long v = hi < 0 ? -(long long)(w >> drop) : (long long)(w >> drop);
    atomicAdd(d, (int)((unsigned)v & kDigitMask));
    atomicAdd(d + 1, (int)((unsigned)(v >> 19) & kDigitMask));
    atomicAdd(d + 2, (int)((unsigned)(v >> 38) & kDigitMask));
    atomicAdd(d + 3, (int)(v >> 57));
    // u without the bits that were added
    const u64 bits = (u64)__double_as_longlong(u) & (~0ull << drop);
    return u - __longlong_as_double((long long)bits);
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

// the FP64 value of the digits at d, rounded once to nearest (integer work: with
// two conversions and three FP64 instructions, 89 cycles of a warp, the end of a
// pass over 1e5 particles in 1000 slices took 7 us more)
__device__ __forceinline__ double digits_value(const int* d, int base) {
    const long long h = (long long)d[3] * (1 << kDigitBits) + (unsigned)d[2];
    const u64 l = ((u64)(unsigned)d[1] << kDigitBits) + (unsigned)d[0];
    // h 2^38 + l in 128 bits, its magnitude
    u64 lo = ((u64)h << 38) + l;
    u64 hi = (u64)(h >> 26) + (lo < l ? 1u : 0u);
    if ((hi | lo) == 0) return 0.0;
    const unsigned sign = (unsigned)(hi >> 32) & 0x80000000u;
    if (sign) {
        lo = 0 - lo;
        hi = ~hi + (lo == 0 ? 1u : 0u);
    }
    // its top 64 bits, whether anything is below them, and 53 bits of it
    const int lz = hi ? __clzll((long long)hi) : 64 + __clzll((long long)lo);
    const u64 top = hi ? (hi << lz) | (lo >> (64 - lz)) : lo << (lz - 64);
    const unsigned below = hi && (lo << lz) != 0 ? 1u : 0u;
    u64 r = top >> 11;
    r += (((unsigned)top & 0x7ffu) << 1 | below) + ((unsigned)r & 1u) > 0x800u ? 1u : 0u;
    r += (u64)(unsigned)(74 - lz + base) << 52;      // r 2^(75 - lz + base - 1075)
    return __hiloint2double((int)((unsigned)(r >> 32) | sign), (int)r);
}
// the unit of the digits, and the FP64 value of a top digit that was taken out
__device__ __forceinline__ double digit_unit(int base) {
    return __hiloint2double((base - 52) << 20, 0);
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
    int any;              // a value was added
};
__device__ __forceinline__ void spill64(Spill64* sp, int q, int s, double u) {
    if (u != 0.0) {
        sp->any = 1;
        atomicAdd(sp->sum[q] + s * sp->stride, u);
    }
}
static __device__ __noinline__ void outside64(Spill64* sp, int q, int s, int* d,
                                              int base, double u) {
    spill64(sp, q, s, add_outside(d, base, u));
}

struct FixHist64 {
    int* w;               // [S][kFix64Words]
    Spill64* sp;          // in shared memory
    int base[2];          // windows of x and y (digit_base)

    __device__ __forceinline__ void add_q(int q, int s, double u) const {
        int* d = w + s * kFix64Words + 1 + 4 * q;
        if (!add_digits(d, base[q], u)) outside64(sp, q, s, d, base[q], u);
    }
    __device__ __forceinline__ void add(int s, double x, double y) const {
        atomicAdd(w + s * kFix64Words, 1);
        add_q(0, s, x);
        add_q(1, s, y);
    }
};

// -------------------------------------------------------------------
// FixHist32: the same for the FP32 coordinates of a batch's bunch (one CTA, in
// the bunch's partial column).  A float is split by adding and subtracting
// 1.5 2^23 units: the low bits of the sum are the value in these units, so the
// sum itself, as an integer, goes to the counter, and the constant is taken off
// at the end, once per value.  Three digits, units 2^36, 2^18 and 1, of at most
// 2^17; the last unit is 2^-42 of the typical value, so that floats from 2^-19
// to 2^11 times it leave no remainder.  Others are added to the column in FP64.
// -------------------------------------------------------------------
// a value outside the window (its digits are the constants)
static __device__ __noinline__ void outside32(int* d, int S, float top, const Spill64* sp,
                                              int q, int s, float u) {
    atomicAdd(d, __float_as_int(top));
    atomicAdd(d + S, __float_as_int(top * 0x1p-18f));
    atomicAdd(d + 2 * S, __float_as_int(top * 0x1p-36f));
    if (u != 0.0f) atomicAdd(sp->sum[q] + s * sp->stride, (double)u);
}

constexpr int kDigitValues32 = 16380;   // at most, between two carries

struct FixHist32 {
    int* cnt;             // [S]
    int* dig;             // [6][S]: x top, middle, low, y
    const Spill64* sp;    // in shared memory
    int S;
    float top[2];         // 1.5 2^23 units of the top digit (digit_top)

    __device__ __forceinline__ void add_q(int q, int s, float u) const {
        const float H = top[q], M = H * 0x1p-18f, L = H * 0x1p-36f;
        const float h = __fadd_rn(u, H), r = __fsub_rn(u, __fsub_rn(h, H));
        const float m = __fadd_rn(r, M), e = __fsub_rn(r, __fsub_rn(m, M));
        const float l = __fadd_rn(e, L);
        int* d = dig + 3 * q * S + s;
        if (fabsf(u) < H * (1.0f / 128.0f) && __fsub_rn(l, L) == e) {
            atomicAdd(d, __float_as_int(h));
            atomicAdd(d + S, __float_as_int(m));
            atomicAdd(d + 2 * S, __float_as_int(l));
        } else {
            outside32(d, S, H, sp, q, s, u);
        }
    }
    __device__ __forceinline__ void add(int s, float x, float y) const {
        atomicAdd(cnt + s, 1);
        add_q(0, s, x);
        add_q(1, s, y);
    }
};

// FixHist32::top for a typical magnitude (float bits; 0: none seen, nothing is
// within the window)
__device__ __forceinline__ float digit_top(unsigned bits) {
    if (bits == 0u) return 0.0f;
    const int e = (int)(bits >> 23) - 127;
    return ldexpf(1.5f, (e < -106 ? -106 : (e > 100 ? 100 : e)) + 17);
}
// the last digit's unit
__device__ __forceinline__ double digit_unit32(float top) {
    const int k = (__float_as_int(top) >> 23) - 127;         // top = 1.5 2^k
    return top == 0.0f ? 0.0 : __hiloint2double((k - 59 + 1023) << 20, 0);
}
// the digits of a slice with n values, without the constants
__device__ __forceinline__ void digits32(const int* d, int S, float top, int n, int (&v)[3]) {
    v[0] = (int)((unsigned)d[0] - (unsigned)n * __float_as_uint(top));
    v[1] = (int)((unsigned)d[S] - (unsigned)n * __float_as_uint(top * 0x1p-18f));
    v[2] = (int)((unsigned)d[2 * S] - (unsigned)n * __float_as_uint(top * 0x1p-36f));
}
__device__ __forceinline__ double digits32_value(const int* d, int S, float top, int n) {
    int v[3];
    digits32(d, S, top, n, v);
    const long long h = ((long long)v[0] << 18) + v[1];
    return fma((double)h, 0x1p18, (double)v[2]) * digit_unit32(top);
}

// Carries the digits of the slices with more than `most` values, at least every
// kDigitValues32 values; a top digit that might overflow before the next carry
// goes to the column (all threads)
static __device__ __noinline__ void carry_slices32(const int* cnt, int* dig, int S, int most,
                                                   const Spill64* sp, const unsigned* typ) {
    __syncthreads();
    for (int s = threadIdx.x; s < S; s += blockDim.x) {
        const int n = cnt[s];
        if (n <= most) continue;
        for (int q = 0; q < 2; ++q) {
            const float top = digit_top(typ[q]);
            int* d = dig + 3 * q * S + s;
            int v[3];
            digits32(d, S, top, n, v);
            const int c2 = v[2] >> 18, c1 = (v[1] + c2) >> 18;
            int c0 = c1;
            if (v[0] + c1 >= (1 << 29) || v[0] + c1 <= -(1 << 29)) {
                c0 = -v[0];
                atomicAdd(sp->sum[q] + s * sp->stride,
                          (double)(v[0] + c1) * 0x1p36 * digit_unit32(top));
            }
            d[0] = (int)((unsigned)d[0] + (unsigned)c0);
            d[S] = (int)((unsigned)d[S] + (unsigned)(c2 - c1 * (1 << 18)));
            d[2 * S] = (int)((unsigned)d[2 * S] - (unsigned)(c2 * (1 << 18)));
        }
    }
    __syncthreads();
}

// A window that is set after the bunch's first tiles: their values (zeros, or
// in the column already) count as the constants (all threads)
static __device__ __noinline__ void open_digits32(const int* cnt, int* dig, int S, float top) {
    for (int s = threadIdx.x; s < S; s += blockDim.x) {
        const unsigned n = (unsigned)cnt[s];
        dig[s] = (int)(n * __float_as_uint(top));
        dig[S + s] = (int)(n * __float_as_uint(top * 0x1p-18f));
        dig[2 * S + s] = (int)(n * __float_as_uint(top * 0x1p-36f));
    }
}

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

// the bits of |u|; 0 for infinity and NaN
__device__ __forceinline__ unsigned finite_high(float u) {
    const unsigned b = __float_as_uint(u) & 0x7fffffffu;
    return b < 0x7f800000u ? b : 0u;
}

// The median of what the warps saw at most (v: lane w holds warp w's), of those
// that saw something: a few stray values, or warps that hold none, do not set it.
// All lanes of a warp call it.
template <int WARPS>
__device__ __forceinline__ unsigned typical_of(unsigned v) {
    const int lane = threadIdx.x & 31;
    if (lane >= WARPS) v = 0u;
    int rank = 0;
#pragma unroll
    for (int j = 0; j < WARPS; ++j) {
        const unsigned o = __shfl_sync(0xffffffffu, v, j);
        rank += o > v || (o == v && j < lane);
    }
    const int seen = __popc(__ballot_sync(0xffffffffu, v != 0u));
    const unsigned at = __ballot_sync(0xffffffffu, lane < WARPS && rank == (seen - 1) / 2);
    return seen ? __shfl_sync(0xffffffffu, v, __ffs(at) - 1) : 0u;
}

// What the warps of a CTA saw at most of x and y: of a sample of the inputs,
// and of the outputs of a tile
template <int WARPS>
struct Seen {
    unsigned in[2][WARPS], out[2][WARPS];
};
template <int WARPS>
__device__ __forceinline__ void note_seen(unsigned (*to)[WARPS], unsigned mx, unsigned my) {
    mx = __reduce_max_sync(0xffffffffu, mx);
    my = __reduce_max_sync(0xffffffffu, my);
    if ((threadIdx.x & 31) == 0) {
        to[0][threadIdx.x >> 5] = mx;
        to[1][threadIdx.x >> 5] = my;
    }
}

// The typical magnitudes (0: none yet) from the sample of the inputs and the
// outputs of this tile, of every warp the larger (a bunch that starts on the
// axis, a large beta at the end of the turn); where all are zero they stay open
// and the next tile is looked at.  mx, my: the largest of this thread's outputs.
// All threads of the CTA call it; true if one is still open.  Out of line, as
// everything in the tile loop that seldom runs: the loop fills the instruction
// cache as it is (inlined, these parts cost 5 % of a pass).
template <int WARPS>
__device__ __noinline__ bool find_typical(Seen<WARPS>* seen, unsigned* typ, unsigned mx,
                                          unsigned my) {
    note_seen<WARPS>(seen->out, mx, my);
    __syncthreads();
    const int q = (threadIdx.x >> 5) & 1, w = threadIdx.x & (WARPS - 1);
    const unsigned t = typical_of<WARPS>(max(seen->in[q][w], seen->out[q][w]));
    if ((threadIdx.x & ~32u) == 0 && typ[q] == 0u) typ[q] = t;
    __syncthreads();
    return typ[0] == 0u || typ[1] == 0u;
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
    int32_t span;       // RF kick: exponents of z that the fixed-point sine takes
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
    k->span = 0;
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
