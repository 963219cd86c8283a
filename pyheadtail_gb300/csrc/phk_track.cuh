// The FP32 fused track kernel, the batched track kernel and the element
// arithmetic of both forms as templates, with their launch helpers.  Included
// by the per-precision translation units (phk_track_f32.cu, phk_track_f64.cu),
// which instantiate and launch them, and by phk_kernels.cu for the host-side
// planning helpers.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <cooperative_groups.h>

#include <type_traits>

#include "phk_device.cuh"
#include "phk_fixed.cuh"
#include "phk_internal.h"

namespace phk {

// ===================================================================
// particle tiles: VEC particles per thread, one register array per
// coordinate; every op below works op-major / particle-minor, reading its
// parameters once per tile
// ===================================================================

template <typename T, int VEC>
struct Tile {
    T c[6][VEC];
};

// ===================================================================
// element arithmetic, plain FP64 form (reference evaluation order)
// ===================================================================

// An FP64 instruction takes its 19 cycles of the pipe even when a short
// branch around it is compiled to predication and it is predicated off (16
// of the 34 FP64 instructions a particle of the undetuned turn with RF were
// such dispersion terms).  The element functions of the plain form are
// therefore compiled twice: PLAIN for the common single-segment turn
// (program_plain64: no dispersion, constant energy, equal optics functions
// with alpha = 0 at both ends of a detuned segment), without any
// alternative, and in full for the op loop.

// Constants of an op's FP64 form that its parameter block holds in another
// shape: made once per launch (batched form: once per bunch and CTA).
struct OpFix {
    TurnFactor k;    // RF kick: h / C, turns per metre
    u64 off;         // RF kick: phase offset and lock, fraction of a turn
    double c[5];     // RF kick: (A / p0_new) 2^-62, p0_old / p0_new,
                     //   dp_inc / p0_new, h 2 pi / C, offset in radians
                     // drift: eta0 L
    Factor m[8];     // transverse: the matrix entries; detuned, J01 J10 J23 J32
    int32_t m_ok;    //   all within range
};
// amplitude detuning: with j = g u^2 + t u u' + b u'^2 (twice the action)
struct DetFix {
    double gx, tx, bx, gy, ty, by;
    double axx, axy, ayy, ayx;   // dQ_x = axx j_x + axy j_y, dQ_y likewise
    // factors of the products on the integer pipes: amplitude detuning gx,
    // gy, bx, by, axy, ayx; chromaticity of order one its two coefficients
    Factor m[6];
    int32_t m_ok;                // all within range
};

// v as a factor; false outside [2^-200, 2^200]
__host__ __device__ inline bool host_factor(double v, Factor* f) {
    u64 bits;
    memcpy(&bits, &v, sizeof(bits));
    *f = factor_bits((unsigned)(bits >> 32), (unsigned)bits);
    const int e = (int)(bits >> 52) & 0x7ff;
    return e > 1023 - 200 && e < 1023 + 200;
}

struct Aux64 {
    const u64* sine;     // staged quarter wave (stage_sine)
    const OpFix* op;     // by op
    const DetFix* det;   // by detuner
};

__host__ __device__ inline void op_fix(const phk_op& op, OpFix* r) {
    const double* p = op.p;
    const int f = op.flags;
    if (op.kind == PHK_OP_DRIFT) {
        r->c[0] = p[1] * p[2];
    } else if (op.kind == PHK_OP_TRANSVERSE && !(f & PHK_FLAG_DETUNED)) {
        r->m_ok = 1;
        for (int i = 0; i < 8; ++i) r->m_ok &= host_factor(p[i], r->m + i);
    } else if (op.kind == PHK_OP_TRANSVERSE) {
        r->m_ok = host_factor(p[9], r->m) & host_factor(p[10], r->m + 1) &
                  host_factor(p[13], r->m + 2) & host_factor(p[14], r->m + 3);
    } else if (op.kind == PHK_OP_RF_KICK) {
        double off = 0.0;
        if (f & PHK_FLAG_PHI_OFFSET) off += p[3];
        if (f & PHK_FLAG_PHI_LOCK) off += p[4];
        // no usable factor, an offset that is not finite or far beyond a turn:
        // every particle takes the library's sine
        const bool far = !turn_factor(p[0], p[2], &r->k) || !(fabs(off) < 0x1p31);
        if (far) r->k.exp = -(1 << 20);
        r->k.span = fabs(off) < 0x1p-8 ? 21 : 4096;
        r->off = far ? 0 : angle_fraction(off);
        r->c[0] = p[5] * p[12] * 0x1p-62;
        r->c[1] = p[6] == p[8] ? 1.0 : p[6] * p[12];
        r->c[2] = (f & PHK_FLAG_P_INC) ? p[7] * p[12] : 0.0;
        r->c[3] = p[0] * p[1] * p[11];
        r->c[4] = off;
    }
}

__host__ __device__ inline void det_fix(const phk_detuner& d, DetFix* f) {
    const double* c = d.c;
    if (d.kind == PHK_DET_CHROMA) {
        f->m_ok = d.nx == 1 && d.ny == 1 && d.zx == 0 && d.zy == 0 &&
                  host_factor(c[0], f->m) & host_factor(c[8], f->m + 1);
        return;
    }
    f->gx = c[4];
    f->tx = c[5];
    f->bx = c[6];
    f->gy = c[7];
    f->ty = c[8];
    f->by = c[9];
    f->axx = 0.5 * c[0] / c[10];
    f->axy = 0.5 * c[2] / c[10];
    f->ayy = 0.5 * c[1] / c[10];
    f->ayx = 0.5 * c[3] / c[10];
    f->m_ok = host_factor(f->gx, f->m) & host_factor(f->gy, f->m + 1) &
              host_factor(f->bx, f->m + 2) & host_factor(f->by, f->m + 3) &
              host_factor(f->axy, f->m + 4) & host_factor(f->ayx, f->m + 5);
}

// whether a program needs the quarter wave
static inline bool program_has_phase(const phk_program& prog) {
    for (int o = 0; o < prog.n_ops; ++o)
        if (prog.op[o].kind == PHK_OP_RF_KICK ||
            (prog.op[o].kind == PHK_OP_TRANSVERSE &&
             (prog.op[o].flags & PHK_FLAG_DETUNED)))
            return true;
    return false;
}

// whether a program is within the PLAIN form (see above)
static inline bool program_plain64(const phk_program& prog) {
    for (int o = 0; o < prog.n_ops; ++o) {
        const phk_op& op = prog.op[o];
        if (op.flags & (PHK_FLAG_DISPERSION | PHK_FLAG_SHRINK | PHK_FLAG_P_INC))
            return false;
        if (op.kind == PHK_OP_RF_KICK && op.p[6] != op.p[8]) return false;
        if (op.kind == PHK_OP_TRANSVERSE && (op.flags & PHK_FLAG_DETUNED)) {
            // I the unit matrix, J without diagonal, no cross terms
            if (op.ij_mask & ~(0x0609 | 0x6090)) return false;
            if (op.p[0] != 1.0 || op.p[3] != 1.0 || op.p[4] != 1.0 || op.p[7] != 1.0)
                return false;
            for (int d = 0; d < op.det_count; ++d) {
                const phk_detuner& t = prog.det[op.det_begin + d];
                if (t.kind == PHK_DET_AMPLITUDE && (t.c[5] != 0.0 || t.c[8] != 0.0))
                    return false;
            }
        }
    }
    return true;
}

// ChromaticitySegment detune: Horner with separately rounded steps, lowest
// coefficient first, then the extra dp factors of the order > 3 path.
__device__ __forceinline__ double chroma_poly(const double* c, int n, int z,
                                             double dp) {
    double r = c[n - 1];
    for (int i = n - 2; i >= 0; --i) r = add(c[i], mul(r, dp));
    r = mul(r, dp);
    for (int i = 0; i < z; ++i) r = mul(r, dp);
    return r;
}

// whether the fixed-point phase takes phi radians (below 2^12, finite)
__device__ __forceinline__ bool phase_near(double phi) {
    return biased_exp(__double2hiint(phi)) < 1035;
}
// sine and cosine of phi radians: phi / 2 pi as a fraction of a turn
// (1 / 2 pi = 0xa2f9... 2^-66)
__device__ __forceinline__ SinCos phase_sincos(const u64* tab, double phi) {
    return sincos_turn(tab, turn_product(phi, 0xa2f9836e4e44152aull, 66));
}
static __device__ __noinline__ void sincos_far(double phi, double* s, double* c) {
    sincos(phi, s, c);
}

// (u, u') through one plane's detuned map
__device__ __forceinline__ void detuned_plane(const double* I, const double* J,
                                              const u64* tab, double phi, double& u,
                                              double& up) {
    double s, c;
    if (phase_near(phi)) {
        const SinCos r = phase_sincos(tab, phi);
        s = unit_double(r.s, r.ns);
        c = unit_double(r.c, r.nc);
    } else {
        sincos_far(phi, &s, &c);
    }
    const double M00 = fma(I[0], c, J[0] * s), M01 = fma(I[1], c, J[1] * s);
    const double M10 = fma(I[2], c, J[2] * s), M11 = fma(I[3], c, J[3] * s);
    const double nu = fma(M00, u, M01 * up);
    up = fma(M10, u, M11 * up);
    u = nu;
}
// the same with unit I and J without diagonal, the products with the sine on
// the integer pipes: of u' and u, first the 64-bit product J s
__device__ __forceinline__ void detuned_plane_unit(const Factor* J, const SinCos& r,
                                                   const Factor& fu, const Factor& fup,
                                                   double& u, double& up) {
    const Factor s = unit_factor(r.s, r.ns);
    const double c = unit_double(r.c, r.nc);
    const double nu = fma(c, u, mul_int(mul_factor(J[0], s), fup));
    up = fma(c, up, mul_int(mul_factor(J[1], s), fu));
    u = nu;
}

// the tune with its detunings, each added as the reference adds them
__device__ __forceinline__ void detuned_tunes(const phk_op& op, const phk_program& prog,
                                              const Aux64& aux, bool cross, double x,
                                              double xp, double y, double yp, double dp,
                                              double& qx, double& qy) {
    qx = op.p[20];
    qy = op.p[21];
    for (int d = 0; d < op.det_count; ++d) {
        const phk_detuner& dt = prog.det[op.det_begin + d];
        if (dt.kind == PHK_DET_CHROMA) {
            qx = add(qx, chroma_poly(dt.c, dt.nx, dt.zx, dp));
            qy = add(qy, chroma_poly(dt.c + 8, dt.ny, dt.zy, dp));
        } else {
            const DetFix& f = aux.det[op.det_begin + d];
            double jx = f.gx * x, jy = f.gy * y;
            if (cross) {
                jx = fma(f.tx, xp, jx);
                jy = fma(f.ty, yp, jy);
            }
            jx = fma(jx, x, f.bx * xp * xp);
            jy = fma(jy, y, f.by * yp * yp);
            qx = add(qx, fma(f.axx, jx, f.axy * jy));
            qy = add(qy, fma(f.ayy, jy, f.ayx * jx));
        }
    }
}

// the detuned map of one particle u = (x, xp, y, yp, dp), all FP64
__device__ __forceinline__ void detuned_map(const phk_op& op, const phk_program& prog,
                                            const Aux64& aux, double& x, double& xp,
                                            double& y, double& yp, double qx, double qy) {
    const double* p = op.p;
    detuned_plane(p, p + 8, aux.sine, mul(qx, p[22]), x, xp);
    detuned_plane(p + 4, p + 12, aux.sine, mul(qy, p[22]), y, yp);
}
// out of line: particles with a zero, subnormal, huge or non-finite coordinate
// or a phase beyond the fixed point
static __device__ __noinline__ void detuned_map_cold(const phk_op& op,
                                                     const phk_program& prog,
                                                     const Aux64& aux, double* u) {
    double qx, qy;
    detuned_tunes(op, prog, aux, false, u[0], u[1], u[2], u[3], u[4], qx, qy);
    detuned_map(op, prog, aux, u[0], u[1], u[2], u[3], qx, qy);
}

// whether the products of a detuned segment's constants run on the integer
// pipes
__device__ __forceinline__ bool detuned_factors_ok(const phk_op& op, const Aux64& aux,
                                                   int o) {
    int ok = aux.op[o].m_ok;
    for (int d = 0; d < op.det_count; ++d) ok &= aux.det[op.det_begin + d].m_ok;
    return ok;
}

// the undetuned map, every product and sum rounded separately in the
// reference's order
__device__ __forceinline__ void linear_planes(const double* p, double& x, double& xp,
                                              double& y, double& yp) {
    const double nx = add(mul(p[0], x), mul(p[1], xp));
    const double nxp = add(mul(p[2], x), mul(p[3], xp));
    const double ny = add(mul(p[4], y), mul(p[5], yp));
    const double nyp = add(mul(p[6], y), mul(p[7], yp));
    x = nx; xp = nxp; y = ny; yp = nyp;
}
// out of line: particles with a zero, subnormal, huge or non-finite coordinate
static __device__ __noinline__ void linear_planes_cold(const double* p, double* u) {
    linear_planes(p, u[0], u[1], u[2], u[3]);
}

// TransverseSegmentMap.track, plain form.  Without detuners every product
// and sum is rounded separately in the reference's order.  With detuners the
// phase (Q + detunings) 2 pi is rounded as the reference rounds it; around
// the sine and cosine of a per-particle phase, which no evaluation
// reproduces bit for bit, the arithmetic is regrouped into few multiply-adds
// (constants from det_fix) and the sine and cosine are fixed-point.  With
// chromaticity and amplitude detuning, PLAIN: 36 FP64 instructions a
// particle, conversions included; before, about 110 and as many again in
// warps with a lane beyond the quarter radian of the former series (a turn
// of 1e6 macroparticles: 395 -> 122 us).
// DET (PLAIN): whether the segment is detuned
template <int VEC, bool PLAIN, bool DET = false>
__device__ __forceinline__ void op_transverse(const phk_op& op, int o,
                                              const phk_program& prog,
                                              const Aux64& aux,
                                              Tile<double, VEC>& t) {
    const double* p = op.p;
    const bool disp = !PLAIN && (op.flags & PHK_FLAG_DISPERSION);
    const double Dx0 = p[16], Dx1 = p[17], Dy0 = p[18], Dy1 = p[19];
    double (&x)[VEC] = t.c[PHK_X];
    double (&xp)[VEC] = t.c[PHK_XP];
    double (&y)[VEC] = t.c[PHK_Y];
    double (&yp)[VEC] = t.c[PHK_YP];
    const double (&dp)[VEC] = t.c[PHK_DP];
    if constexpr (PLAIN && DET) {
        // FP64 keeps the additions, the multiply-adds and the phase's product
        // (18 a particle of the segment's 36); products run on the integer
        // pipes
        const OpFix& f = aux.op[o];
        const unsigned off = detuned_factors_ok(op, aux, o) ? 0u : kOffCentre;
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            bool cold = ((off_centre(x[j]) | off_centre(xp[j]) | off_centre(y[j]) |
                          off_centre(yp[j]) | off_centre(dp[j]) | off) & kOffCentre) != 0u;
            if (!cold) {
                const Factor u = factor_of(x[j]), up = factor_of(xp[j]);
                const Factor v = factor_of(y[j]), vp = factor_of(yp[j]);
                double qx = p[20], qy = p[21];
                for (int d = 0; d < op.det_count; ++d) {
                    const phk_detuner& dt = prog.det[op.det_begin + d];
                    const DetFix& g = aux.det[op.det_begin + d];
                    if (dt.kind == PHK_DET_CHROMA) {
                        const Factor w = factor_of(dp[j]);
                        qx = add(qx, mul_int(g.m[0], w));
                        qy = add(qy, mul_int(g.m[1], w));
                    } else {
                        const double jx = add(mul_int(mul_factor(g.m[0], u), u),
                                              mul_int(mul_factor(g.m[2], up), up));
                        const double jy = add(mul_int(mul_factor(g.m[1], v), v),
                                              mul_int(mul_factor(g.m[3], vp), vp));
                        qx = add(qx, fma(g.axx, jx, mul_int(g.m[4], factor_of(jy))));
                        qy = add(qy, fma(g.ayy, jy, mul_int(g.m[5], factor_of(jx))));
                    }
                }
                const double phx = mul(qx, p[22]), phy = mul(qy, p[22]);
                if (phase_near(phx) && phase_near(phy)) {
                    detuned_plane_unit(f.m, phase_sincos(aux.sine, phx), u, up, x[j],
                                       xp[j]);
                    detuned_plane_unit(f.m + 2, phase_sincos(aux.sine, phy), v, vp, y[j],
                                       yp[j]);
                } else {
                    cold = true;
                }
            }
            if (cold) {
                double c[5] = {x[j], xp[j], y[j], yp[j], dp[j]};
                detuned_map_cold(op, prog, aux, c);
                x[j] = c[0]; xp[j] = c[1]; y[j] = c[2]; yp[j] = c[3];
            }
        }
        return;
    }
    // the detuning sees the coordinates before the dispersion is taken out
    const bool detuned = !PLAIN && (op.flags & PHK_FLAG_DETUNED);
    double qx[VEC], qy[VEC];
    if (detuned)
#pragma unroll
        for (int j = 0; j < VEC; ++j)
            detuned_tunes(op, prog, aux, true, x[j], xp[j], y[j], yp[j], dp[j], qx[j],
                          qy[j]);
    if (disp) {
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            x[j] = sub(x[j], mul(Dx0, dp[j]));
            y[j] = sub(y[j], mul(Dy0, dp[j]));
        }
    }
    if (detuned) {
#pragma unroll
        for (int j = 0; j < VEC; ++j)
            detuned_map(op, prog, aux, x[j], xp[j], y[j], yp[j], qx[j], qy[j]);
    } else if (PLAIN) {
        // the products on the integer pipes, the same bits (mul_int): eight
        // of the twelve FP64 instructions, which are what bounds the pass
        const OpFix& f = aux.op[o];
        const unsigned ok = f.m_ok ? 0x40000000u : 0u;
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            if (mid_range(x[j]) & mid_range(xp[j]) & mid_range(y[j]) &
                mid_range(yp[j]) & ok) {
                const Factor u = factor_of(x[j]), up = factor_of(xp[j]);
                const Factor v = factor_of(y[j]), vp = factor_of(yp[j]);
                x[j] = add(mul_int(f.m[0], u), mul_int(f.m[1], up));
                xp[j] = add(mul_int(f.m[2], u), mul_int(f.m[3], up));
                y[j] = add(mul_int(f.m[4], v), mul_int(f.m[5], vp));
                yp[j] = add(mul_int(f.m[6], v), mul_int(f.m[7], vp));
            } else {
                double c[4] = {x[j], xp[j], y[j], yp[j]};
                linear_planes_cold(p, c);
                x[j] = c[0]; xp[j] = c[1]; y[j] = c[2]; yp[j] = c[3];
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < VEC; ++j) linear_planes(p, x[j], xp[j], y[j], yp[j]);
    }
    if (disp) {
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            x[j] = add(x[j], mul(Dx1, dp[j]));
            y[j] = add(y[j], mul(Dy1, dp[j]));
        }
    }
}

template <int VEC>
__device__ __forceinline__ void op_drift(const phk_op& op,
                                         Tile<double, VEC>& t) {
    const double br = op.p[0], eta0 = op.p[1], L = op.p[2];
    const bool shrink = op.flags & PHK_FLAG_SHRINK;
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
        const double z = t.c[PHK_Z][j];
        const double zz = shrink ? mul(br, z) : z;
        t.c[PHK_Z][j] = sub(zz, mul(mul(eta0, t.c[PHK_DP][j]), L));
    }
}

// Drift of an RFSystems element (Drift, Kick, Drift), PLAIN: beside the
// kick's inexact sine, one multiply-add with eta0 L.  Other element
// sequences keep the separately rounded form above.
template <int VEC>
__device__ __forceinline__ void op_drift_rf(const OpFix& f, Tile<double, VEC>& t) {
#pragma unroll
    for (int j = 0; j < VEC; ++j)
        t.c[PHK_Z][j] = fma(-f.c[0], t.c[PHK_DP][j], t.c[PHK_Z][j]);
}

// The sine, times 2^62, of what the fixed point does not hold to 53 bits.  Phases
// below about 2^-10 without an offset (sine_turn's error is at most 2^-61,
// whatever the sine): the significand of the phase keeps its 62 bits, times 1 -
// theta^2/6 + theta^4/120 (next term 2^-66).  Phases of 2^9 turns and more, NaN,
// infinities, small phases beside a small offset: the library's sine.  One warp
// in forty comes here at a bunch length of a radian (1 % of a pass; without, the
// kick of a particle at a phase of 1e-10 was off by 4e-9 of itself).
static __device__ __noinline__ double rf_sine_cold(double z, u64 kmant, int kexp, double hk,
                                                   double off) {
    const int hi = __double2hiint(z), lo = __double2loint(z);
    const int be = biased_exp(hi);
    if (z == 0.0 && off == 0.0) return 0.0;
    if (off != 0.0 || be > 968 + kexp || be < 200) return sin(fma(hk, z, off)) * 0x1p62;
    const u64 m = __umul64hi(mant64(hi, lo), kmant);
    const int r = 958 + kexp - be;                        // phase: m 2^(-64 - r) turns
    const u64 th = __umul64hi(m, 0xc90fdaa22168c235ull);  // theta, units of 2^(-61 - r)
    const u64 x = shr_clamp(th, r - 5);                   // 2^-66
    const u64 q = __umul64hi(x, x);                       // theta^2, 2^-68
    const unsigned q4 = __umulhi((unsigned)(q >> 20), (unsigned)(q >> 20));   // 2^-64
    const u64 c = __umul64hi(q, 0x2aaaaaaaaaaaaaabull) -
                  ((u64)__umulhi(q4, 0x02222222u) << 4);
    const double s = (double)(th - (__umul64hi(th, c) >> 4));
    return __hiloint2double((__double2hiint(s) + ((1 - r) << 20)) | (hi & 0x80000000),
                            __double2loint(s));
}

// RF kick, plain form.  The per-particle sine makes the step inexact whatever
// the evaluation order, so the phase and its sine are fixed-point
// (turn_product, sine_turn) and the momentum update
//   dp' = (dp p0_old + A sin(phi) - dp_inc) / p0_new
// is dp (p0_old / p0_new) + (A / p0_new) sin(phi) - dp_inc / p0_new with
// the ratios formed once: two FP64 instructions a particle instead of 27.
template <int VEC, bool PLAIN>
__device__ __forceinline__ void op_rfkick(const phk_op& op, const OpFix& f,
                                          const u64* sine,
                                          Tile<double, VEC>& t) {
    const bool disp = !PLAIN && (op.flags & PHK_FLAG_DISPERSION);
    const double Dx = op.p[9], Dy = op.p[10];
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
        double& dp = t.c[PHK_DP][j];
        if (disp) {
            t.c[PHK_X][j] = sub(t.c[PHK_X][j], mul(Dx, dp));
            t.c[PHK_Y][j] = sub(t.c[PHK_Y][j], mul(Dy, dp));
        }
        const double z = t.c[PHK_Z][j];
        double s;      // sine, times 2^62
        if ((unsigned)(968 + f.k.exp - biased_exp(__double2hiint(z))) <= (unsigned)f.k.span) {
            unsigned sign;
            const u64 m = sine_turn(sine, turn_product(z, f.k.mant, f.k.exp) + f.off, &sign);
            s = (double)(long long)m;
            s = __hiloint2double((int)((unsigned)__double2hiint(s) | sign),
                                 __double2loint(s));
        } else {
            s = rf_sine_cold(z, f.k.mant, f.k.exp, f.c[3], f.c[4]);
        }
        if (PLAIN) dp = fma(f.c[0], s, dp);
        else dp = fma(dp, f.c[1], fma(f.c[0], s, -f.c[2]));
        if (disp) {
            t.c[PHK_X][j] = add(t.c[PHK_X][j], mul(Dx, dp));
            t.c[PHK_Y][j] = add(t.c[PHK_Y][j], mul(Dy, dp));
        }
    }
}

template <int VEC, bool PLAIN>
__device__ __forceinline__ void op_linear_long(const phk_op& op,
                                               Tile<double, VEC>& t) {
    const double* p = op.p;
    const double cs = p[0], sn = p[1], lf = p[2], Dx = p[3], Dy = p[4];
    const double ilf = p[5];
    const bool disp = !PLAIN && (op.flags & PHK_FLAG_DISPERSION);
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
        double& z = t.c[PHK_Z][j];
        double& dp = t.c[PHK_DP][j];
        if (disp) {
            t.c[PHK_X][j] = sub(t.c[PHK_X][j], mul(Dx, dp));
            t.c[PHK_Y][j] = sub(t.c[PHK_Y][j], mul(Dy, dp));
        }
        const double z0 = z, dp0 = dp;
        z = sub(mul(z0, cs), mul(mul(lf, dp0), sn));
        dp = add(mul(dp0, cs), mul(div_by(z0, lf, ilf), sn));
        if (disp) {
            t.c[PHK_X][j] = add(t.c[PHK_X][j], mul(Dx, dp));
            t.c[PHK_Y][j] = add(t.c[PHK_Y][j], mul(Dy, dp));
        }
    }
}

template <int VEC>
__device__ __forceinline__ void op_scale(const phk_op& op,
                                         Tile<double, VEC>& t) {
    const double f = op.p[0];
#pragma unroll
    for (int j = 0; j < VEC; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) t.c[q][j] = mul(t.c[q][j], f);
}

// the device means a damper op reads (phk_stats.means, FP64 then FP32)
__device__ __forceinline__ const double* damper_means(const phk_op& op) {
    unsigned long long bits;
    memcpy(&bits, &op.p[31], sizeof(bits));
    return reinterpret_cast<const double*>(bits);
}

// TransverseDamper.track_all (feedback/transverse_damper.py:64-86): the
// reference's order, xp -= (g sin) <xp>, then xp -= ((g cos) <x>) / beta
template <int VEC>
__device__ __forceinline__ void op_damper(const phk_op& op,
                                          Tile<double, VEC>& t) {
    const double* m = damper_means(op);
    const bool reactive = op.flags & PHK_FLAG_REACTIVE;
#pragma unroll
    for (int pl = 0; pl < 2; ++pl) {
        if (!(op.flags & (pl == 0 ? PHK_FLAG_DAMP_X : PHK_FLAG_DAMP_Y))) continue;
        const int u = pl == 0 ? PHK_X : PHK_Y, up = pl == 0 ? PHK_XP : PHK_YP;
        const double* g = op.p + 3 * pl;
        const double c1 = mul(g[0], __ldg(m + up));
        const double c2 = reactive ? __ddiv_rn(mul(g[1], __ldg(m + u)), g[2]) : 0.0;
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            t.c[up][j] = __dsub_rn(t.c[up][j], c1);
            if (reactive) t.c[up][j] = __dsub_rn(t.c[up][j], c2);
        }
    }
}

// ===================================================================
// element arithmetic, FP32 precision form (parameters packed as floats)
// ===================================================================

__device__ __forceinline__ float chroma_poly_f32(const float* c, int n, int z,
                                                 float dp) {
    float r = c[n - 1];
    for (int i = n - 2; i >= 0; --i) r = fmaf(r, dp, c[i]);
    r *= dp;
    for (int i = 0; i < z; ++i) r *= dp;
    return r;
}

// dq += the chromatic detuning of VEC particles (ChromaticitySegment.detune,
// trackers/detuners.py:64-98): Horner orders 1-3 inline, anything else
// through the general loop.  The branches are uniform.
template <int VEC>
__device__ __forceinline__ void chroma_add_f32(const float* c, int n, int z,
                                               const float (&dp)[VEC],
                                               float (&dq)[VEC]) {
    if (z == 0 && n == 1) {
#pragma unroll
        for (int j = 0; j < VEC; ++j) dq[j] = fmaf(c[0], dp[j], dq[j]);
    } else if (z == 0 && n == 2) {
#pragma unroll
        for (int j = 0; j < VEC; ++j)
            dq[j] = fmaf(fmaf(c[1], dp[j], c[0]), dp[j], dq[j]);
    } else if (z == 0 && n == 3) {
#pragma unroll
        for (int j = 0; j < VEC; ++j)
            dq[j] = fmaf(fmaf(fmaf(c[2], dp[j], c[1]), dp[j], c[0]), dp[j],
                         dq[j]);
    } else {
#pragma unroll
        for (int j = 0; j < VEC; ++j) dq[j] += chroma_poly_f32(c, n, z, dp[j]);
    }
}

// dqx, dqy += the detuning of VEC particles by one detuner
template <int VEC>
__device__ __forceinline__ void detune_f32(const phk_detuner& dt,
                                           const Tile<float, VEC>& t,
                                           float (&dqx)[VEC],
                                           float (&dqy)[VEC]) {
    const float* c = reinterpret_cast<const float*>(dt.c);
    if (dt.kind == PHK_DET_CHROMA) {
        chroma_add_f32<VEC>(c, dt.nx, dt.zx, t.c[PHK_DP], dqx);
        chroma_add_f32<VEC>(c + 8, dt.ny, dt.zy, t.c[PHK_DP], dqy);
    } else {
        // c = dapp_x/p0, dapp_y/p0, dapp_xy/p0, dapp_yx/p0,
        //     (1+ax^2)/bx, 2ax, bx, (1+ay^2)/by, 2ay, by
        const float ax = c[0], ay = c[1], axy = c[2], ayx = c[3];
        const float c1x = c[4], tax = c[5], bx = c[6];
        const float c1y = c[7], tay = c[8], by = c[9];
        const float (&x)[VEC] = t.c[PHK_X];
        const float (&xp)[VEC] = t.c[PHK_XP];
        const float (&y)[VEC] = t.c[PHK_Y];
        const float (&yp)[VEC] = t.c[PHK_YP];
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            const float Jx = 0.5f * fmaf(bx * xp[j], xp[j],
                                         fmaf(tax * x[j], xp[j], c1x * x[j] * x[j]));
            const float Jy = 0.5f * fmaf(by * yp[j], yp[j],
                                         fmaf(tay * y[j], yp[j], c1y * y[j] * y[j]));
            dqx[j] += fmaf(ax, Jx, axy * Jy);
            dqy[j] += fmaf(ay, Jy, ayx * Jx);
        }
    }
}

// OP0: the op is prog.op[0] of a specialised shape, whose detuners start at
// det[0] (program_shape checks it), so the first two are read at
// compile-time offsets of the parameter block.
// detune_f32 of two particles on the paired FP32 pipes
__device__ __forceinline__ void detune_f32_x2(const phk_detuner& dt,
                                              const Tile<float, 2>& t,
                                              float2& dqx, float2& dqy) {
    const float* c = reinterpret_cast<const float*>(dt.c);
    const float2 DP = make_float2(t.c[PHK_DP][0], t.c[PHK_DP][1]);
    if (dt.kind == PHK_DET_CHROMA) {
        const int n[2] = {dt.nx, dt.ny}, z[2] = {dt.zx, dt.zy};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const float* cq = c + 8 * q;
            float2& dq = q ? dqy : dqx;
            if (z[q] == 0 && n[q] == 1) {
                dq = fma2(f2(cq[0]), DP, dq);
            } else if (z[q] == 0 && n[q] == 2) {
                dq = fma2(fma2(f2(cq[1]), DP, f2(cq[0])), DP, dq);
            } else if (z[q] == 0 && n[q] == 3) {
                dq = fma2(fma2(fma2(f2(cq[2]), DP, f2(cq[1])), DP, f2(cq[0])),
                          DP, dq);
            } else {
                dq.x += chroma_poly_f32(cq, n[q], z[q], DP.x);
                dq.y += chroma_poly_f32(cq, n[q], z[q], DP.y);
            }
        }
    } else {
        const float2 X = make_float2(t.c[PHK_X][0], t.c[PHK_X][1]);
        const float2 XP = make_float2(t.c[PHK_XP][0], t.c[PHK_XP][1]);
        const float2 Y = make_float2(t.c[PHK_Y][0], t.c[PHK_Y][1]);
        const float2 YP = make_float2(t.c[PHK_YP][0], t.c[PHK_YP][1]);
        const float2 Jx = mul2(f2(0.5f),
                               fma2(mul2(f2(c[6]), XP), XP,
                                    fma2(mul2(f2(c[5]), X), XP,
                                         mul2(mul2(f2(c[4]), X), X))));
        const float2 Jy = mul2(f2(0.5f),
                               fma2(mul2(f2(c[9]), YP), YP,
                                    fma2(mul2(f2(c[8]), Y), YP,
                                         mul2(mul2(f2(c[7]), Y), Y))));
        dqx = add2(dqx, fma2(f2(c[0]), Jx, mul2(f2(c[2]), Jy)));
        dqy = add2(dqy, fma2(f2(c[1]), Jy, mul2(f2(c[3]), Jx)));
    }
}

// op_transverse for two particles per thread on the paired FP32 pipes:
// the same operations as the scalar form below, lane for lane
template <bool OP0>
__device__ __forceinline__ void op_transverse_x2(const phk_op& op,
                                                 const phk_program& prog,
                                                 Tile<float, 2>& t) {
    const float* p = reinterpret_cast<const float*>(op.p);
    const bool disp = op.flags & PHK_FLAG_DISPERSION;
    float2 X = make_float2(t.c[PHK_X][0], t.c[PHK_X][1]);
    float2 XP = make_float2(t.c[PHK_XP][0], t.c[PHK_XP][1]);
    float2 Y = make_float2(t.c[PHK_Y][0], t.c[PHK_Y][1]);
    float2 YP = make_float2(t.c[PHK_YP][0], t.c[PHK_YP][1]);
    const float2 DP = make_float2(t.c[PHK_DP][0], t.c[PHK_DP][1]);
    float2 M[8];
    const bool detuned = op.flags & PHK_FLAG_DETUNED;
    if (detuned) {
        float2 dqx = f2(0.f), dqy = f2(0.f);
        const int nd = op.det_count;
        if (OP0) {
            if (nd > 0) detune_f32_x2(prog.det[0], t, dqx, dqy);
            if (nd > 1) detune_f32_x2(prog.det[1], t, dqx, dqy);
            for (int d = 2; d < nd; ++d) detune_f32_x2(prog.det[d], t, dqx, dqy);
        } else {
            for (int d = 0; d < nd; ++d)
                detune_f32_x2(prog.det[op.det_begin + d], t, dqx, dqy);
        }
        float2 sx, cx, sy, cy;
        sincos_turns_x2(f2(p[16]), f2(p[17]), dqx, &sx, &cx);
        sincos_turns_x2(f2(p[18]), f2(p[19]), dqy, &sy, &cy);
        // I and J are float-float (p[40..55] their low parts)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            M[e] = fma2(f2(p[e]), cx,
                        fma2(f2(p[8 + e]), sx,
                             fma2(f2(p[40 + e]), cx, mul2(f2(p[48 + e]), sx))));
            M[4 + e] = fma2(f2(p[4 + e]), cy,
                            fma2(f2(p[12 + e]), sy,
                                 fma2(f2(p[44 + e]), cy, mul2(f2(p[52 + e]), sy))));
        }
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) M[e] = f2(p[e]);
    }
    if (disp) {
        X = fma2(f2(-p[32]), DP, X);
        Y = fma2(f2(-p[34]), DP, Y);
    }
    float2 cxr = f2(0.f), cxp = f2(0.f), cyr = f2(0.f), cyp = f2(0.f);
    if (!detuned) {
        // low parts of the constant matrix
        cxr = fma2(f2(p[40]), X, mul2(f2(p[41]), XP));
        cxp = fma2(f2(p[42]), X, mul2(f2(p[43]), XP));
        cyr = fma2(f2(p[44]), Y, mul2(f2(p[45]), YP));
        cyp = fma2(f2(p[46]), Y, mul2(f2(p[47]), YP));
    }
    const float2 nx = fma2(M[0], X, fma2(M[1], XP, cxr));
    const float2 nxp = fma2(M[2], X, fma2(M[3], XP, cxp));
    const float2 ny = fma2(M[4], Y, fma2(M[5], YP, cyr));
    const float2 nyp = fma2(M[6], Y, fma2(M[7], YP, cyp));
    X = nx; XP = nxp; Y = ny; YP = nyp;
    if (disp) {
        X = fma2(f2(p[33]), DP, X);
        Y = fma2(f2(p[35]), DP, Y);
    }
    t.c[PHK_X][0] = X.x; t.c[PHK_X][1] = X.y;
    t.c[PHK_XP][0] = XP.x; t.c[PHK_XP][1] = XP.y;
    t.c[PHK_Y][0] = Y.x; t.c[PHK_Y][1] = Y.y;
    t.c[PHK_YP][0] = YP.x; t.c[PHK_YP][1] = YP.y;
}

template <int VEC, bool OP0 = false>
__device__ __forceinline__ void op_transverse(const phk_op& op,
                                              const phk_program& prog,
                                              Tile<float, VEC>& t) {
    if constexpr (VEC == 2) {
        op_transverse_x2<OP0>(op, prog, t);
    } else {
        const float* p = reinterpret_cast<const float*>(op.p);
        const bool disp = op.flags & PHK_FLAG_DISPERSION;
        const float Dx0 = p[32], Dx1 = p[33], Dy0 = p[34], Dy1 = p[35];
        float (&x)[VEC] = t.c[PHK_X];
        float (&xp)[VEC] = t.c[PHK_XP];
        float (&y)[VEC] = t.c[PHK_Y];
        float (&yp)[VEC] = t.c[PHK_YP];
        const float (&dp)[VEC] = t.c[PHK_DP];
        float M[8][VEC];
        if (op.flags & PHK_FLAG_DETUNED) {
            float dqx[VEC], dqy[VEC];
    #pragma unroll
            for (int j = 0; j < VEC; ++j) { dqx[j] = 0.f; dqy[j] = 0.f; }
            const int nd = op.det_count;
            if (OP0) {
                if (nd > 0) detune_f32<VEC>(prog.det[0], t, dqx, dqy);
                if (nd > 1) detune_f32<VEC>(prog.det[1], t, dqx, dqy);
                for (int d = 2; d < nd; ++d) detune_f32<VEC>(prog.det[d], t, dqx, dqy);
            } else {
                for (int d = 0; d < nd; ++d)
                    detune_f32<VEC>(prog.det[op.det_begin + d], t, dqx, dqy);
            }
            const float qxh = p[16], qxl = p[17], qyh = p[18], qyl = p[19];
    #pragma unroll
            for (int j = 0; j < VEC; ++j) {
                float sx, cx, sy, cy;
                sincos_turns(qxh, qxl, dqx[j], &sx, &cx);
                sincos_turns(qyh, qyl, dqy[j], &sy, &cy);
                // I and J are float-float (p[40..55] their low parts)
    #pragma unroll
                for (int e = 0; e < 4; ++e) {
                    M[e][j] = fmaf(p[e], cx, fmaf(p[8 + e], sx,
                                                  fmaf(p[40 + e], cx, p[48 + e] * sx)));
                    M[4 + e][j] = fmaf(p[4 + e], cy,
                                       fmaf(p[12 + e], sy,
                                            fmaf(p[44 + e], cy, p[52 + e] * sy)));
                }
            }
        } else {
    #pragma unroll
            for (int j = 0; j < VEC; ++j)
    #pragma unroll
                for (int e = 0; e < 8; ++e) M[e][j] = p[e];
        }
        // low parts of a constant matrix (zero for a per-particle one)
        const bool ml = !(op.flags & PHK_FLAG_DETUNED);
    #pragma unroll
        for (int j = 0; j < VEC; ++j) {
            if (disp) {
                x[j] = fmaf(-Dx0, dp[j], x[j]);
                y[j] = fmaf(-Dy0, dp[j], y[j]);
            }
            float cxr = 0.f, cxp = 0.f, cyr = 0.f, cyp = 0.f;
            if (ml) {
                cxr = fmaf(p[40], x[j], p[41] * xp[j]);
                cxp = fmaf(p[42], x[j], p[43] * xp[j]);
                cyr = fmaf(p[44], y[j], p[45] * yp[j]);
                cyp = fmaf(p[46], y[j], p[47] * yp[j]);
            }
            const float nx = fmaf(M[0][j], x[j], fmaf(M[1][j], xp[j], cxr));
            const float nxp = fmaf(M[2][j], x[j], fmaf(M[3][j], xp[j], cxp));
            const float ny = fmaf(M[4][j], y[j], fmaf(M[5][j], yp[j], cyr));
            const float nyp = fmaf(M[6][j], y[j], fmaf(M[7][j], yp[j], cyp));
            x[j] = nx; xp[j] = nxp; y[j] = ny; yp[j] = nyp;
            if (disp) {
                x[j] = fmaf(Dx1, dp[j], x[j]);
                y[j] = fmaf(Dy1, dp[j], y[j]);
            }
        }
    }
}

template <int VEC>
__device__ __forceinline__ void op_drift(const phk_op& op,
                                         Tile<float, VEC>& t) {
    // p: beta_ratio, eta0 * L (hi, lo), beta_ratio lo
    const float* p = reinterpret_cast<const float*>(op.p);
    const float br = p[0], etaL = p[1], etaLl = p[2], brl = p[3];
    const bool shrink = op.flags & PHK_FLAG_SHRINK;
    if constexpr (VEC == 2) {
        const float2 Z = make_float2(t.c[PHK_Z][0], t.c[PHK_Z][1]);
        const float2 DP = make_float2(t.c[PHK_DP][0], t.c[PHK_DP][1]);
        const float2 zs = shrink ? fma2(f2(br), Z, mul2(f2(brl), Z)) : Z;
        const float2 zn = fma2(f2(-etaL), DP, fma2(f2(-etaLl), DP, zs));
        t.c[PHK_Z][0] = zn.x; t.c[PHK_Z][1] = zn.y;
    } else {
    #pragma unroll
        for (int j = 0; j < VEC; ++j) {
            // z = beta_ratio * z - (eta0 * L) * dp, constants float-float
            const float z = t.c[PHK_Z][j];
            const float dp = t.c[PHK_DP][j];
            const float zs = shrink ? fmaf(br, z, brl * z) : z;
            t.c[PHK_Z][j] = fmaf(-etaL, dp, fmaf(-etaLl, dp, zs));
        }
    }
}

template <int VEC>
__device__ __forceinline__ void op_rfkick(const phk_op& op,
                                          Tile<float, VEC>& t) {
    // p: h/C (hi, lo) turns per metre, (phi_offset+phi_lock)/2pi (hi, lo),
    //    A/p0_new, p0_old/p0_new, p_inc/p0_new, -, D_x, D_y, then the low
    //    parts of A/p0_new and p0_old/p0_new
    const float* p = reinterpret_cast<const float*>(op.p);
    const float mh = p[0], ml = p[1], oh = p[2], ol = p[3];
    const float A = p[4], ratio = p[5], pinc = p[6], Dx = p[8], Dy = p[9];
    const float Al = p[10], ratiol = p[11];
    const bool disp = op.flags & PHK_FLAG_DISPERSION;
    if constexpr (VEC == 2) {
        float2 DP = make_float2(t.c[PHK_DP][0], t.c[PHK_DP][1]);
        float2 X = make_float2(t.c[PHK_X][0], t.c[PHK_X][1]);
        float2 Y = make_float2(t.c[PHK_Y][0], t.c[PHK_Y][1]);
        if (disp) {
            X = fma2(f2(-Dx), DP, X);
            Y = fma2(f2(-Dy), DP, Y);
        }
        const float2 s = sin_turns_of_product_x2(
            make_float2(t.c[PHK_Z][0], t.c[PHK_Z][1]), mh, ml, oh, ol);
        DP = fma2(f2(A), s, fma2(f2(Al), s,
                                 fma2(DP, f2(ratio), fma2(DP, f2(ratiol), f2(-pinc)))));
        if (disp) {
            X = fma2(f2(Dx), DP, X);
            Y = fma2(f2(Dy), DP, Y);
        }
        t.c[PHK_DP][0] = DP.x; t.c[PHK_DP][1] = DP.y;
        t.c[PHK_X][0] = X.x; t.c[PHK_X][1] = X.y;
        t.c[PHK_Y][0] = Y.x; t.c[PHK_Y][1] = Y.y;
    } else {
    #pragma unroll
        for (int j = 0; j < VEC; ++j) {
            float& dp = t.c[PHK_DP][j];
            if (disp) {
                t.c[PHK_X][j] = fmaf(-Dx, dp, t.c[PHK_X][j]);
                t.c[PHK_Y][j] = fmaf(-Dy, dp, t.c[PHK_Y][j]);
            }
            const float s = sin_turns_of_product(t.c[PHK_Z][j], mh, ml, oh, ol);
            dp = fmaf(A, s, fmaf(Al, s, fmaf(dp, ratio, fmaf(dp, ratiol, -pinc))));
            if (disp) {
                t.c[PHK_X][j] = fmaf(Dx, dp, t.c[PHK_X][j]);
                t.c[PHK_Y][j] = fmaf(Dy, dp, t.c[PHK_Y][j]);
            }
        }
    }
}

template <int VEC>
__device__ __forceinline__ void op_linear_long(const phk_op& op,
                                               Tile<float, VEC>& t) {
    // p: cos (hi, lo), longfac*sin (hi, lo), D_x, D_y, sin/longfac (hi, lo)
    const float* p = reinterpret_cast<const float*>(op.p);
    const float cs = p[0], csl = p[1], a = p[2], al = p[3];
    const float b = p[6], bl = p[7];
    const float Dx = p[4], Dy = p[5];
    const bool disp = op.flags & PHK_FLAG_DISPERSION;
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
        float& z = t.c[PHK_Z][j];
        float& dp = t.c[PHK_DP][j];
        if (disp) {
            t.c[PHK_X][j] = fmaf(-Dx, dp, t.c[PHK_X][j]);
            t.c[PHK_Y][j] = fmaf(-Dy, dp, t.c[PHK_Y][j]);
        }
        const float z0 = z, dp0 = dp;
        z = fmaf(z0, cs, fmaf(-a, dp0, fmaf(z0, csl, -al * dp0)));
        dp = fmaf(dp0, cs, fmaf(b, z0, fmaf(dp0, csl, bl * z0)));
        if (disp) {
            t.c[PHK_X][j] = fmaf(Dx, dp, t.c[PHK_X][j]);
            t.c[PHK_Y][j] = fmaf(Dy, dp, t.c[PHK_Y][j]);
        }
    }
}

template <int VEC>
__device__ __forceinline__ void op_scale(const phk_op& op,
                                         Tile<float, VEC>& t) {
    const float f = reinterpret_cast<const float*>(op.p)[0];
#pragma unroll
    for (int j = 0; j < VEC; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) t.c[q][j] *= f;
}

template <int VEC>
__device__ __forceinline__ void op_damper(const phk_op& op,
                                          Tile<float, VEC>& t) {
    const float* m = reinterpret_cast<const float*>(damper_means(op) + 6);
    const float* f = reinterpret_cast<const float*>(op.p);
    const bool reactive = op.flags & PHK_FLAG_REACTIVE;
#pragma unroll
    for (int pl = 0; pl < 2; ++pl) {
        if (!(op.flags & (pl == 0 ? PHK_FLAG_DAMP_X : PHK_FLAG_DAMP_Y))) continue;
        const int u = pl == 0 ? PHK_X : PHK_Y, up = pl == 0 ? PHK_XP : PHK_YP;
        const float* g = f + 3 * pl;
        const float c1 = g[0] * __ldg(m + up);
        const float c2 = reactive ? __fdiv_rn(g[1] * __ldg(m + u), g[2]) : 0.f;
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            t.c[up][j] -= c1;
            if (reactive) t.c[up][j] -= c2;
        }
    }
}

// one dispatch per op per tile (uniform across the CTA)
template <typename T, int VEC>
__device__ __forceinline__ void run_program(const phk_program& prog,
                                            const Aux64& aux, Tile<T, VEC>& t) {
    for (int o = 0; o < prog.n_ops; ++o) {
        const phk_op& op = prog.op[o];
        switch (op.kind) {
            case PHK_OP_TRANSVERSE:
                if constexpr (std::is_same<T, double>::value)
                    op_transverse<VEC, false>(op, o, prog, aux, t);
                else
                    op_transverse<VEC>(op, prog, t);
                break;
            case PHK_OP_DRIFT: op_drift<VEC>(op, t); break;
            case PHK_OP_RF_KICK:
                if constexpr (std::is_same<T, double>::value)
                    op_rfkick<VEC, false>(op, aux.op[o], aux.sine, t);
                else
                    op_rfkick<VEC>(op, t);
                break;
            case PHK_OP_LINEAR_LONG:
                if constexpr (std::is_same<T, double>::value)
                    op_linear_long<VEC, false>(op, t);
                else
                    op_linear_long<VEC>(op, t);
                break;
            case PHK_OP_SCALE_TRANS: op_scale<VEC>(op, t); break;
            case PHK_OP_DAMPER: op_damper<VEC>(op, t); break;
            default: break;
        }
    }
}

// Element sequences with a compile-time shape: the op parameters are then
// read at fixed offsets of the kernel's parameter block (constant-bank
// operands) instead of through a per-tile dispatch loop.
enum TrackShape {
    SHAPE_GENERIC = 0,   // any program: run_program's loop
    SHAPE_NONE = 1,      // no ops (slicing / kicks only)
    SHAPE_T = 2,         // one transverse segment
    SHAPE_T_RF = 3,      // transverse, drift, RF kick, drift (RFSystems)
    SHAPE_T_LIN = 4,     // transverse, linear longitudinal map
    // FP64 form: the same with a detuned transverse segment
    SHAPE_DETUNED = 8,   // flag
    SHAPE_DT = SHAPE_T | SHAPE_DETUNED,
    SHAPE_DT_RF = SHAPE_T_RF | SHAPE_DETUNED,
    SHAPE_DT_LIN = SHAPE_T_LIN | SHAPE_DETUNED,
};

template <typename T, int VEC, int SHAPE>
__device__ __forceinline__ void run_program_shape(const phk_program& prog,
                                                  const Aux64& aux,
                                                  Tile<T, VEC>& t) {
    if constexpr (SHAPE == SHAPE_GENERIC) {
        run_program<T, VEC>(prog, aux, t);
    } else if constexpr (SHAPE != SHAPE_NONE && std::is_same<T, double>::value) {
        constexpr bool DET = (SHAPE & SHAPE_DETUNED) != 0;
        op_transverse<VEC, true, DET>(prog.op[0], 0, prog, aux, t);
        if constexpr ((SHAPE & ~SHAPE_DETUNED) == SHAPE_T_RF) {
            op_drift_rf<VEC>(aux.op[1], t);
            op_rfkick<VEC, true>(prog.op[2], aux.op[2], aux.sine, t);
            op_drift_rf<VEC>(aux.op[3], t);
        } else if constexpr ((SHAPE & ~SHAPE_DETUNED) == SHAPE_T_LIN) {
            op_linear_long<VEC, true>(prog.op[1], t);
        }
    } else if constexpr (SHAPE != SHAPE_NONE) {
        op_transverse<VEC, true>(prog.op[0], prog, t);
        if constexpr (SHAPE == SHAPE_T_RF) {
            op_drift<VEC>(prog.op[1], t);
            op_rfkick<VEC>(prog.op[2], t);
            op_drift<VEC>(prog.op[3], t);
        } else if constexpr (SHAPE == SHAPE_T_LIN) {
            op_linear_long<VEC>(prog.op[1], t);
        }
    }
}

// ===================================================================
// per-slice accumulation in shared memory
//
// Fixed-point sums (FixHist below; FixHist64 and FixHist32, the FP32 batch's, in
//   phk_fixed.cuh), one histogram per CTA updated with 32-bit integer atomics:
//   integer addition is associative, so the sums are bit-identical whatever the
//   order.
//
// FP64 batch: each warp owns a private histogram (count, sum x, sum y per
//   slice) of plain double sums; lanes of a warp holding the same slice are
//   serialised by bids (warp_accumulate), so a bin is updated in a fixed lane
//   order and the sums do not depend on scheduling.  When the per-warp copies
//   do not fit the shared-memory plan, warps share copies through atomics; the
//   order of the warps sharing a copy is then not fixed, so those sums can
//   differ in their last bits between launches.  (In the FP32 batch, bids
//   with compensated float sums took 40 % of the shared-memory pipe and a
//   fifth of the instructions: 207 us a pass at 64 bunches and 1.03e7
//   particles against 188 us as exact fixed-point sums.)
// ===================================================================

// All 32 lanes of the warp must call this together; s < 0 means "no bin".
// Lanes of a warp that hold the same slice are serialised by bids: in each
// round every pending lane bids atomicMax(tag[s], epoch << 5 | lane) on the
// warp's private tag array; the standing bid (the highest pending lane of
// that slice) updates the bin with plain loads and stores.  A bin is thus
// always updated in descending lane order: the sums are deterministic.
__device__ __forceinline__ void warp_accumulate(int s, double vx, double vy,
                                                double* hx, double* hy,
                                                int* hc, int* tag,
                                                unsigned& epoch,
                                                bool shared_hist) {
    if (shared_hist) {
        if (s >= 0) {
            atomicAdd(hc + s, 1);
            atomicAdd(hx + s, vx);
            atomicAdd(hy + s, vy);
        }
        return;
    }
    const int lane = threadIdx.x & 31;
    bool pending = s >= 0;
    while (__any_sync(0xffffffffu, pending)) {
        ++epoch;
        const int bid = (int)((epoch << 5) | (unsigned)lane);
        if (pending) atomicMax(tag + s, bid);
        __syncwarp();
        if (pending && tag[s] == bid) {
            hc[s] += 1;
            hx[s] = add(hx[s], vx);
            hy[s] = add(hy[s], vy);
            pending = false;
        }
        __syncwarp();
    }
}

// -------------------------------------------------------------------
// FixHist: exact, order-independent per-slice sums of FP32 coordinates.
//
// Every thread-block cluster agrees on one power-of-two scale per
// coordinate, 2^k with k chosen from the largest finite |u| of its first
// tiles so that it maps to [2^26, 2^27).  A value u becomes the integer v = rint(u 2^k) (u 2^k is exact; the rounding is
// the only approximation, at most 2^-27 of that largest value, the order
// of the FP32 rounding of u itself).  Level A, |u 2^k| < 2^30: v is split into two
// 15-bit digits d0 = v & 0x7fff in [0, 2^15) and d1 = v >> 15 (arithmetic)
// in [-2^15, 2^15), added to 32-bit counters with shared-memory atomics
// (two per coordinate, one for the count: five per particle); 2^16 values
// per counter stay inside the int32 range (a CTA adds its counters to level
// B at least every 2^16 values).  Level B, larger
// finite values (2^30 <= |u 2^k| < 2^40, rare): 64-bit atomics at the same
// scale on the cluster's partial column in global memory, zeroed by the
// cluster's rank 0 before the first add.  Level C: NaN, +-inf and
// |u 2^k| >= 2^40 set flag bits of the slice; the slice's sum then becomes
// NaN (NaN, both infinities, or a finite value out of range) or +-inf, but for
// the finite ones as a floating-point sum would.  At the end rank 0 adds the digits of its cluster's CTAs and
// the level-B sums as 64-bit integers, converts once to FP64 (x 2^-k) and
// writes the partial column.  Every step is integer arithmetic or a fixed
// sequence of FP64 operations: the result is bit-identical on every launch.
// -------------------------------------------------------------------
constexpr float kFixLevelA = 1073741824.0f;        // 2^30
constexpr float kFixLevelB = 1099511627776.0f;     // 2^40
constexpr int64_t kFixMaxPerCta = (int64_t)1 << 16;  // values per counter

// Levels B and C of one value (rare; kept out of line): v = u 2^k.
static __device__ __noinline__ void fix_add_slow(long long* spill,
                                                 unsigned* flag, int shift,
                                                 float u, float v) {
    if (fabsf(v) < kFixLevelB) {
        atomicAdd(reinterpret_cast<unsigned long long*>(spill),
                  (unsigned long long)__float2ll_rn(v));
        return;
    }
    // 1 NaN, 2 +inf, 4 -inf, 8 finite beyond the 64-bit range
    const unsigned b = isnan(u) ? 1u : (isinf(u) ? (u > 0.f ? 2u : 4u) : 8u);
    atomicOr(flag, b << shift);
}

// level-B columns of a CTA's FixHist (read on the rare slow path only):
// element s of coordinate q at spill[q] + s * stride
struct FixSpill {
    long long* spill[2];
    int64_t stride;
};

struct FixHist {
    int* cnt;             // [S] counts
    int* dig;             // [4][S]: x d0 d1, y d0 d1
    unsigned* flag;       // [(S + 3) / 4]: one byte per slice, x low nibble
    const FixSpill* sp;   // in shared memory
    int S;
    float scale[2];       // 2^k of x and y

    __device__ __forceinline__ void add_q(int q, int s, float u) const {
        const float v = u * scale[q];
        if (fabsf(v) < kFixLevelA) {
            const int iv = __float2int_rn(v);
            int* d = dig + 2 * q * S + s;
            atomicAdd(d, iv & 0x7fff);
            atomicAdd(d + S, iv >> 15);
        } else {
            fix_add_slow(sp->spill[q] + (int64_t)s * sp->stride,
                         flag + (s >> 2), 8 * (s & 3) + 4 * q, u, v);
        }
    }
    __device__ __forceinline__ void add(int s, float x, float y) const {
        atomicAdd(cnt + s, 1);
        add_q(0, s, x);
        add_q(1, s, y);
    }
    // the sum held by the two digit counters at d and d + S
    static __device__ __forceinline__ long long total(const int* d, int S) {
        return (long long)d[0] + ((long long)d[S] << 15);
    }
};

// 2^k, the FixHist scale for the largest finite magnitude m (as float bits;
// 0 when there is none): m 2^k in [2^26, 2^27)
__device__ __forceinline__ float fix_scale(unsigned mbits) {
    int k = 40;                         // no finite non-zero value seen
    if (mbits != 0u && mbits < 0x7f800000u) {
        const int e = (int)(mbits >> 23) - 127;   // denormals: e = -127
        k = 26 - e;
    }
    k = k > 100 ? 100 : (k < -100 ? -100 : k);
    return ldexpf(1.0f, k);
}

template <typename T>
struct FixOf;
template <>
struct FixOf<float> { using type = FixHist; };
template <>
struct FixOf<double> { using type = FixHist64; };

// the FP64 value of a slice sum from its 64-bit total and flag nibble
__device__ __forceinline__ double fix_value(long long total, unsigned fl,
                                            float scale) {
    if (fl) {
        if ((fl & 9u) || (fl & 6u) == 6u)
            return __longlong_as_double(0x7ff8000000000000ll);
        return (fl & 2u) ? __longlong_as_double(0x7ff0000000000000ll)
                         : __longlong_as_double((long long)0xfff0000000000000ull);
    }
    return (double)total * (1.0 / (double)scale);
}

// ===================================================================
// the fused track kernel
// ===================================================================

template <typename T, int VEC>
struct VecIO;
template <>
struct VecIO<double, 2> {
    static __device__ __forceinline__ void ld(const double* p, double (&o)[2]) {
        const double2 t = *reinterpret_cast<const double2*>(p);
        o[0] = t.x; o[1] = t.y;
    }
    static __device__ __forceinline__ void st(double* p, const double (&v)[2]) {
        *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
    }
};
template <>
struct VecIO<float, 2> {
    static __device__ __forceinline__ void ld(const float* p, float (&o)[2]) {
        const float2 t = *reinterpret_cast<const float2*>(p);
        o[0] = t.x; o[1] = t.y;
    }
    static __device__ __forceinline__ void st(float* p, const float (&v)[2]) {
        *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
    }
};
template <>
struct VecIO<float, 4> {
    static __device__ __forceinline__ void ld(const float* p, float (&o)[4]) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        o[0] = t.x; o[1] = t.y; o[2] = t.z; o[3] = t.w;
    }
    static __device__ __forceinline__ void st(float* p, const float (&v)[4]) {
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    }
};
template <typename T>
struct VecIO<T, 1> {
    static __device__ __forceinline__ void ld(const T* p, T (&o)[1]) { o[0] = *p; }
    static __device__ __forceinline__ void st(T* p, const T (&v)[1]) { *p = v[0]; }
};

struct TrackArgs {
    void* c[6];
    int64_t n;
    int64_t n_tiles;
    int32_t has_pk;
    int32_t has_acc;
    int32_t load_mask;
    int32_t store_mask;
    int32_t n_hist;      // histogram copies per CTA (1 or warps per CTA)
    int32_t kicks_smem;  // kick tables staged in shared memory
    int32_t cluster;     // CTAs per thread-block cluster (accumulation)
    int32_t stages;      // TMA ring stages (0: plain loads)
    int32_t kick_comb;   // kicks staged as one summed table per target
    int32_t comb_slot[3];  // table of target xp, yp, dp (-1: none)
    uint32_t wait_limit;   // polls of a copy wait before giving up
    int32_t n_tables;      // kick tables staged (summed targets or kicks)
    int32_t reserved;
};

constexpr size_t kSineBytes = ((size_t)kSineEntries * sizeof(u64) + 15) & ~(size_t)15;

template <typename T>
__device__ __forceinline__ T tadd(T a, T b);
template <>
__device__ __forceinline__ double tadd<double>(double a, double b) { return add(a, b); }
template <>
__device__ __forceinline__ float tadd<float>(float a, float b) { return a + b; }
template <typename T>
__device__ __forceinline__ T tmul(T a, T b);
template <>
__device__ __forceinline__ double tmul<double>(double a, double b) { return mul(a, b); }
template <>
__device__ __forceinline__ float tmul<float>(float a, float b) { return a * b; }

// FP32 histograms of track_smem_layout: FixHist, FixHist32
constexpr int kFixSingle = 1, kFixBatch = 2;

// shared memory layout, in this order (every region 16-byte aligned):
//   histogram: bid-serialised words [3][n_hist][Sa] (sum x, sum y as double;
//              count as int in the third region), or with `fix` (FP32) the
//              integer counters: count [Sa], digits [4][Sa] and flag bytes [Sa]
//              of FixHist, digits [6][Sa] of FixHist32
//   accumulation edges [Sa + 1] T, pending-kick edges [Sp + 1] T,
//   kick tables [n_tables][Sp] T (when staged), bid tags [n_hist][Sa] int
//   (none with `fix`), TMA ring [stages][6][tile] T, one mbarrier per stage
__host__ __device__ inline size_t align16(size_t b) { return (b + 15) & ~size_t(15); }

template <typename T>
__host__ __device__ inline size_t track_smem_layout(int Sa, int Sp, int n_hist,
                                                    int n_tables, int kicks_smem,
                                                    int stages, int tile,
                                                    size_t* off, int fix = 0) {
    size_t b = 0;
    if (fix) {
        off[0] = b; b = align16(b + (size_t)4 * Sa);                            // count
        off[1] = b; b = align16(b + (size_t)4 * (fix == kFixBatch ? 6 : 4) * Sa); // digits
        off[2] = b;                                                             // flags
        if (fix == kFixSingle) b = align16(b + (size_t)4 * ((Sa + 3) / 4));
    } else {
        off[0] = b; b = align16(b + (size_t)8 * n_hist * Sa);   // sum x words
        off[1] = b; b = align16(b + (size_t)8 * n_hist * Sa);   // sum y words
        off[2] = b; b = align16(b + (size_t)4 * n_hist * Sa);   // count
    }
    off[3] = b; b = align16(b + sizeof(T) * (Sa > 0 ? Sa + 1 : 0));
    off[4] = b; b = align16(b + sizeof(T) * (Sp > 0 ? Sp + 1 : 0));
    off[5] = b; b = align16(b + (kicks_smem ? sizeof(T) * (size_t)n_tables * Sp : 0));
    off[6] = b; b = align16(b + (fix ? 0 : (size_t)4 * n_hist * Sa));  // bid tags
    off[7] = b; b = align16(b + (size_t)stages * 6 * tile * sizeof(T));
    off[8] = b; b = align16(b + (size_t)8 * stages);         // mbarriers
    return b;
}

// Exact slice lookup against a staged edge table.  FP32: the float edges
// themselves.  FP64: order-preserving int64 keys of the edges, so that the
// lookup needs no FP64 instruction (the first estimate is FP32).
template <typename T>
__device__ __forceinline__ void stage_edge(T* dst, int i, T e);
template <>
__device__ __forceinline__ void stage_edge<float>(float* dst, int i, float e) {
    dst[i] = e;
}
template <>
__device__ __forceinline__ void stage_edge<double>(double* dst, int i,
                                                   double e) {
    reinterpret_cast<long long*>(dst)[i] = order_key(e);
}

template <typename T>
struct Bins;
template <>
struct Bins<float> {
    const float* e;
    int S, neg;
    float tail, iw, mg;   // tail = e[0]
    // mg bounds |u - u_ref|, u = (zz - e0) * iw the FP32 position in slice
    // units and u_ref the reference's (z - tail) / width of the same z.
    // The table's end edges lie within one FP32 ulp of the real cuts, so
    // with A = |e0| + |eS|: |u - u_ref| <= 2^-23 A iw (the cuts) +
    // 4 * 2^-24 (S + 1) (the four roundings of D = eS - e0, S / D,
    // zz - e0 and the product), plus FP64 roundings of order 2^-52 S.
    // mg takes twice that; a margin of 1/4 slice or more switches the fast
    // path off.
    __device__ __forceinline__ void init(const float* edges, int n, int negate) {
        e = edges; S = n; neg = negate;
        const float e0 = e[0], eS = e[S];
        tail = e0;
        const float span = eS - e0;
        iw = span > 0.f ? (float)S / span : 0.f;
        const float m = 4.76837158203125e-7f *      // 2^-21
                        ((fabsf(e0) + fabsf(eS)) * iw + (float)S + 2.f);
        mg = m < 0.25f ? m : 2.f;
    }
    // The fast path also needs every edge within mg of its uniform
    // position: u(e_k) within mg of k.  Then for u at least mg inside
    // slice k (and u monotone in z), e_k <= z < e_{k+1}.  Tables of
    // uniform-bin slicers pass (the bound above); tables of other slicers
    // (uniform charge) fail and keep the search.  u - k is exact here
    // (Sterbenz) whenever it is small.
    __device__ __forceinline__ bool edges_uniform(int tid, int nthreads) const {
        if (mg >= 1.f) return true;
        bool ok = true;
        for (int i = tid; i <= S; i += nthreads)
            ok = ok && fabsf((e[i] - tail) * iw - (float)i) < mg;
        return ok;
    }
    __device__ __forceinline__ void disable_fast() { mg = 2.f; }
    // Exact slice of VEC particles.  Fast path: when u lies at least mg
    // inside a slice of [0, S), floor(u) is the reference's index.  Only
    // particles within mg of a slice edge (or outside the cuts, or NaN)
    // read the edge table: the estimate and both bracketing edges, then
    // corrections that walk at most to the table ends (e0 <= zz < eS holds
    // inside), so no access leaves e[0..S].
    template <int VEC>
    __device__ __forceinline__ void index_vec(const float (&z)[VEC],
                                              int (&out)[VEC]) const {
        float zz[VEC];
        bool slow = false;
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            zz[j] = neg ? -z[j] : z[j];
            const float u = (zz[j] - tail) * iw;
            const float fl = floorf(u);
            const float fr = u - fl;             // exact
            const int ki = (int)fl;              // saturating, NaN -> 0
            const bool ok = fr >= mg && fr <= 1.f - mg &&
                            (unsigned)ki < (unsigned)S;
            out[j] = ok ? ki : -2;
            slow |= !ok;
        }
        if (!slow) return;
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            if (out[j] != -2) continue;
            if (!(zz[j] >= tail) || !(zz[j] < e[S])) { out[j] = -1; continue; }
            int kk = (int)((zz[j] - tail) * iw);
            kk = kk < 0 ? 0 : (kk > S - 1 ? S - 1 : kk);
            float l = e[kk], h = e[kk + 1];
            while (zz[j] < l) { --kk; h = l; l = e[kk]; }
            while (zz[j] >= h) { ++kk; h = e[kk + 1]; }
            out[j] = kk;
        }
    }
    __device__ __forceinline__ int index(float z) const {
        float zv[1] = {z};
        int o[1];
        index_vec<1>(zv, o);
        return o[0];
    }
};
template <>
struct Bins<double> {
    const long long* k;
    int S, neg;
    float tail, iw;
    long long k0, kS;
    __device__ __forceinline__ void init(const double* edges, int n, int negate) {
        k = reinterpret_cast<const long long*>(edges); S = n; neg = negate;
        k0 = k[0]; kS = k[S];
        // undo the key map for the two end edges (keys of finite doubles)
        const float lo = approx_float(key_to_double(k0));
        const float hi = approx_float(key_to_double(kS));
        tail = lo;
        const float span = hi - lo;
        iw = span > 0.f ? (float)S / span : 0.f;
    }
    template <int VEC>
    __device__ __forceinline__ void index_vec(const double (&z)[VEC],
                                              int (&out)[VEC]) const {
        long long kz[VEC], lo[VEC], hi[VEC];
        int b[VEC];
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            const double zz = neg ? -z[j] : z[j];
            kz[j] = order_key(zz);
            int kk = (int)((approx_float(zz) - tail) * iw);
            b[j] = kk < 0 ? 0 : (kk > S - 1 ? S - 1 : kk);
        }
#pragma unroll
        for (int j = 0; j < VEC; ++j) { lo[j] = k[b[j]]; hi[j] = k[b[j] + 1]; }
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            if (kz[j] < k0 || kz[j] >= kS) { out[j] = -1; continue; }
            int kk = b[j];
            long long l = lo[j], h = hi[j];
            while (kz[j] < l) { --kk; h = l; l = k[kk]; }
            while (kz[j] >= h) { ++kk; h = k[kk + 1]; }
            out[j] = kk;
        }
    }
    __device__ __forceinline__ int index(double z) const {
        double zv[1] = {z};
        int o[1];
        index_vec<1>(zv, o);
        return o[0];
    }
    // no table-free path in the FP64 form
    __device__ __forceinline__ bool edges_uniform(int, int) const { return true; }
    __device__ __forceinline__ void disable_fast() {}
};

// After Bins::init over a staged table: the table-free lookup stays on
// only if every edge passes edges_uniform (a block-wide vote; every
// thread of the block calls this, `active` being the same for all).
template <typename T>
__device__ __forceinline__ void vote_fast_path(Bins<T>& b, bool active,
                                               int tid, int nthreads) {
    const bool ok = !active || b.edges_uniform(tid, nthreads);
    if (!__syncthreads_and(ok) && active) b.disable_fast();
}

// Stages the pending kicks' slice edges (as lookup keys) into `epk` and,
// when a.kicks_smem, their tables into `ktab`: one table per kick, or with
// a.kick_comb one summed table per target (slot a.comb_slot[target]).
// Called by all threads of a CTA; a __syncthreads() must follow.
// edges_staged: the edge table is there already.
template <typename T>
__device__ __forceinline__ void stage_pending(const phk_kick_set& pk,
                                              const TrackArgs& a, T* epk,
                                              T* ktab, int tid, int nthreads,
                                              bool edges_staged = false) {
    const int Sp = pk.slicer.n_slices;
    const int nk = pk.n_kicks;
    const T* e = reinterpret_cast<const T*>(pk.slicer.edges);
    if (!edges_staged) for (int i = tid; i <= Sp; i += nthreads) stage_edge<T>(epk, i, e[i]);
    if (a.kick_comb) {
        for (int i = tid; i < Sp; i += nthreads) {
            T v[3] = {T(0), T(0), T(0)};
            for (int k = 0; k < nk; ++k) {
                const int tg = pk.target[k];
                const int q = tg == PHK_XP ? 0 : (tg == PHK_YP ? 1 : 2);
                v[q] = tadd<T>(v[q], reinterpret_cast<const T*>(pk.kick[k])[i]);
            }
            for (int q = 0; q < 3; ++q)
                if (a.comb_slot[q] >= 0) ktab[a.comb_slot[q] * Sp + i] = v[q];
        }
    } else if (a.kicks_smem) {
        for (int i = tid; i < nk * Sp; i += nthreads) {
            const int k = i / Sp;
            ktab[i] = reinterpret_cast<const T*>(pk.kick[k])[i - k * Sp];
        }
    }
}

static __device__ __noinline__ double add_cold(double a, double b) {
    return add(a, b);
}

// Wake kicks left pending by the previous WakeField.track, applied in
// kick order to the VEC particles of a tile in registers
// (DipoleWakeKickX/Y.apply, impedances/wake_kicks.py:207-260, and the
// quadrupolar / constant kicks :185-202, :284-361).  `ktab` holds the
// staged tables (stage_pending); particles outside the cuts or past the
// end are left alone.
template <typename T, int VEC, bool FULL>
__device__ __forceinline__ void apply_pending(const phk_kick_set& pk,
                                              const TrackArgs& a,
                                              const Bins<T>& bpk,
                                              const T* ktab, Tile<T, VEC>& t,
                                              int64_t i0) {
    const int Sp = pk.slicer.n_slices;
    const int nk = pk.n_kicks;
    int sl[VEC];
    bpk.index_vec(t.c[PHK_Z], sl);
    if (a.kick_comb) {
        // FP32 form, dipolar kicks only: one table per target, the
        // kicks of that target summed at staging
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            const bool on = sl[j] >= 0 && (FULL || i0 + j < a.n);
            const int s = on ? sl[j] : 0;
            if (a.comb_slot[0] >= 0)
                t.c[PHK_XP][j] = tadd<T>(t.c[PHK_XP][j], on ? ktab[a.comb_slot[0] * Sp + s] : T(0));
            if (a.comb_slot[1] >= 0)
                t.c[PHK_YP][j] = tadd<T>(t.c[PHK_YP][j], on ? ktab[a.comb_slot[1] * Sp + s] : T(0));
            if (a.comb_slot[2] >= 0) {
                const T kick = on ? ktab[a.comb_slot[2] * Sp + s] : T(0);
                // rarely there: out of line, it costs the FP64 pipe nothing
                if constexpr (std::is_same<T, double>::value)
                    t.c[PHK_DP][j] = add_cold(t.c[PHK_DP][j], kick);
                else
                    t.c[PHK_DP][j] = tadd<T>(t.c[PHK_DP][j], kick);
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            const int s = sl[j];
            if (s < 0 || (!FULL && i0 + j >= a.n)) continue;
            const T kx = t.c[PHK_X][j], ky = t.c[PHK_Y][j];
            for (int k = 0; k < nk; ++k) {
                T val = a.kicks_smem
                            ? ktab[k * Sp + s]
                            : __ldg(reinterpret_cast<const T*>(pk.kick[k]) + s);
                const int qd = pk.quad[k];
                if (qd == PHK_X) val = tmul<T>(val, kx);
                else if (qd == PHK_Y) val = tmul<T>(val, ky);
                const int tg = pk.target[k];
                if (tg == PHK_XP) t.c[PHK_XP][j] = tadd<T>(t.c[PHK_XP][j], val);
                else if (tg == PHK_YP) t.c[PHK_YP][j] = tadd<T>(t.c[PHK_YP][j], val);
                else t.c[PHK_DP][j] = tadd<T>(t.c[PHK_DP][j], val);
            }
        }
    }
}

// Per-CTA state shared by the tile loops of the track kernels.  H: the
// accumulation's histogram
template <typename T, int VEC, class H = typename FixOf<T>::type>
struct TrackCtx {
    T* cp[6];
    Bins<T> bpk, bac;
    const T* ktab;
    double* hx;           // FP64 batch
    double* hy;
    int* hc;
    int* tag;
    unsigned epoch;
    bool shared_hist;
    H fix;                // single bunch, FP32 batch
    Aux64 aux;            // FP64 form
};

// One tile of VEC particles per thread, already in registers.  All threads
// of the CTA call this together (the FP64 batch's accumulation is
// warp-synchronous); lanes whose particles are past the end pass live = false.

// 1. wake kicks of the previous WakeField.track, in kick order;
// 2. element program
template <typename T, int VEC, int SHAPE, bool FULL, class H>
__device__ __forceinline__ void tile_advance(const phk_program& prog,
                                             const phk_kick_set& pk,
                                             const TrackArgs& a,
                                             TrackCtx<T, VEC, H>& cx,
                                             Tile<T, VEC>& t, int64_t i0) {
    if (a.has_pk) apply_pending<T, VEC, FULL>(pk, a, cx.bpk, cx.ktab, t, i0);
    run_program_shape<T, VEC, SHAPE>(prog, cx.aux, t);
}

// 3. slice accumulation; 4. stores
template <typename T, int VEC, bool FULL, bool FIX, class H>
__device__ __forceinline__ void tile_finish(const phk_accum& acc,
                                            const TrackArgs& a,
                                            TrackCtx<T, VEC, H>& cx,
                                            Tile<T, VEC>& t, int64_t i0,
                                            bool full) {
    if (a.has_acc) {
        int sl[VEC];
        cx.bac.index_vec(t.c[PHK_Z], sl);
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            const bool live = FULL || i0 + j < a.n;
            const int s = live ? sl[j] : -1;
            if (acc.idx_out && live)
                acc.idx_out[i0 + j] =
                    s >= 0 ? s
                           : outside_index((double)t.c[PHK_Z][j],
                                           acc.slicer.tail, acc.slicer.width);
            if constexpr (FIX) {
                if (s >= 0) cx.fix.add(s, t.c[PHK_X][j], t.c[PHK_Y][j]);
            } else {
                warp_accumulate(s, t.c[PHK_X][j], t.c[PHK_Y][j], cx.hx, cx.hy,
                                   cx.hc, cx.tag, cx.epoch, cx.shared_hist);
            }
        }
    }
    // 4. stores of the coordinates the tile changed
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        if (!((a.store_mask >> q) & 1)) continue;
        if (FULL || full) {
            VecIO<T, VEC>::st(cx.cp[q] + i0, t.c[q]);
        } else {
#pragma unroll
            for (int j = 0; j < VEC; ++j)
                if (i0 + j < a.n) cx.cp[q][i0 + j] = t.c[q][j];
        }
    }
}

template <typename T, int VEC, int SHAPE, bool FULL, bool FIX = false>
__device__ __forceinline__ void run_tile(const phk_program& prog,
                                         const phk_kick_set& pk,
                                         const phk_accum& acc,
                                         const TrackArgs& a,
                                         TrackCtx<T, VEC>& cx, Tile<T, VEC>& t,
                                         int64_t i0, bool full) {
    tile_advance<T, VEC, SHAPE, FULL>(prog, pk, a, cx, t, i0);
    tile_finish<T, VEC, FULL, FIX>(acc, a, cx, t, i0, full);
}

template <typename T, int VEC, class H>
__device__ __forceinline__ void load_tile_plain(const TrackArgs& a,
                                                const TrackCtx<T, VEC, H>& cx,
                                                Tile<T, VEC>& t, int64_t i0,
                                                bool full) {
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        if (!((a.load_mask >> q) & 1)) {
#pragma unroll
            for (int j = 0; j < VEC; ++j) t.c[q][j] = T(0);
            continue;
        }
        if (full) {
            VecIO<T, VEC>::ld(cx.cp[q] + i0, t.c[q]);
        } else {
#pragma unroll
            for (int j = 0; j < VEC; ++j)
                t.c[q][j] = (i0 + j < a.n) ? cx.cp[q][i0 + j] : T(0);
        }
    }
}

// CTAs per thread-block cluster of an accumulating FP32 launch (FP64: see
// launch_track64_t).  The cluster's
// barrier releases and acquires at cluster scope (its default), global memory
// included, and only the cluster touches its partial column until the kernel
// ends: no fence of the whole device is needed beside it.  Two of those waited
// for the particles' stores: 0.9 us of a pass (1e6 particles, the turn 40.6 to
// 39.7 us).
constexpr int kCluster = 4;

// FP32 single-bunch kernel: particles per thread, resident CTAs per SM it
// is compiled for (register cap) and the shared memory a CTA may plan for
constexpr int kF32Vec = 2;
constexpr int kF32MinBlocks = 4;
constexpr size_t kF32SmemBudget = 56 * 1024;
// shared memory a CTA may use at three CTAs per SM
constexpr size_t kF32SmemBudget3 = 75 * 1024;

// polls of one mbarrier phase before a kernel gives up (order of a second)
constexpr unsigned kWaitLimit = 1u << 22;
// stages of the TMA ring at most
constexpr int kMaxStages = 4;

// FixHist counters are added to the level-B column after this many tiles
// of a CTA (kFixMaxPerCta values per counter at most)
template <int TILE>
constexpr int64_t fix_flush_tiles() { return kFixMaxPerCta / TILE; }

// Adds the FixHist digits of this CTA to the level-B column and clears them
// (all threads, between two barriers).
__device__ __forceinline__ void fix_flush(const FixHist& f, int tid,
                                          int nthreads) {
    for (int s = tid; s < f.S; s += nthreads) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            int* d = f.dig + 2 * q * f.S + s;
            const long long t = FixHist::total(d, f.S);
            if (t != 0)
                atomicAdd(reinterpret_cast<unsigned long long*>(
                              f.sp->spill[q] + (int64_t)s * f.sp->stride),
                          (unsigned long long)t);
            d[0] = 0; d[f.S] = 0;
        }
    }
}

// The precision form's pass (T is float; the plain form's is track64_kernel):
// four resident CTAs per SM (<= 64 registers)
template <typename T, int VEC, int SHAPE>
__global__ void __launch_bounds__(kTrackThreads, kF32MinBlocks)
track_kernel(const __grid_constant__ phk_program prog,
             const __grid_constant__ phk_kick_set pk,
             const __grid_constant__ phk_accum acc, const TrackArgs a) {
    static_assert(std::is_same<T, float>::value, "the precision form's pass");
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int TILE = kTrackThreads * VEC;
    const int Sa = a.has_acc ? acc.slicer.n_slices : 0;
    const int Sp = a.has_pk ? pk.slicer.n_slices : 0;
    size_t off[9];
    track_smem_layout<T>(Sa, Sp, a.n_hist, a.n_tables, a.kicks_smem, a.stages,
                         TILE, off, kFixSingle);
    int* hcnt = reinterpret_cast<int*>(smem + off[0]);
    int* fdig = reinterpret_cast<int*>(smem + off[1]);
    unsigned* fflag = reinterpret_cast<unsigned*>(smem + off[2]);
    T* eacc = reinterpret_cast<T*>(smem + off[3]);
    T* epk = reinterpret_cast<T*>(smem + off[4]);
    T* ktab = reinterpret_cast<T*>(smem + off[5]);
    T* ring = reinterpret_cast<T*>(smem + off[7]);
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(smem + off[8]);
    __shared__ unsigned s_max[2];   // FixHist: largest finite |x|, |y| bits
    __shared__ FixSpill s_spill;
    // TMA ring: warps that finished each stage, the last tile issued into
    // each stage (-1: none), a wait that gave up somewhere in the CTA
    __shared__ int s_rel[kMaxStages], s_last[kMaxStages], s_abort;

    const int tid = threadIdx.x;
    const int64_t full_tiles = a.n / TILE;
    const int64_t mine = (a.stages > 0 && blockIdx.x < full_tiles)
                             ? (full_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x
                             : 0;
    const bool has_partial = a.stages > 0 && a.n % TILE != 0 &&
                             blockIdx.x == (int)(full_tiles % gridDim.x);
    int nq = 0;
    for (int q = 0; q < 6; ++q) nq += (a.load_mask >> q) & 1;
    const unsigned stage_bytes = (unsigned)(nq * TILE * sizeof(T));
    // bulk copies of this CTA's k-th tile into stage st (one thread)
    auto issue = [&](int64_t k, int st) {
        const int64_t tile = blockIdx.x + k * gridDim.x;
        fence_proxy_async_smem();
        mbar_expect_tx(bars + st, stage_bytes);
        for (int q = 0; q < 6; ++q)
            if ((a.load_mask >> q) & 1)
                bulk_g2s(ring + ((size_t)st * 6 + q) * TILE,
                         reinterpret_cast<T*>(a.c[q]) + tile * TILE,
                         TILE * sizeof(T), bars + st);
        s_last[st] = (int)k;
    };
    if (tid == 0) {
        s_max[0] = s_max[1] = 0u;
        s_abort = 0;
        for (int st = 0; st < kMaxStages; ++st) s_rel[st] = 0, s_last[st] = -1;
        for (int st = 0; st < a.stages; ++st) mbar_init(bars + st, 1);
        if (a.stages > 0) {
            mbar_fence_init();
            // the first tiles are on their way while the CTA stages its
            // tables (the ring has shared memory of its own)
            for (int64_t k = 0; k < mine && k < a.stages; ++k) issue(k, (int)k);
        }
    }
    if (a.has_acc) {
        const T* e = reinterpret_cast<const T*>(acc.slicer.edges);
        for (int i = tid; i <= Sa; i += blockDim.x) stage_edge<T>(eacc, i, e[i]);
        for (int i = tid; i < Sa; i += blockDim.x) hcnt[i] = 0;
        for (int i = tid; i < 4 * Sa; i += blockDim.x) fdig[i] = 0;
        for (int i = tid; i < (Sa + 3) / 4; i += blockDim.x) fflag[i] = 0u;
    }
    if (a.has_pk) stage_pending<T>(pk, a, epk, ktab, tid, blockDim.x);
    __syncthreads();

    TrackCtx<T, VEC> cx;
#pragma unroll
    for (int q = 0; q < 6; ++q) cx.cp[q] = reinterpret_cast<T*>(a.c[q]);
    if (a.has_pk) cx.bpk.init(epk, Sp, pk.slicer.negate);
    if (a.has_acc) cx.bac.init(eacc, Sa, acc.slicer.negate);
    vote_fast_path<T>(cx.bpk, a.has_pk, tid, blockDim.x);
    vote_fast_path<T>(cx.bac, a.has_acc, tid, blockDim.x);
    cx.ktab = ktab;

    // partial column of this CTA's cluster
    const bool clustered = a.has_acc && a.cluster > 1;
    const unsigned crank = clustered ? cg::this_cluster().block_rank() : 0u;
    const int column = clustered ? (int)(blockIdx.x / a.cluster) : (int)blockIdx.x;
    const int G = acc.grid;
    double* P = acc.partials;

    bool bad = false;   // a bounded copy wait of this thread gave up

    if (a.has_acc) {
        // ---- the cluster's scale: largest finite |x|, |y| of the inputs
        // of every member's first tile (the maps change them by factors
        // of order one; larger values take level B)
        unsigned m[2] = {0u, 0u};
        auto see = [&](float u, int q) {
            const unsigned b = __float_as_uint(u) & 0x7fffffffu;
            if (b < 0x7f800000u && b > m[q]) m[q] = b;
        };
        if (mine > 0) {
            bad = !mbar_wait(bars, 0u, a.wait_limit);
            if (!bad) {
                const T* src = ring + tid * VEC;
#pragma unroll
                for (int j = 0; j < VEC; ++j) {
                    see(src[(size_t)PHK_X * TILE + j], 0);
                    see(src[(size_t)PHK_Y * TILE + j], 1);
                }
            }
        } else {
            const int64_t i0 = (a.stages > 0 ? full_tiles * TILE
                                             : (int64_t)blockIdx.x * TILE) +
                               tid * VEC;
            if (a.stages == 0 || has_partial) {
#pragma unroll
                for (int j = 0; j < VEC; ++j) {
                    if (i0 + j < a.n) {
                        see(cx.cp[PHK_X][i0 + j], 0);
                        see(cx.cp[PHK_Y][i0 + j], 1);
                    }
                }
            }
        }
        m[0] = __reduce_max_sync(0xffffffffu, m[0]);
        m[1] = __reduce_max_sync(0xffffffffu, m[1]);
        if ((tid & 31) == 0) {
            atomicMax(&s_max[0], m[0]);
            atomicMax(&s_max[1], m[1]);
        }
        if (tid == 0) {
            s_spill.spill[0] = reinterpret_cast<long long*>(P) + (int64_t)Sa * G + column;
            s_spill.spill[1] = reinterpret_cast<long long*>(P) + (int64_t)2 * Sa * G + column;
            s_spill.stride = G;
        }
        // rank 0 clears its column's level-B sums before any member adds
        if (crank == 0) {
            for (int s = tid; s < Sa; s += blockDim.x) {
                reinterpret_cast<long long*>(P)[(int64_t)(Sa + s) * G + column] = 0;
                reinterpret_cast<long long*>(P)[(int64_t)(2 * Sa + s) * G + column] = 0;
            }
        }
        unsigned M[2];
        if (clustered) {
            cg::cluster_group cl = cg::this_cluster();
            cl.sync();                   // orders the clears, see kCluster
            M[0] = M[1] = 0u;
            for (unsigned r = 0; r < cl.num_blocks(); ++r) {
                const unsigned* sm = cl.map_shared_rank(s_max, r);
                M[0] = max(M[0], sm[0]);
                M[1] = max(M[1], sm[1]);
            }
        } else {
            __syncthreads();
            M[0] = s_max[0];
            M[1] = s_max[1];
        }
        cx.fix.cnt = hcnt;
        cx.fix.dig = fdig;
        cx.fix.flag = fflag;
        cx.fix.sp = &s_spill;
        cx.fix.S = Sa;
        cx.fix.scale[0] = fix_scale(M[0]);
        cx.fix.scale[1] = fix_scale(M[1]);
    }

    if (a.stages > 0) {
        // ---- full tiles through a TMA ring of `stages` stages.  Warps run
        // decoupled: each waits for a stage's copies, processes its part of
        // the tile and releases the stage; the warp whose release completes
        // the stage issues the copies of the tile `stages` ahead into it.
        // A wait that gives up marks the CTA aborted: no more copies are
        // issued, the remaining tiles are skipped (every warp still takes
        // part in the same barriers), and the copies in flight are drained.
        const int nwarps = (int)(blockDim.x >> 5);
        const int lane = tid & 31;
        volatile int* abort_flag = &s_abort;
        int st = 0;
        unsigned ph = 0u;
        for (int64_t k = 0; k < mine; ++k) {
            bool ok = false;
            if (!bad && !*abort_flag) {
                ok = mbar_wait(bars + st, ph, a.wait_limit);
                if (!ok) {
                    bad = true;
                    *abort_flag = 1;
                }
            }
            if (ok) {
                Tile<T, VEC> t;
                const T* src = ring + (size_t)st * 6 * TILE + tid * VEC;
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    if ((a.load_mask >> q) & 1) {
                        VecIO<T, VEC>::ld(src + (size_t)q * TILE, t.c[q]);
                    } else {
#pragma unroll
                        for (int j = 0; j < VEC; ++j) t.c[q][j] = T(0);
                    }
                }
                const int64_t i0 = (blockIdx.x + k * gridDim.x) * TILE + tid * VEC;
                run_tile<T, VEC, SHAPE, true, true>(prog, pk, acc, a, cx, t, i0, true);
            }
            __syncwarp();                    // this warp's part of stage st read
            if (lane == 0) {
                __threadfence_block();
                if (atomicAdd(&s_rel[st], 1) == nwarps - 1) {
                    s_rel[st] = 0;
                    if (k + a.stages < mine && !*abort_flag) issue(k + a.stages, st);
                }
            }
            if (++st == a.stages) {
                st = 0;
                ph ^= 1u;
            }
            if (a.has_acc && (k + 1) % fix_flush_tiles<TILE>() == 0) {
                __syncthreads();
                fix_flush(cx.fix, tid, blockDim.x);
                __syncthreads();
            }
        }
        __syncthreads();
        if (s_abort) {
            // report, then wait (bounded) for the last copies issued into
            // each stage so that none lands in shared memory after the CTA
            // has exited (earlier ones completed before their stage was
            // released)
            if (tid == 0) {
                bool drained = true;
                for (int q = 0; q < a.stages; ++q)
                    if (s_last[q] >= 0 &&
                        !mbar_wait(bars + q, (unsigned)((s_last[q] / a.stages) & 1),
                                   kWaitLimit))
                        drained = false;
                if (prog.status)
                    atomicMax(prog.status, drained ? PHK_DEV_TIMEOUT
                                                   : PHK_DEV_TIMEOUT_UNDRAINED);
            }
            __syncthreads();
        } else if (has_partial) {
            // ---- the partial last tile, plain loads
            const int64_t i0 = full_tiles * TILE + tid * VEC;
            const bool full = i0 + VEC <= a.n;
            Tile<T, VEC> t;
            load_tile_plain<T, VEC>(a, cx, t, i0, full);
            run_tile<T, VEC, SHAPE, false, true>(prog, pk, acc, a, cx, t, i0, full);
        }
    } else {
        // ---- plain loads; every warp runs whole tiles (lanes past the end
        // carry dead particles) so the warp-level accumulation sees 32 lanes
        const int64_t n_tiles_grid = (a.n_tiles + gridDim.x - 1) / gridDim.x;
        for (int64_t it = 0; it < n_tiles_grid; ++it) {
            const int64_t tile = blockIdx.x + it * gridDim.x;
            const int64_t i0 = (tile * blockDim.x + tid) * VEC;
            const bool full = i0 + VEC <= a.n;
            Tile<T, VEC> t;
            load_tile_plain<T, VEC>(a, cx, t, i0, full);
            run_tile<T, VEC, SHAPE, false, true>(prog, pk, acc, a, cx, t, i0, full);
            if (a.has_acc && (it + 1) % fix_flush_tiles<TILE>() == 0) {
                __syncthreads();
                fix_flush(cx.fix, tid, blockDim.x);
                __syncthreads();
            }
        }
    }

    if (!a.has_acc) return;
    // ---- rank 0 adds its cluster's counters and level-B sums as 64-bit
    // integers and writes the partial column in FP64
    unsigned nb = 1;
    if (clustered) {
        // level-B adds before the barrier (see kCluster)
        cg::cluster_group cl = cg::this_cluster();
        cl.sync();
        nb = cl.num_blocks();
    } else {
        __syncthreads();
    }
    if (crank == 0) {
        const long long* lp = reinterpret_cast<const long long*>(P);
        for (int s = tid; s < Sa; s += blockDim.x) {
            long long c = 0, tq[2];
            unsigned fl = 0;
            tq[0] = __ldcg(lp + (int64_t)(Sa + s) * G + column);
            tq[1] = __ldcg(lp + (int64_t)(2 * Sa + s) * G + column);
            // unrolled over the cluster's members, so that the loads of
            // every member are in flight together
#pragma unroll
            for (int r = 0; r < kCluster; ++r) {
                if (r >= (int)nb) break;
                const int* rc = hcnt;
                const int* rd = fdig;
                const unsigned* rf = fflag;
                if (clustered) {
                    cg::cluster_group cl = cg::this_cluster();
                    rc = cl.map_shared_rank(hcnt, r);
                    rd = cl.map_shared_rank(fdig, r);
                    rf = cl.map_shared_rank(fflag, r);
                }
                c += rc[s];
                fl |= (rf[s >> 2] >> (8 * (s & 3))) & 0xffu;
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    tq[q] += FixHist::total(rd + 2 * q * Sa + s, Sa);
            }
            P[(int64_t)s * G + column] = (double)c;
            P[(int64_t)(Sa + s) * G + column] =
                fix_value(tq[0], fl & 15u, cx.fix.scale[0]);
            P[(int64_t)(2 * Sa + s) * G + column] =
                fix_value(tq[1], fl >> 4, cx.fix.scale[1]);
        }
    }
    if (clustered) cg::this_cluster().sync();  // members keep their counters until read
}

// ===================================================================
// launch configuration
// ===================================================================

// Shared-memory plan of an FP32 launch: TMA ring stages (aligned launches),
// chosen so that the occupancy the kernel is compiled for is reached
// whenever possible.  n_tables: kick tables staged per CTA.
static inline size_t smem_for(int Sa, int Sp, int n_tables, bool tma,
                              int* kicks_smem, int* stages, size_t budget_in = 0,
                              int forced_stages = -1) {
    const int tile = kTrackThreads * kF32Vec;
    *kicks_smem = n_tables > 0 && (size_t)n_tables * Sp * sizeof(float) <= 48 * 1024;
    auto bytes = [&](int st) {
        size_t off[9];
        return track_smem_layout<float>(Sa, Sp, 1, n_tables, *kicks_smem, st, tile,
                                        off, kFixSingle);
    };
    if (tma) {
        const size_t budget = budget_in ? budget_in : kF32SmemBudget;
        const bool forced = forced_stages == 0 ||
                            (forced_stages >= 2 && forced_stages <= kMaxStages);
        if (forced && bytes(forced_stages) <= budget) {
            *stages = forced_stages;
            return bytes(forced_stages);
        }
        // by default two ring stages (measured fastest at 500 slices; more
        // take a launch plan) at four CTAs per SM; where they do not fit
        // (about 700 slices and more), two stages at three CTAs per SM,
        // measured faster than plain loads at 1000 slices
        const size_t most = budget_in == 0 && forced_stages < 0 ? kF32SmemBudget3
                                                                : budget;
        if (bytes(2) <= most) {
            *stages = 2;
            return bytes(2);
        }
    }
    *stages = 0;
    return bytes(0);
}

// Kick tables a launch stages: with dipolar kicks only, the kicks of one
// target are summed once per slice into one table per target (one rounding
// per slice instead of one per kick and particle; quadrupolar kicks keep
// the per-kick loop).  Sets
// a->kicks_smem, a->kick_comb, a->comb_slot and a->n_tables.
template <typename T>
static void plan_kick_tables(const phk_kick_set* pk, TrackArgs* a) {
    a->kick_comb = 0;
    a->comb_slot[0] = a->comb_slot[1] = a->comb_slot[2] = -1;
    a->n_tables = 0;
    a->kicks_smem = 0;
    if (!pk) return;
    const int nk = pk->n_kicks, Sp = pk->slicer.n_slices;
    bool dip = true;
    for (int k = 0; k < nk; ++k) dip = dip && pk->quad[k] < 0;
    int slot[3] = {-1, -1, -1}, n = 0;
    if (dip) {
        for (int k = 0; k < nk; ++k) {
            const int tg = pk->target[k];
            const int q = tg == PHK_XP ? 0 : (tg == PHK_YP ? 1 : 2);
            if (slot[q] < 0) slot[q] = n++;
        }
    }
    const int tables = dip ? n : nk;
    a->kicks_smem = tables > 0 && (size_t)tables * Sp * sizeof(T) <= 48 * 1024;
    if (dip && a->kicks_smem) {
        a->kick_comb = 1;
        for (int q = 0; q < 3; ++q) a->comb_slot[q] = slot[q];
        a->n_tables = n;
    } else {
        a->kicks_smem = nk > 0 && (size_t)nk * Sp * sizeof(T) <= 48 * 1024;
        a->n_tables = nk;
    }
}

// Opt the track kernel into the device's full dynamic shared memory, once
// per instantiation and device (never inside a stream capture's hot path).
template <typename T, int VEC, int SHAPE>
static void prepare_track_kernel() {
    static int done_for[64] = {0};
    const DeviceInfo& d = device_info();
    const int dev = d.device < 64 ? d.device : 63;
    if (done_for[dev]) return;
    // dynamic + static shared memory must stay within the opt-in limit
    cudaFuncAttributes fa;
    size_t static_smem = 0;
    if (cudaFuncGetAttributes(&fa, track_kernel<T, VEC, SHAPE>) == cudaSuccess)
        static_smem = fa.sharedSizeBytes;
    else
        cudaGetLastError();
    if (cudaFuncSetAttribute(track_kernel<T, VEC, SHAPE>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             d.max_smem_optin - (int)static_smem) != cudaSuccess)
        cudaGetLastError();
    done_for[dev] = 1;
}

// largest dynamic shared memory a track launch may request
template <typename T, int VEC, int SHAPE>
static size_t track_dynamic_smem_limit() {
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, track_kernel<T, VEC, SHAPE>) != cudaSuccess) {
        cudaGetLastError();
        return (size_t)device_info().max_smem_optin - 1024;
    }
    return (size_t)device_info().max_smem_optin - fa.sharedSizeBytes;
}


template <typename T, int VEC, int SHAPE>
static int occupancy_blocks(size_t smem) {
    int b = 0;
    prepare_track_kernel<T, VEC, SHAPE>();
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &b, track_kernel<T, VEC, SHAPE>, kTrackThreads, smem) != cudaSuccess)
        b = 1;
    return b < 1 ? 1 : b;
}

// clusters of kCluster CTAs that can be resident at once
template <typename T, int VEC, int SHAPE>
static int occupancy_clusters(size_t smem) {
    prepare_track_kernel<T, VEC, SHAPE>();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kCluster * device_info().sm_count, 1, 1);
    cfg.blockDim = dim3(kTrackThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = kCluster;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, track_kernel<T, VEC, SHAPE>, &cfg) !=
            cudaSuccess || n < 1) {
        cudaGetLastError();
        n = device_info().sm_count / kCluster;
    }
    return n < 1 ? 1 : n;
}

template <typename T, int VEC, int SHAPE>
static int launch_track_t(const phk_program* prog, const phk_coords* c,
                          const phk_kick_set* pk, const phk_accum* acc,
                          int load_mask, int store_mask, cudaStream_t st) {
    TrackArgs a;
    memset(&a, 0, sizeof(a));
    a.c[0] = c->x; a.c[1] = c->xp; a.c[2] = c->y;
    a.c[3] = c->yp; a.c[4] = c->z; a.c[5] = c->dp;
    a.n = c->n;
    a.has_pk = pk != nullptr;
    a.has_acc = acc != nullptr;
    a.load_mask = load_mask;
    a.store_mask = store_mask;
    a.cluster = 1;
    a.stages = 0;
    a.kick_comb = 0;
    a.comb_slot[0] = a.comb_slot[1] = a.comb_slot[2] = -1;
    a.wait_limit = wait_limit();
    const int64_t per_tile = (int64_t)kTrackThreads * VEC;
    a.n_tiles = (c->n + per_tile - 1) / per_tile;
    static phk_kick_set zero_pk;
    static phk_accum zero_acc;
    const int Sa = acc ? acc->slicer.n_slices : 0;
    const int Sp = pk ? pk->slicer.n_slices : 0;
    // the TMA ring needs 16-byte aligned coordinates (VEC > 1 launches)
    const bool tma = VEC > 1;
    plan_kick_tables<T>(pk, &a);
    int kicks_smem = 0;
    a.n_hist = 1;
    const TrackPlan pl = track_plan();
    const size_t smem = smem_for(Sa, Sp, a.n_tables, tma, &kicks_smem, &a.stages,
                                 pl.smem_kb > 0 ? (size_t)pl.smem_kb * 1024 : 0,
                                 pl.stages);
    if (kicks_smem != a.kicks_smem)
        return set_error(PHK_EPARAM, "phk_track: inconsistent kick-table plan");
    if (smem > track_dynamic_smem_limit<T, VEC, SHAPE>())
        return set_error(PHK_ESIZE, "phk_track: %zu bytes of shared memory "
                         "needed for %d + %d slices", smem, Sa, Sp);
    prepare_track_kernel<T, VEC, SHAPE>();
    cudaError_t e;
    if (acc) {
        // one partial column per cluster of kCluster CTAs
        a.cluster = kCluster;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)acc->grid * kCluster, 1, 1);
        cfg.blockDim = dim3(kTrackThreads, 1, 1);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = kCluster;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, track_kernel<T, VEC, SHAPE>, *prog, pk ? *pk : zero_pk,
                               *acc, a);
    } else {
        const int bps = occupancy_blocks<T, VEC, SHAPE>(smem);
        int64_t g = (int64_t)device_info().sm_count * bps;
        if (a.n_tiles < g) g = a.n_tiles;
        const int grid = (int)(g < 1 ? 1 : g);
        track_kernel<T, VEC, SHAPE><<<grid, kTrackThreads, smem, st>>>(
            *prog, pk ? *pk : zero_pk, zero_acc, a);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess)
        return set_error(PHK_ECUDA, "phk_track launch: %s", cudaGetErrorString(e));
    count_launches(1);
    note_track_launch(0, a.stages, smem);
    return PHK_OK;
}

static inline int op_mask(const phk_program* prog, int* load, int* store) {
    // which coordinates the program reads / writes
    int ld = 0, stm = 0;
    for (int o = 0; o < prog->n_ops; ++o) {
        const phk_op& op = prog->op[o];
        const bool disp = op.flags & PHK_FLAG_DISPERSION;
        switch (op.kind) {
            case PHK_OP_TRANSVERSE:
                ld |= 0x0F | 0x20;  // x xp y yp dp
                stm |= 0x0F;
                break;
            case PHK_OP_DRIFT:
                ld |= 0x30; stm |= 0x10;
                break;
            case PHK_OP_RF_KICK:
            case PHK_OP_LINEAR_LONG:
                ld |= 0x30; stm |= (op.kind == PHK_OP_RF_KICK ? 0x20 : 0x30);
                if (disp) { ld |= 0x05; stm |= 0x05; }
                break;
            case PHK_OP_SCALE_TRANS:
                ld |= 0x0F; stm |= 0x0F;
                break;
            case PHK_OP_DAMPER:
                if (op.flags & PHK_FLAG_DAMP_X) { ld |= 0x03; stm |= 0x02; }
                if (op.flags & PHK_FLAG_DAMP_Y) { ld |= 0x0C; stm |= 0x08; }
                break;
        }
    }
    *load = ld; *store = stm;
    return 0;
}

// ===================================================================
// batched form: many bunches, one persistent launch
// ===================================================================

struct BatchArgs {
    TrackArgs a;             // coordinates, masks, has_pk / has_acc, n_hist
    const phk_unit* units;
    const int32_t* cta_first;
    const phk_program* programs;
    const void* kicks;
    int32_t* status;
    int32_t n_bunches;
    int32_t n_units;
    int32_t n_columns;
};

constexpr size_t kProgSmem = (sizeof(phk_program) + 15) & ~(size_t)15;
// the quarter wave of an FP64 batch (reserved whatever the programs, so that
// the grid follows from the sizes alone)
template <typename T>
constexpr size_t batch_head() {
    return kProgSmem + (sizeof(T) == 8 ? kSineBytes : 0);
}

// Per CTA: its units in order.  When the bunch changes, the CTA's per-slice
// sums of the previous bunch go to that bunch's partial column, and the new
// bunch's program and kick tables are staged in shared memory.
template <typename T, int VEC, int THREADS, int SHAPE>
__global__ void __launch_bounds__(THREADS, (sizeof(T) == 4 ? 1024 : 512) / THREADS)
batch_track_kernel(const __grid_constant__ phk_kick_set pk,
                   const __grid_constant__ phk_accum acc, const BatchArgs b) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int TILE = THREADS * VEC;
    constexpr bool F64 = sizeof(T) == 8;
    constexpr bool FIX = !F64;
    const TrackArgs& a = b.a;
    const int Sa = a.has_acc ? acc.slicer.n_slices : 0;
    const int Sp = a.has_pk ? pk.slicer.n_slices : 0;
    const int nk = a.has_pk ? pk.n_kicks : 0;
    phk_program* sprog = reinterpret_cast<phk_program*>(smem);
    u64* sine = reinterpret_cast<u64*>(smem + kProgSmem);
    __shared__ OpFix s_op[F64 ? PHK_MAX_OPS : 1];
    __shared__ DetFix s_det[F64 ? PHK_MAX_DETUNERS : 1];
    unsigned char* rest = smem + batch_head<T>();
    size_t off[9];
    track_smem_layout<T>(Sa, Sp, a.n_hist, nk, 1, 0, TILE, off, FIX ? kFixBatch : 0);
    // FIX: one set of counters per CTA
    double* hsx = reinterpret_cast<double*>(rest + off[0]);
    double* hsy = reinterpret_cast<double*>(rest + off[1]);
    int* hcnt = reinterpret_cast<int*>(rest + (FIX ? off[0] : off[2]));
    int* fdig = reinterpret_cast<int*>(rest + off[1]);
    constexpr int WARPS = THREADS / 32;
    __shared__ Spill64 s_spill;
    __shared__ Seen<WARPS> s_seen;
    __shared__ unsigned s_typ[2];
    T* eacc = reinterpret_cast<T*>(rest + off[3]);
    T* epk = reinterpret_cast<T*>(rest + off[4]);
    T* ktab = reinterpret_cast<T*>(rest + off[5]);
    int* htag = reinterpret_cast<int*>(rest + off[6]);
    const int tid = threadIdx.x;

    if (a.has_acc) {
        const T* e = reinterpret_cast<const T*>(acc.slicer.edges);
        for (int i = tid; i <= Sa; i += THREADS) stage_edge<T>(eacc, i, e[i]);
    }
    auto clear = [&]() {
        if constexpr (FIX) {
            for (int i = tid; i < Sa; i += THREADS) hcnt[i] = 0;
            for (int i = tid; i < 6 * Sa; i += THREADS) fdig[i] = 0;
        } else {
            for (int i = tid; i < a.n_hist * Sa; i += THREADS) {
                hsx[i] = 0.0; hsy[i] = 0.0;
                hcnt[i] = 0; htag[i] = 0;
            }
        }
    };
    clear();
    if (a.has_pk) {
        const T* e = reinterpret_cast<const T*>(pk.slicer.edges);
        for (int i = tid; i <= Sp; i += THREADS) stage_edge<T>(epk, i, e[i]);
    }
    if (F64) stage_sine(sine, tid, THREADS);

    using H = typename std::conditional<FIX, FixHist32, FixHist64>::type;
    TrackCtx<T, VEC, H> cx;
    cx.aux = Aux64{sine, s_op, s_det};
#pragma unroll
    for (int q = 0; q < 6; ++q) cx.cp[q] = reinterpret_cast<T*>(a.c[q]);
    cx.ktab = ktab;
    if constexpr (FIX) {
        cx.fix.cnt = hcnt;
        cx.fix.dig = fdig;
        cx.fix.sp = &s_spill;
        cx.fix.S = Sa;
        if (tid < 2 * WARPS) s_seen.in[tid / WARPS][tid % WARPS] = 0u;   // no sample
    } else {
        const int h = (a.n_hist > 1) ? (tid >> 5) % a.n_hist : 0;
        cx.hx = hsx + h * Sa;
        cx.hy = hsy + h * Sa;
        cx.hc = hcnt + h * Sa;
        cx.tag = htag + h * Sa;
        cx.epoch = 0;
        cx.shared_hist = a.n_hist < THREADS / 32;
    }
    __syncthreads();
    if (a.has_pk) cx.bpk.init(epk, Sp, pk.slicer.negate);
    if (a.has_acc) cx.bac.init(eacc, Sa, acc.slicer.negate);
    vote_fast_path<T>(cx.bpk, a.has_pk, tid, blockDim.x);
    vote_fast_path<T>(cx.bac, a.has_acc, tid, blockDim.x);

    int u0 = b.cta_first[blockIdx.x], u1 = b.cta_first[blockIdx.x + 1];
    if (u0 < 0 || u1 > b.n_units || u0 > u1) {
        if (tid == 0 && b.status) atomicMax(b.status, PHK_DEV_BAD_TABLE);
        u0 = u1 = 0;
    }
    int cur = -1, col = -1;
    constexpr int kTiles = kDigitValues32 / TILE;
    int until_carry = kTiles;    // FIX
    bool open = false;           // FIX: a window is still to be set
    // write the CTA's sums of the current bunch to its column, then zero
    auto flush = [&]() {
        __syncthreads();
        const int G = b.n_columns;
        double* P = acc.partials;
        for (int s = tid; s < Sa; s += THREADS) {
            int c = hcnt[s];
            double v[2];
            if constexpr (FIX) {
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    v[q] = __ldcg(s_spill.sum[q] + (int64_t)s * G) +
                           digits32_value(fdig + 3 * q * Sa + s, Sa, cx.fix.top[q], c);
            } else {
                v[0] = hsx[s];
                v[1] = hsy[s];
                for (int k = 1; k < a.n_hist; ++k) {
                    c += hcnt[k * Sa + s];
                    v[0] = add(v[0], hsx[k * Sa + s]);
                    v[1] = add(v[1], hsy[k * Sa + s]);
                }
            }
            P[(int64_t)s * G + col] = (double)c;
            P[(int64_t)(Sa + s) * G + col] = v[0];
            P[(int64_t)(2 * Sa + s) * G + col] = v[1];
        }
        __syncthreads();
        clear();
    };
    for (int u = u0; u < u1; ++u) {
        const phk_unit U = b.units[u];
        const bool ok = U.bunch >= 0 && U.bunch < b.n_bunches &&
                        U.start >= 0 && U.start <= U.end && U.end <= a.n &&
                        (U.start & 3) == 0 &&
                        (!a.has_acc || (U.column >= 0 && U.column < b.n_columns));
        if (!ok) {
            if (tid == 0 && b.status) atomicMax(b.status, PHK_DEV_BAD_TABLE);
            continue;
        }
        if (U.bunch != cur) {
            if (cur >= 0 && a.has_acc) flush();
            __syncthreads();       // the previous bunch's program is done
            const int4* src = reinterpret_cast<const int4*>(b.programs + U.bunch);
            int4* dst = reinterpret_cast<int4*>(sprog);
            for (int i = tid; i < (int)(sizeof(phk_program) / 16); i += THREADS)
                dst[i] = src[i];
            if constexpr (F64) {
                const phk_program& bp = b.programs[U.bunch];
                if (tid < PHK_MAX_OPS) op_fix(bp.op[tid], s_op + tid);
                if (tid < PHK_MAX_DETUNERS && tid < bp.n_det)
                    det_fix(bp.det[tid], s_det + tid);
            }
            if (a.has_pk) {
                const T* kt = reinterpret_cast<const T*>(b.kicks) +
                              (int64_t)U.bunch * nk * Sp;
                if (a.kick_comb) {
                    for (int i = tid; i < Sp; i += THREADS) {
                        T v[3] = {T(0), T(0), T(0)};
                        for (int k = 0; k < nk; ++k) {
                            const int tg = pk.target[k];
                            const int q = tg == PHK_XP ? 0 : (tg == PHK_YP ? 1 : 2);
                            v[q] = tadd<T>(v[q], kt[k * Sp + i]);
                        }
                        for (int q = 0; q < 3; ++q)
                            if (a.comb_slot[q] >= 0) ktab[a.comb_slot[q] * Sp + i] = v[q];
                    }
                } else {
                    for (int i = tid; i < nk * Sp; i += THREADS) ktab[i] = kt[i];
                }
            }
            cur = U.bunch;
            col = U.column;
            if constexpr (FIX) if (a.has_acc) {
                const int64_t G = b.n_columns;
                double* P = acc.partials + col;
                if (tid == 0) {
                    s_spill.sum[0] = P + Sa * G;
                    s_spill.sum[1] = P + 2 * Sa * G;
                    s_spill.stride = G;
                    s_typ[0] = s_typ[1] = 0u;
                }
                for (int s = tid; s < 2 * Sa; s += THREADS) P[(Sa + s) * G] = 0.0;
                cx.fix.top[0] = cx.fix.top[1] = 0.f;
                until_carry = kTiles;
                open = true;
            }
            __syncthreads();
        }
        TrackArgs ua = a;
        ua.n = U.end;
        for (int64_t base = U.start; base < U.end; base += TILE) {
            const int64_t i0 = base + (int64_t)tid * VEC;
            const bool full = i0 + VEC <= U.end;
            Tile<T, VEC> t;
            load_tile_plain<T, VEC>(ua, cx, t, i0, full);
            tile_advance<T, VEC, SHAPE, false>(*sprog, pk, ua, cx, t, i0);
            if constexpr (FIX) {
                if (open) {
                    unsigned m[2] = {0u, 0u};
#pragma unroll
                    for (int j = 0; j < VEC; ++j)
                        if (i0 + j < ua.n) {
                            m[0] = max(m[0], finite_high(t.c[PHK_X][j]));
                            m[1] = max(m[1], finite_high(t.c[PHK_Y][j]));
                        }
                    open = find_typical<WARPS>(&s_seen, s_typ, m[0], m[1]);
#pragma unroll
                    for (int q = 0; q < 2; ++q)
                        if (cx.fix.top[q] == 0.f && s_typ[q]) {
                            cx.fix.top[q] = digit_top(s_typ[q]);
                            open_digits32(hcnt, fdig + 3 * q * Sa, Sa, cx.fix.top[q]);
                        }
                    __syncthreads();
                }
            }
            tile_finish<T, VEC, false, FIX>(acc, ua, cx, t, i0, full);
            if constexpr (FIX) {
                if (a.has_acc && --until_carry == 0) {
                    // before a counter can overflow in the next kTiles tiles
                    until_carry = kTiles;
                    carry_slices32(hcnt, fdig, Sa, kDigitValues32 - kTiles * TILE, &s_spill,
                                   s_typ);
                }
            }
        }
    }
    if (cur >= 0 && a.has_acc) flush();
}

static_assert(sizeof(phk_program) % 16 == 0, "program copied as int4");

template <typename T>
static size_t batch_smem(int Sa, int Sp, int nk, int threads, int* n_hist) {
    const int tile = threads * (sizeof(T) == 8 ? 2 : kF32Vec);
    size_t off[9];
    const int warps = threads / 32;
    // FP32: one set of fixed-point counters; FP64: one private histogram copy
    // per warp when it stays within 48 KB
    constexpr int fix = sizeof(T) == 4 ? kFixBatch : 0;
    int nh = Sa > 0 && !fix ? warps : 1;
    size_t bytes = track_smem_layout<T>(Sa, Sp, nh, nk, 1, 0, tile, off, fix);
    if (bytes > 48 * 1024 && Sa > 0 && !fix) {
        nh = 1;
        bytes = track_smem_layout<T>(Sa, Sp, nh, nk, 1, 0, tile, off, fix);
    }
    *n_hist = nh;
    return batch_head<T>() + bytes;
}

template <typename T, int VEC, int THREADS, int SHAPE>
static int batch_occupancy(size_t smem) {
    static int done_for[64] = {0};
    const DeviceInfo& d = device_info();
    const int dev = d.device < 64 ? d.device : 63;
    if (!done_for[dev]) {
        cudaFuncAttributes fa;
        size_t st = 0;
        if (cudaFuncGetAttributes(&fa, batch_track_kernel<T, VEC, THREADS, SHAPE>) ==
            cudaSuccess)
            st = fa.sharedSizeBytes;
        else
            cudaGetLastError();
        if (cudaFuncSetAttribute(batch_track_kernel<T, VEC, THREADS, SHAPE>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 d.max_smem_optin - (int)st) != cudaSuccess)
            cudaGetLastError();
        done_for[dev] = 1;
    }
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &nb, batch_track_kernel<T, VEC, THREADS, SHAPE>, THREADS, smem) !=
        cudaSuccess) {
        cudaGetLastError();
        nb = 0;
    }
    return nb;
}

template <typename T, int VEC, int THREADS, int SHAPE>
static int launch_batch_t(const phk_batch* bt, const phk_coords* c,
                          const phk_kick_set* pk, const phk_accum* acc,
                          int ld, int stm, cudaStream_t st) {
    BatchArgs b;
    memset(&b, 0, sizeof(b));
    TrackArgs& a = b.a;
    a.c[0] = c->x; a.c[1] = c->xp; a.c[2] = c->y;
    a.c[3] = c->yp; a.c[4] = c->z; a.c[5] = c->dp;
    a.n = c->n;
    a.has_pk = pk != nullptr;
    a.has_acc = acc != nullptr;
    a.load_mask = ld;
    a.store_mask = stm;
    a.kicks_smem = 1;
    a.comb_slot[0] = a.comb_slot[1] = a.comb_slot[2] = -1;
    if (sizeof(T) == 4 && pk) {
        // FP32 form, dipolar kicks only: one staged table per target
        bool dip = true;
        for (int k = 0; k < pk->n_kicks; ++k) dip = dip && pk->quad[k] < 0;
        if (dip) {
            a.kick_comb = 1;
            int n = 0;
            for (int k = 0; k < pk->n_kicks; ++k) {
                const int tg = pk->target[k];
                const int q = tg == PHK_XP ? 0 : (tg == PHK_YP ? 1 : 2);
                if (a.comb_slot[q] < 0) a.comb_slot[q] = n++;
            }
        }
    }
    a.cluster = 1;
    a.stages = 0;
    const int Sa = acc ? acc->slicer.n_slices : 0;
    const int Sp = pk ? pk->slicer.n_slices : 0;
    const int nk = pk ? pk->n_kicks : 0;
    const size_t smem = batch_smem<T>(Sa, Sp, nk, THREADS, &a.n_hist);
    if (batch_occupancy<T, VEC, THREADS, SHAPE>(smem) < 1)
        return set_error(PHK_ESIZE, "phk_track_batch: %zu bytes of shared "
                         "memory for %d + %d slices do not fit", smem, Sa, Sp);
    b.units = bt->units;
    b.cta_first = bt->cta_first;
    b.programs = bt->programs;
    b.kicks = bt->kicks;
    b.status = bt->status;
    b.n_bunches = bt->n_bunches;
    b.n_units = bt->n_units;
    b.n_columns = bt->n_columns;
    static phk_kick_set zero_pk;
    static phk_accum zero_acc;
    batch_track_kernel<T, VEC, THREADS, SHAPE><<<bt->grid, THREADS, smem, st>>>(
        pk ? *pk : zero_pk, acc ? *acc : zero_acc, b);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return set_error(PHK_ECUDA, "phk_track_batch launch: %s",
                         cudaGetErrorString(e));
    count_launches(1);
    return PHK_OK;
}

static inline void track_masks(const phk_program* prog, const phk_kick_set* pk,
                        const phk_accum* acc, int* ld_out, int* stm_out) {
    int ld, stm;
    op_mask(prog, &ld, &stm);
    if (pk) {
        ld |= 1 << PHK_Z;
        for (int k = 0; k < pk->n_kicks; ++k) {
            ld |= 1 << pk->target[k];
            stm |= 1 << pk->target[k];
            if (pk->quad[k] >= 0) ld |= 1 << pk->quad[k];
        }
    }
    if (acc) ld |= (1 << PHK_Z) | (1 << PHK_X) | (1 << PHK_Y);
    ld |= stm;
    *ld_out = ld;
    *stm_out = stm;
}

// ---- per-precision entry points (phk_track_f32.cu / phk_track_f64.cu)
int program_shape(const phk_program* prog);
// the FP64 form's: GENERIC unless PLAIN, with the detuned flag
static inline int program_shape64(const phk_program* prog) {
    const int s = program_plain64(*prog) ? program_shape(prog) : (int)SHAPE_GENERIC;
    return s == SHAPE_GENERIC || s == SHAPE_NONE ||
                   !(prog->op[0].flags & PHK_FLAG_DETUNED)
               ? s : s | (int)SHAPE_DETUNED;
}
int launch_track_f32(const phk_program* prog, const phk_coords* c,
                     const phk_kick_set* pk, const phk_accum* acc, int ld,
                     int stm, bool vec_ok, cudaStream_t st);
int launch_track_f64(const phk_program* prog, const phk_coords* c,
                     const phk_kick_set* pk, const phk_accum* acc, int ld,
                     int stm, bool vec_ok, cudaStream_t st);
int track_clusters_f32(size_t smem);
int track_ctas_f64(size_t smem);
int launch_batch_f32(const phk_batch* bt, const phk_coords* c,
                     const phk_kick_set* pk, const phk_accum* acc, int ld,
                     int stm, cudaStream_t st);
int launch_batch_f64(const phk_batch* bt, const phk_coords* c,
                     const phk_kick_set* pk, const phk_accum* acc, int ld,
                     int stm, cudaStream_t st);
int batch_per_sm_f32(int threads, size_t smem);
int batch_per_sm_f64(int threads, size_t smem);

}  // namespace phk
