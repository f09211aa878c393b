// scatter64.cuh -- the FP64 form of the HG deflection (src/stokes.f90) and of the
// azimuth's turns, for the single-pass transport kernel (transport.cu).
#pragma once

#include "transport_common.cuh"

namespace tam {
namespace {

// (sin, cos) of TWOPI u, u = (x + 1/2) 2^-32 (TWOPI: the truncated constant of
// src/constants.f90:13), from a table of 256 steps of the turn and the Taylor terms
// of the rest, at most 0.0123: next terms 8e-18 and 1e-20.  16 FP64 operations against
// some 45 of the library's, and the angle itself is never rounded.
static __device__ const double2 g_turn[257] = {
#include "turn_table.inc"
};
__device__ __forceinline__ void turn(uint32_t x, double &sn, double &cs)
{
    const uint32_t i = ((x >> 23) + 1u) >> 1;
    const int r = (int)(x - (i << 24));
    const double k = TWOPI_R * 0x1p-32;
    const double b = __fma_rn(__hiloint2double(0x43380000 + (r >> 31), r) - 0x1.8p52, k, 0.5 * k), b2 = b * b;
    const double sb = __fma_rn(b * b2, __fma_rn(b2, 1.0 / 120, -1.0 / 6), b);
    const double cm = b2 * __fma_rn(b2, __fma_rn(b2, -1.0 / 720, 1.0 / 24), -0.5);
    const double2 t = g_turn[i];
    sn = t.x + __fma_rn(t.x, cm, t.y * sb);
    cs = t.y + __fma_rn(t.y, cm, -(t.x * sb));
}
// An azimuth in [0, TWOPI] as (cos, sin); cos and sin of the truncated constants.
struct Azimuth {
    double c, s;
};
constexpr double COS_PI = -0x1.ffffffffff87cp-1, SIN_PI = 0x1.5ee4b2791a46fp-21;
constexpr double COS_2PI = 0x1.ffffffffffe57p-1, SIN_2PI = -0x1.49d4e1c46983ep-22;
// phi -> a - phi, phi -> phi + a, phi -> phi - a for an angle a given as (ca, sa)
__device__ __forceinline__ Azimuth mirrored(Azimuth p, double ca, double sa) { return {ca * p.c + sa * p.s, sa * p.c - ca * p.s}; }
__device__ __forceinline__ Azimuth turned(Azimuth p, double ca, double sa) { return {p.c * ca - p.s * sa, p.s * ca + p.c * sa}; }
// phi -> PI - phi, plus TWOPI below 0
__device__ __forceinline__ Azimuth mirror_x(Azimuth p)
{
    const Azimuth q = mirrored(p, COS_PI, SIN_PI);
    return p.s < 0.0 || (p.c < 0.0 && p.s < SIN_PI) ? turned(q, COS_2PI, SIN_2PI) : q;
}

// HG deflection of src/stokes.f90:6-153 (PI/TWOPI are the truncated constants of
// src/constants.f90:13).  Leaves the direction unchanged when the sampled cosine is
// exactly +-1 (the `goto 100`).  The azimuth is carried as (cos, sin) and turned by
// the deflection angle, whose cosine is at hand: no acos, and no sincos of the sum.
// The reference wraps phi by the truncated TWOPI, a turn of 3e-7: wrapped here at the
// same angles.
//
// The FP64 pipe bounds the walk (83 % busy).  A pass of 2e5 packets through a 100^3
// cube (3.9e7 scatters, 9.7e7 voxel steps) took 1.385e10 of its operations, without
// the acos and that sincos 1.288e10 (1e6 packets 181 -> 165 ms), with quotients and
// roots of their own and compares on the bits 1.032e10 (123 ms), with single voxel steps
// and fuller event batches 9.1e9 (114 ms).  The cosine of the deflection keeps its
// operations one by one: near +-1 the angle multiplies its last bit by 1e8.
__device__ __forceinline__ bool stokes(double hgg, double g2, uint32_t d0, uint32_t d1, double &cost,
                                       double &sint, Azimuth &phi)
{
    const double u0 = Uniform<double>::from(d0);
    if (hgg == 0.0) {
        cost = 2.0 * u0 - 1.0;
        const double s2 = 1.0 - cost * cost;
        sint = s2 <= 0.0 ? 0.0 : sqrt64(s2);
        turn(d1, phi.s, phi.c);
        return true;
    }
    const double costp = cost, sintp = sint;
    const double t = div64(1.0 - g2, 1.0 - hgg + 2.0 * hgg * u0);
    const double num = (1.0 + g2) - t * t;
    const double bmu = is_tiny(hgg) ? num / (2.0 * hgg) : div64(num, 2.0 * hgg);
    const double cosb2 = bmu * bmu;
    if (above_one(bmu) || (ieee::bits(bmu) & ~ieee::SIGN) == ieee::ONE) return false;  // direction unchanged
    const double sinbt = sqrt64(1.0 - cosb2);
    const double ri1 = TWOPI_R * Uniform<double>::from(d1);
    const bool upper = less_pos(PI_R, ri1);
    const double ang = upper ? TWOPI_R - ri1 : ri1;
    double sa, ca;
    ::sincos(ang, &sa, &ca);
    double cosi2 = 0.0, sini2;
    cost = costp * bmu + sintp * sinbt * ca;
    if (below_one(cost)) {
        sint = sqrt64(1.0 - cost * cost);
        sini2 = div64(sa * sintp, sint);
        const double bott = sint * sinbt;
        cosi2 = div64(costp, bott) - div64(cost * bmu, bott);
    } else {
        sint = 0.0;
        sini2 = 0.0;
        if (cost >= 1.0) cosi2 = -1.0;
        if (cost <= -1.0) cosi2 = 1.0;
    }
    double cd = -cosi2 * ca + sini2 * sa * bmu;
    if (above_one(cd)) cd = is_minus(cd) ? -1.0 : 1.0;
    double sd = sqrt64((1.0 - cd) * (1.0 + cd));
    sd = upper ? sd : -sd;
    const Azimuth p = phi;
    phi = turned(p, cd, sd);
    // above TWOPI: minus TWOPI; below 0: plus TWOPI (a turn by up to PI from [0, TWOPI])
    const bool low0 = is_minus(p.s), low = is_minus(phi.s), near = low && less_pos(-phi.s, -SIN_2PI);
    if (upper ? (low0 && !low) || (near && !is_minus(phi.c)) : !low0 && low)
        phi = turned(phi, COS_2PI, upper ? -SIN_2PI : SIN_2PI);
    // back to length 1 (one Newton step)
    const double k = 1.5 - 0.5 * (phi.c * phi.c + phi.s * phi.s);
    phi.c *= k;
    phi.s *= k;
    return true;
}

}  // namespace
}  // namespace tam
