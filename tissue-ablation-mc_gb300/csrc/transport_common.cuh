// transport_common.cuh -- device pieces of the photon transport shared by
// the single-pass kernel (transport.cu) and the batched kernel
// (transport_batch.cu): the HG deflection of src/stokes.f90 in its FP32 form
// (FP64: scatter64.cuh), the Fresnel reflectance, and the incremental DDA's
// per-axis set-up and position reconstruction.
#pragma once

#include "ieee_bits.h"
#include "tam_device.cuh"
#include "tam_kernels.h"

namespace tam {
namespace {

// a < b for values that are not negative (nor NaN): FP64 on the bit patterns,
// which order alike, off GB300's narrow FP64 pipe.
__device__ __forceinline__ bool less_pos(float a, float b) { return a < b; }
__device__ __forceinline__ bool less_pos(double a, double b)
{
    return (int64_t)ieee::bits(a) < (int64_t)ieee::bits(b);
}

// FP64 reciprocal and quotient for normal operands, from the hardware's approximation
// (relative error e of 1e-6): the reciprocal by two of Newton's steps; the quotient by
// one step of third order, y0 (1 + e + e^2), and one correction by its remainder
// (Markstein, 1990).  No special cases and no call, 4 and 6 operations of the FP64 pipe;
// the same bits as IEEE division for all of 2e8 pairs over 1e-280 to 1e280.
__device__ __forceinline__ double rcp_seed(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
__device__ __forceinline__ double rcp64(double x)
{
    double y = rcp_seed(x);
    y = __fma_rn(y, __fma_rn(-x, y, 1.0), y);
    return __fma_rn(y, __fma_rn(-x, y, 1.0), y);
}
__device__ __forceinline__ double div64(double a, double b)
{
    const double y0 = rcp_seed(b), e = __fma_rn(-b, y0, 1.0), y = __fma_rn(y0, __fma_rn(e, e, e), y0), q = a * y;
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}
// |n| below 1e-289, where the reciprocal leaves the normal numbers
__device__ __forceinline__ bool is_tiny(double n) { return (__double2hiint(n) & 0x7fffffff) < 0x03e00000; }
// Square root of a normal operand or zero (a subnormal one, whose root is below 1e-153,
// is returned as it is): g -> sqrt(x) and h -> 1 / (2 sqrt(x)) together
// from the hardware's approximation (Goldschmidt), then one correction by the remainder
// (Markstein): 7 operations, the bits of the IEEE square root for all of 2e8 operands.
__device__ __forceinline__ double sqrt64(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double g = x * y, h = 0.5 * y;
    const double r = __fma_rn(-h, g, 0.5);
    g = __fma_rn(g, r, g);
    h = __fma_rn(h, r, h);
    g = __fma_rn(__fma_rn(-g, g, x), h, g);
    return (__double2hiint(x) & 0x7fffffff) < 0x00100000 ? x : g;
}
// |a| > 1, |a| < 1 and the sign, off the FP64 pipe (a NaN counts as neither)
__device__ __forceinline__ bool above_one(double a) { return (ieee::bits(a) & ~ieee::SIGN) - (ieee::ONE + 1) < ieee::PINF - ieee::ONE; }
__device__ __forceinline__ bool below_one(double a) { return (ieee::bits(a) & ~ieee::SIGN) < ieee::ONE; }
__device__ __forceinline__ bool is_minus(double a) { return (int64_t)ieee::bits(a) < 0; }

// PTX approximate forms (relative error ~2^-22) for the FP32 path, whose
// results are checked statistically against the FP64 path.
__device__ __forceinline__ float rcp_ax(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float sqrt_ax(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt_ax(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// FP32 constants of one material's HG sampling: with u uniform,
// t = n1 / (d0 + d1 u) and the cosine is (b0 - t^2) ib.
struct HgF {
    float g, n1, d0, d1, b0, ib;
};
__device__ __forceinline__ HgF hg_consts(float g, float g2)
{
    return HgF{g, 1.f - g2, 1.f - g, 2.f * g, 1.f + g2, rcp_ax(2.f * g)};
}

// FP32 form of the same HG deflection.  The azimuth is carried as the pair
// (cos phi, sin phi) and rotated by the deflection angle dph, since
// phi' = phi +- dph (src/stokes.f90:136-140) gives
//   cos phi' = cos phi cos dph -+ sin phi sin dph,  sin dph = sqrt(1 - cos^2 dph),
// which replaces acos(cosdph) and the sincos of phi by one square root; the
// pair is renormalised so that rounding cannot drift over many scatters.
// Every sampled quantity (t, bmu, ang, cost, cosdph) follows the reference's
// formulas; only the evaluation of phi differs.
__device__ __forceinline__ bool stokes_f32(const HgF &c, float u0, float u1, float &cost, float &sint, float &cp,
                                           float &sp)
{
    const float PI = (float)PI_R, TWOPI = (float)TWOPI_R;
    if (c.g == 0.f) {
        cost = 2.f * u0 - 1.f;
        const float s2 = 1.f - cost * cost;
        sint = s2 <= 0.f ? 0.f : sqrt_ax(s2);
        __sincosf(TWOPI * u1, &sp, &cp);
        return true;
    }
    const float costp = cost, sintp = sint;
    const float t = c.n1 * rcp_ax(__fmaf_rn(c.d1, u0, c.d0));
    const float bmu = __fmaf_rn(-t, t, c.b0) * c.ib;
    if (fabsf(bmu) >= 1.f) return false;  // clamped to +-1: direction unchanged
    const float sinbt = sqrt_ax(1.f - bmu * bmu);
    const float ri1 = TWOPI * u1;
    const bool upper = ri1 > PI;
    float sa, ca;
    __sincosf(upper ? TWOPI - ri1 : ri1, &sa, &ca);
    cost = costp * bmu + sintp * sinbt * ca;
    float sini2, cosi2;
    if (fabsf(cost) < 1.f) {
        sint = sqrt_ax(1.f - cost * cost);
        const float rs = rcp_ax(sint);
        sini2 = sa * sintp * rs;
        cosi2 = (costp - cost * bmu) * rs * rcp_ax(sinbt);
    } else {
        sint = 0.f;
        sini2 = 0.f;
        cosi2 = cost >= 1.f ? -1.f : 1.f;
    }
    float cosdph = -cosi2 * ca + sini2 * sa * bmu;
    cosdph = fminf(fmaxf(cosdph, -1.f), 1.f);
    float sdph = sqrt_ax(1.f - cosdph * cosdph);
    sdph = upper ? sdph : -sdph;
    const float ncp = cp * cosdph - sp * sdph, nsp = sp * cosdph + cp * sdph;
    const float rn = rsqrt_ax(ncp * ncp + nsp * nsp);
    cp = ncp * rn;
    sp = nsp * rn;
    return true;
}

// Unpolarised Fresnel reflectance n1 -> n2 at incidence cosine cosi.
template <typename Real> __device__ __forceinline__ Real fresnel(Real n1, Real n2, Real cosi)
{
    if (n1 == n2) return (Real)0;
    if (cosi > (Real)1) cosi = (Real)1;
    const Real sini = M<Real>::sqrt((Real)1 - cosi * cosi);
    const Real st = n1 / n2 * sini;
    if (st >= (Real)1) return (Real)1;
    const Real ct = M<Real>::sqrt((Real)1 - st * st);
    const Real rs = M<Real>::div(n1 * cosi - n2 * ct, n1 * cosi + n2 * ct);
    const Real rp = M<Real>::div(n1 * ct - n2 * cosi, n1 * ct + n2 * cosi);
    return (Real)0.5 * (rs * rs + rp * rp);
}

template <typename Real> __device__ __forceinline__ Real clamp0h(Real f, Real h)
{
    return f < (Real)0 ? (Real)0 : (f > h ? h : f);
}

// Voxel steps per warp vote of the flight phase: the votes are a sizeable
// share of a step, and a lane that stops early only idles for the rest (its
// packet's walk does not depend on when the event batch runs).
constexpr int VSTEPS = 4;

// Dead lanes of a warp that make it draw new packets: the launch code runs
// for the dead lanes only, so refilling them together spends fewer of its
// warp instructions per packet, while they idle in the flight phase meanwhile.
// On the 200^3 bench pass: 1 -> 516.2, 2 -> 513.4, 4 -> 526.3, 8 -> 573.2 ms
// per 1e8 packets.
#ifndef TAM_REFILL_MIN
#define TAM_REFILL_MIN 2
#endif

// Lanes that must wait before a warp with `live` live lanes runs its event
// batch: scat_min of 32, and the same share of fewer (FP32: in FP64 the event
// batch keeps the FP64 pipe busy as long for few lanes as for many, and taking
// it earlier costs 7 % on passes of 1e5 packets).
__device__ __forceinline__ int wait_min(int scat_min, int live)
{
    return live >= 31 ? scat_min : max(1, (scat_min * live) >> 5);
}

// Packets that a warp holds at a time: with fewer packets than lanes, a pass
// takes as long as its longest packet's walk, whose events wait for those of
// the other lanes, so a small pass spreads over the SMs, one block each, before
// its warps fill up.  100^3 cube, FP32, 1 / 4 / 32 packets a warp: 1.08 / 1.16 /
// 1.33 ms for 1000 packets, 2.2 / 1.83 / 1.91 ms for 10,000, 7.9 / 4.2 / 2.4 ms
// for 100,000.
inline int packets_per_warp(int64_t n, int64_t warps)
{
    const int64_t k = (n + warps - 1) / warps;
    return (int)(k < 1 ? 1 : (k > 32 ? 32 : k));
}

__device__ __forceinline__ bool not_negative(float a) { return a >= 0.f; }
__device__ __forceinline__ bool not_negative(double a) { return (int64_t)ieee::bits(a) >= 0; }

// Per-flight DDA set-up from the in-cell position f and direction n of one
// axis: td = cell width along the ray, tm = distance to the next face.
template <typename Real>
__device__ __forceinline__ void axis_setup(Real n, Real f, Real h, Real BIG, Real &td, Real &tm, int &sg);
// FP64: no compare and no division with special cases; a tiny |n| counts as
// parallel to the faces.
template <>
__device__ __forceinline__ void axis_setup<double>(double n, double f, double h, double BIG, double &td, double &tm, int &sg)
{
    const bool par = is_tiny(n), minus = is_minus(n);
    const double inv = rcp64(n);
    const double to = (minus ? -f : h - f) * inv;
    td = par ? BIG : h * fabs(inv);
    tm = par ? BIG : (is_minus(to) ? 0.0 : to);
    sg = par || minus ? -1 : 1;
}
// FP32: approximate reciprocal; |n| below 1e-30 counts as parallel to the
// faces (its reciprocal would overflow and turn 0 * inf into NaN).
template <>
__device__ __forceinline__ void axis_setup<float>(float n, float f, float h, float BIG, float &td, float &tm, int &sg)
{
    const float inv = rcp_ax(n);
    const bool par = fabsf(n) < 1e-30f;
    td = par ? BIG : h * fabsf(inv);
    tm = par ? BIG : (n > 0.f ? h - f : -f) * inv;
    tm = tm < 0.f ? 0.f : tm;
    sg = n > 0.f ? 1 : -1;
}

// In-cell position of one axis at distance t along the flight.
template <typename Real> __device__ __forceinline__ Real axis_pos(Real n, Real f, Real h, Real tm, Real t)
{
    const Real r = n > (Real)0 ? h - (tm - t) * n : (n < (Real)0 ? -(tm - t) * n : f);
    return clamp0h(r, h);
}
template <> __device__ __forceinline__ double axis_pos<double>(double n, double f, double h, double tm, double t)
{
    const bool minus = is_minus(n);
    const double d = tm - t, r = is_tiny(n) ? f : __fma_rn(-d, n, minus ? 0.0 : h);
    return is_minus(r) ? 0.0 : (less_pos(h, r) ? h : r);
}

// VSTEPS voxel steps (src/inttau2.f90:37-63) of the FP32 distance-tracked
// flight in a uniform medium, as predicated PTX: per step the deposit of the
// cell's path (one red.f64), the crossing of the nearest face (ties go z over
// y over x, src/inttau2.f90:116-118; a two-output setp gives "this axis" and
// "a later axis" at once) and the test whether the flight goes on (the cell
// is inside the grid and the next face lies before the interaction point at
// distance tau).  `go` (0 or 1) and tmin = min(tmx, tmy, tmz) are kept ahead
// by one step; a lane without `go` is left unchanged.
//
// The transport is bound by instruction issue.  As C++ the compiler turns
// each conditional update into an operation and a select; predicated, a step
// is 27 instructions against 44.
#define TAM_VSTEP_PTX                                                                                       \
    "sub.f32 a, %5, %3;\n\t"                                                                                \
    "mul.f32 a, %14, a;\n\t"                                                                               \
    "fma.rn.f32 a, a, %15, %4;\n\t"                                                                        \
    "mad.lo.s32 c, %8, %21, %7;\n\t"                                                                       \
    "mad.lo.s32 c, c, %20, %6;\n\t"                                                                        \
    "mul.wide.s32 l, c, 8;\n\t"                                                                            \
    "add.s64 l, l, %23;\n\t"                                                                               \
    "cvt.f64.f32 d, a;\n\t"                                                                             \
    "@p red.global.add.f64 [l], d;\n\t"                                                                    \
    "@p mov.f32 %4, 0f00000000;\n\t"                                                                       \
    "@p mov.f32 %3, %5;\n\t"                                                                               \
    "@p add.u32 %9, %9, 1;\n\t"                                                                            \
    "setp.eq.and.f32 pz|q, %2, %5, p;\n\t"                                                                 \
    "setp.eq.and.f32 py|px, %1, %5, q;\n\t"                                                                \
    "@px add.f32 %0, %0, %11;\n\t"                                                                         \
    "@py add.f32 %1, %1, %12;\n\t"                                                                         \
    "@pz add.f32 %2, %2, %13;\n\t"                                                                         \
    "@px add.s32 %6, %6, %17;\n\t"                                                                         \
    "@py add.s32 %7, %7, %18;\n\t"                                                                         \
    "@pz add.s32 %8, %8, %19;\n\t"                                                                         \
    "setp.lt.and.u32 p, %6, %20, p;\n\t"                                                                   \
    "setp.lt.and.u32 p, %7, %21, p;\n\t"                                                                   \
    "setp.lt.and.u32 p, %8, %22, p;\n\t"                                                                   \
    "min.f32 %5, %0, %1, %2;\n\t"                                                                          \
    "setp.lt.and.f32 p, %5, %16, p;\n\t"
__device__ __forceinline__ void fly_steps(float &tmx, float &tmy, float &tmz, float &t, float &dep, float &tmin, int &ix,
                                          int &iy, int &iz, uint32_t &nsteps, int &go, float tdx, float tdy, float tdz,
                                          float w, float mua, float tau, int sgx, int sgy, int sgz, int NX, int NY, int NZ,
                                          double *tally)
{
    static_assert(VSTEPS == 4, "the steps below");
    asm volatile("{\n\t"
                 ".reg .pred p, q, px, py, pz;\n\t"
                 ".reg .f32 a;\n\t"
                 ".reg .s32 c;\n\t"
                 ".reg .s64 l;\n\t"
                 ".reg .f64 d;\n\t"
                 "setp.ne.s32 p, %10, 0;\n\t"
                 TAM_VSTEP_PTX TAM_VSTEP_PTX TAM_VSTEP_PTX TAM_VSTEP_PTX
                 "selp.s32 %10, 1, 0, p;\n\t"
                 "}"
                 : "+f"(tmx), "+f"(tmy), "+f"(tmz), "+f"(t), "+f"(dep), "+f"(tmin), "+r"(ix), "+r"(iy), "+r"(iz),
                   "+r"(nsteps), "+r"(go)
                 : "f"(tdx), "f"(tdy), "f"(tdz), "f"(w), "f"(mua), "f"(tau), "r"(sgx), "r"(sgy), "r"(sgz), "r"(NX),
                   "r"(NY), "r"(NZ), "l"(tally)
                 : "memory");
}
#undef TAM_VSTEP_PTX

// The crossing of one step in FP32 without the deposit, for media whose cells
// differ: the caller deposits before it and looks the new cell up after it.
// dtx, dty, dtz: what a crossing adds to the crossed axis's face distance;
// ahead: the optical depth to the face.
__device__ __forceinline__ void fly_cross(float &tmx, float &tmy, float &tmz, float &t, float &dep, float &tmin, float &tau,
                                          int &ix, int &iy, int &iz, uint32_t &nsteps, int &go, float dtx, float dty,
                                          float dtz, float ahead, int sgx, int sgy, int sgz, int NX, int NY, int NZ)
{
    asm("{\n\t"
        ".reg .pred p, q, px, py, pz;\n\t"
        "setp.ne.s32 p, %11, 0;\n\t"
        "@p sub.f32 %6, %6, %15;\n\t"
        "@p mov.f32 %4, 0f00000000;\n\t"
        "@p mov.f32 %3, %5;\n\t"
        "@p add.u32 %10, %10, 1;\n\t"
        "setp.eq.and.f32 pz|q, %2, %5, p;\n\t"
        "setp.eq.and.f32 py|px, %1, %5, q;\n\t"
        "@px add.f32 %0, %0, %12;\n\t"
        "@py add.f32 %1, %1, %13;\n\t"
        "@pz add.f32 %2, %2, %14;\n\t"
        "@px add.s32 %7, %7, %16;\n\t"
        "@py add.s32 %8, %8, %17;\n\t"
        "@pz add.s32 %9, %9, %18;\n\t"
        "setp.lt.and.u32 p, %7, %19, p;\n\t"
        "setp.lt.and.u32 p, %8, %20, p;\n\t"
        "setp.lt.and.u32 p, %9, %21, p;\n\t"
        "min.f32 %5, %0, %1, %2;\n\t"
        "selp.s32 %11, 1, 0, p;\n\t"
        "}"
        : "+f"(tmx), "+f"(tmy), "+f"(tmz), "+f"(t), "+f"(dep), "+f"(tmin), "+f"(tau), "+r"(ix), "+r"(iy), "+r"(iz),
          "+r"(nsteps), "+r"(go)
        : "f"(dtx), "f"(dty), "f"(dtz), "f"(ahead), "r"(sgx), "r"(sgy), "r"(sgz), "r"(NX), "r"(NY), "r"(NZ));
}

// Whether a direction lies (nearly) in a plane of the grid: the two functions
// below do not take it.
__device__ __forceinline__ bool in_plane(float nx, float ny, float nz)
{
    return fminf(fminf(fabsf(nx), fabsf(ny)), fabsf(nz)) < 1e-30f;
}
// axis_setup and axis_pos of a component that is not parallel to the faces,
// and of 0 <= f <= h: the same values (a sign moves through a product, and
// h - f and f are not negative) with about half the instructions.
__device__ __forceinline__ void axis_setup_steep(float n, float f, float h, float &td, float &tm, int &sg)
{
    const float inv = fabsf(rcp_ax(n));
    td = h * inv;
    tm = (n > 0.f ? h - f : f) * inv;
    sg = n > 0.f ? 1 : -1;
}
__device__ __forceinline__ float axis_pos_steep(float n, float h, float tm, float t)
{
    const float e = tm - t;
    const float r = n > 0.f ? __fmaf_rn(-e, n, h) : -e * n;
    return fminf(fmaxf(r, 0.f), h);
}

// One FP32 scatter: the packet's in-cell position at distance t of its
// flight, the HG rotation of its direction, and the new flight's set-up.
// True when the new direction needs a closer look (NaN, or in a plane of the
// grid: the face distances then come from axis_setup); the test, a few
// instructions and rarely true, stands in for a branch at each of its parts.
__device__ __forceinline__ bool scatter_f32(const HgF &hg, float u0, float u1, float hx, float hy, float hz, float t,
                                            float &fx, float &fy, float &fz, float &nx, float &ny, float &nz, float &sint,
                                            float &cpv, float &spv, float &tdx, float &tdy, float &tdz, float &tmx,
                                            float &tmy, float &tmz, int &sgx, int &sgy, int &sgz)
{
    if (in_plane(nx, ny, nz)) {
        fx = axis_pos(nx, fx, hx, tmx, t);
        fy = axis_pos(ny, fy, hy, tmy, t);
        fz = axis_pos(nz, fz, hz, tmz, t);
    } else {
        fx = axis_pos_steep(nx, hx, tmx, t);
        fy = axis_pos_steep(ny, hy, tmy, t);
        fz = axis_pos_steep(nz, hz, tmz, t);
    }
    float cost = nz;
    if (stokes_f32(hg, u0, u1, cost, sint, cpv, spv)) {
        nx = sint * cpv;
        ny = sint * spv;
        nz = cost;
    }
    axis_setup_steep(nx, fx, hx, tdx, tmx, sgx);
    axis_setup_steep(ny, fy, hy, tdy, tmy, sgy);
    axis_setup_steep(nz, fz, hz, tdz, tmz, sgz);
    return in_plane(nx, ny, nz) || !(nz == nz) || !(nx == nx) || !(ny == ny);
}

}  // namespace
}  // namespace tam
