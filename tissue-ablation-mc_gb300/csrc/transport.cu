// transport.cu -- photon-packet transport on sm_103a.
//
// One packet per thread, persistent warps that refill dead lanes from a
// global packet counter (warp-aggregated).  Each lane walks its packet
// through the voxel grid with a cell-relative DDA, scatters with the
// Henyey-Greenstein rotation of src/stokes.f90:6-153, applies Fresnel faces
// and Russian roulette, and deposits w*d*mua per voxel visit (the path-length
// absorption estimator of src/inttau2.f90:46,53) into the FP64 tally with one
// red.global.add.f64 per visit.
//
// Follows: src/sourceph.f90:7-49 (launch), src/inttau2.f90:7-121 (tau
// integration and wall distance), src/stokes.f90:6-153 (HG), src/ch_opt.f90
// (optical constants via the material table).  Random numbers come from
// Philox4x32-10 with counter {event, packet_lo, packet_hi, stream}.
#include <curand_philox4x32_x.h>

#include <algorithm>
#include <type_traits>

#include "tam_device.cuh"
#include "tam_kernels.h"
#include "scatter64.cuh"
#include "transport_common.cuh"

namespace tam {

namespace {

constexpr int TPB = 256;
// Resident blocks per SM requested for the FP32 transport kernel (register cap).
#ifndef TAM_TR_MINB
#define TAM_TR_MINB 4
#endif

// Tally update of one voxel visit: an FP64 reduction into jmean (L2-resident
// for grids up to ~16 M voxels), or -- for grids whose FP64 tally is far
// larger than L2 -- an FP32 reduction into a box-sized tally around the
// beam's entry, which stays L2-resident and which the host flushes into
// jmean every few million packets; the rare deposits outside the box go to
// jmean directly.
template <bool T32, typename Real>
__device__ __forceinline__ void deposit(const TransportArgs &a, int cidx, int ix, int iy, int iz, Real dep)
{
    if constexpr (T32) {
        const unsigned bx = (unsigned)(ix - a.bx0), by = (unsigned)(iy - a.by0), bz = (unsigned)(iz - a.bz0);
        if (bx < (unsigned)a.bnx && by < (unsigned)a.bny && bz < (unsigned)a.bnz) {
            atomicAdd(a.jmean32 + (bx + (unsigned)a.bnx * (by + (unsigned)a.bny * bz)), (float)dep);
            return;
        }
    }
    atomicAdd(a.jmean + cidx, (double)dep);
}

// Optical properties of the current cell: extinction and absorption for the
// DDA, the material id for the albedo / HG / index lookups at events.  A
// uniform medium (every voxel the same material) needs no per-cell fetch.
template <typename Real, int MED>
__device__ __forceinline__ void fetch(const TransportArgs &a, const MatR<Real> *lut, int ix, int iy, int iz,
                                      int cidx, Real &mut, Real &mua, int &mid)
{
    if (MED == MED_RHOKAP) {
        const int64_t hx = a.nx + 2, hy = a.ny + 2;
        const Real v = (Real)__ldg(a.rhokap + ((ix + 1) + hx * ((iy + 1) + hy * (int64_t)(iz + 1))));
        mut = v;
        mua = v;
        mid = 0;
    } else if (MED == MED_MATERIAL) {
        // large grids: most cells lie in bricks of one material, whose id the
        // small (L2- and mostly L1-resident) brick table holds; the material
        // grid itself is read only inside mixed bricks
        int id;
        if (a.btab) {
            id = __ldg(a.btab + ((ix >> 3) + a.bbx * ((iy >> 3) + a.bby * (iz >> 3))));
            if (id == 0xFF) id = __ldg(a.mat + cidx);
        } else {
            id = __ldg(a.mat + cidx);
        }
        id = id < a.nmat ? id : 0;
        mid = id;
        mut = lut[id].mut;
        mua = lut[id].mua;
    } else {
        mid = a.uniform_id;
        mut = lut[mid].mut;
        mua = lut[mid].mua;
    }
}

// A lane is alive (holds a packet) or dead, and while alive its packet either
// flies on (`go`: its next event is the crossing of a voxel face) or waits for
// the event batch, at an interaction point or on an outer face.  `go` is
// worked out ahead, at the end of the step before, so a flight of k crossings
// takes k steps and a lane that has stopped is left as it is by further steps:
// the step is straight-line code under one predicate, without branches.  The
// events (Philox block, HG rotation, roulette, new optical depth; Fresnel
// reflect-or-escape) are the expensive part; the event batch runs once at
// least scat_min lanes of the warp wait (in FP32 fewer when lanes are dead, see
// wait_min), or when no lane flies, so it executes with most lanes active.
// Every packet sees the same sequence of events and random numbers as a
// straight loop.
//
// What bounds it is instruction issue (80 % of cycles; 23 of 32 lanes active):
// on the 200^3 bench pass (1e8 packets) this form takes 369 ms against 510 ms
// for a step that tested the lane's state, the cap and the interaction in
// nested branches (5491 -> about 3900 warp instructions per packet); 47 against
// 64 ms per 1e7 packets on the three-layer slab, 154 against 192 ms on a 384^3
// vessel grid.  scat_min 12 to 24 are within 1 % of each other; 2, 3 and 6
// voxel steps per vote are 5, 3 and 2 % slower than 4.  FP64: see SCAT_MIN64.
//
// The DDA is incremental (Amanatides & Woo): per flight, the distance tm to
// the next face of each axis and the cell width td along the ray; a crossing
// moves tm of the crossed axis by td.  In-cell positions are reconstructed
// only at events (interaction, outer face).
template <typename Real> __device__ __forceinline__ const TrConst<Real> &consts(const TransportArgs &a)
{
    if constexpr (sizeof(Real) == 4) return a.cf;
    else return a.cd;
}

template <typename Real> __device__ __forceinline__ const MatR<Real> *mats(const TransportArgs &a)
{
    if constexpr (sizeof(Real) == 4) return a.mf;
    else return a.md;
}

template <typename Real, int MED, bool T32>
__global__ void __launch_bounds__(TPB, sizeof(Real) == 4 ? TAM_TR_MINB : 2) transport_kernel(const __grid_constant__ TransportArgs a, int scat_min, unsigned lanes)
{
    __shared__ MatR<Real> lut[MAX_MAT];
    __shared__ HgF hgt[sizeof(Real) == 4 ? MAX_MAT : 1];
    if constexpr (MED != MED_RHOKAP) {
        for (int t = threadIdx.x; t < MAX_MAT; t += blockDim.x) {
            lut[t] = mats<Real>(a)[t];
            if constexpr (sizeof(Real) == 4) hgt[t] = hg_consts(lut[t].g, lut[t].g2);
        }
    }
    // per-packet (rare) tallies accumulate in shared memory, not registers
    __shared__ double s_tal[5];  // specular, reflected, transmitted, side, roulette net
    __shared__ unsigned long long s_cnt[2];  // voxel steps, scatters
    __shared__ unsigned s_entered[MAX_MAT];  // packets launched into each material (FP32)
    __shared__ unsigned s_err;
    constexpr bool SCAT64 = sizeof(Real) == 8 && MED != MED_RHOKAP;  // the reference medium only absorbs
    if (threadIdx.x < 5) s_tal[threadIdx.x] = 0.0;
    if (threadIdx.x < 2) s_cnt[threadIdx.x] = 0ull;
    if (threadIdx.x < MAX_MAT) s_entered[threadIdx.x] = 0u;
    if (threadIdx.x == 0) s_err = 0u;
    __syncthreads();

    const unsigned FULL = 0xffffffffu;
    const TrConst<Real> &K = consts<Real>(a);
    const Real hx = K.hx, hy = K.hy, hz = K.hz;
    const Real BIG = (Real)1.0e30;
    const Real TWOPI = (Real)TWOPI_R;
    // after a crossing the next face along the crossed axis is (h - nudge)
    // away along the axis: tm advances by td * (1 - nudge / h)
    const Real knx = K.knx, kny = K.kny, knz = K.knz;
    const uint32_t strm = a.stream_dev ? *a.stream_dev : a.stream;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned warp_id = blockIdx.x * (TPB / 32) + (threadIdx.x >> 5), nwarps = gridDim.x * (TPB / 32);
    const bool one_draw = (unsigned long long)nwarps * __popc(lanes) >= (unsigned long long)a.n;
    bool first = true;
    const Real wmin = K.wmin, rm = K.rm, inv_rm = K.inv_rm;
    // weights below this need a look after a scatter: roulette, or the end of a packet without weight
    const Real w_rare = a.roulette && wmin > (Real)0 ? wmin : (Real)1.401298464e-45;
    const int NX = a.nx, NY = a.ny, NZ = a.nz;
    const uint32_t max_steps = a.max_steps > 0xfffffff0ll ? 0xfffffff0u : (uint32_t)a.max_steps;
    const Real namb = K.namb;
    // FP32 in a uniform medium: the flight is tracked by distance (tau / mut
    // once per flight) instead of optical depth per voxel step
    constexpr bool DIST = sizeof(Real) == 4 && MED == MED_UNIFORM;
    const Real inv_mut = DIST ? (Real)1 / lut[a.uniform_id >= 0 ? a.uniform_id : 0].mut : (Real)0;
    // a uniform medium's properties stay in registers (no fetch per crossing)
    const int mid_u = MED == MED_UNIFORM ? (a.uniform_id >= 0 ? a.uniform_id : 0) : 0;
    const Real mut_u = lut[mid_u].mut, mua_u = lut[mid_u].mua;
    // only the reference medium nudges a crossed coordinate past the face
    // (config mode's factor is exactly 1)
    constexpr bool NUDGE = MED == MED_RHOKAP;

    bool alive = false;
    bool exhausted = false;
    int ix = 0, iy = 0, iz = 0, mid = 0, sgx = 1, sgy = 1, sgz = 1;
    auto cell = [&]() { return ix + NX * (iy + NY * iz); };
    Real fx = 0, fy = 0, fz = 0, nx = 0, ny = 0, nz = 0, sint = 0;
    Real cpv = 1, spv = 0;  // (cos phi, sin phi)
    Real tdx = 0, tdy = 0, tdz = 0, tmx = 0, tmy = 0, tmz = 0, t = 0;
    Real w = 0, tau = 0, dep = 0, mut = 0, mua = 0;
    uint32_t ev = 0, plo = 0, phi32 = 0, nsteps = 0;
    uint32_t cScat = 0;
    // The specular tally: FP64 additions to one shared word go lane by lane, a compare
    // and swap each, 32 of them whenever a warp launches together, which packets that
    // end after a few steps do often.  So FP64 sums in a register, and FP32, short of
    // registers, counts the packets that entered each material, one instruction for the
    // warp (2e6 packets, 128^3, mua 50 / mus 10 per cm: 939 -> 697 us).
    constexpr bool SPEC_REG = sizeof(Real) == 8;
    double spec = 0.0;
    uint64_t cSteps = 0;  // voxel steps of this thread's finished packets (reduced once at the end)
    auto props = [&]() {
        if constexpr (MED == MED_UNIFORM) {
            mid = mid_u;
            mut = mut_u;
            mua = mua_u;
        } else {
            fetch<Real, MED>(a, lut, ix, iy, iz, cell(), mut, mua, mid);
        }
    };

    for (;;) {
        // ---------------------------------------------- refill dead lanes --
        // (exhausted is warp-uniform: set once the counter has passed n)
        unsigned live = __ballot_sync(FULL, alive);
        const unsigned need = exhausted ? 0u : ~live & lanes;
        if (need && (__popc(need) >= TAM_REFILL_MIN || live == 0u)) {
            // the first packets by the warp's place in the launch, the others
            // from the counter of those drawn beyond them
            unsigned long long base = first ? (unsigned long long)warp_id * __popc(lanes) : 0;
            if (!first) {
                const int leader = __ffs(need) - 1;
                if ((int)lane == leader) base = atomicAdd(a.work, (unsigned long long)__popc(need));
                base = __shfl_sync(FULL, base, leader) + (unsigned long long)nwarps * __popc(lanes);
            }
            first = false;
            exhausted = base + (unsigned long long)__popc(need) >= (unsigned long long)a.n || one_draw;
            if (need >> lane & 1u) {
                const unsigned long long my = base + __popc(need & ((1u << lane) - 1u));
                if (my < (unsigned long long)a.n) {
                    // launch (src/sourceph.f90:7-49; Gaussian beam in config mode)
                    const uint64_t pid = (uint64_t)a.p0 + my;
                    plo = (uint32_t)pid;
                    phi32 = (uint32_t)(pid >> 32);
                    const U4 r = philox4x32_10_rk(0u, plo, phi32, strm, a.rk);
                    ev = 1;
                    const Real u0 = Uniform<Real>::from(r.x), u1 = Uniform<Real>::from(r.y);
                    const Real u2 = Uniform<Real>::from(r.z), u3 = Uniform<Real>::from(r.w);
                    const Real R = K.src_r;
                    auto root = [](Real x) {
                        if constexpr (sizeof(Real) == 8) return sqrt64(x);
                        else return M<Real>::sqrt(x);
                    };
                    const Real rad = a.source == SRC_DISK ? root(u0 * (R * R)) : R * root((Real)0.5 * M<Real>::neglog(u0));
                    Real st, ct, sp, cp;
                    if constexpr (sizeof(Real) == 8) turn(r.y, st, ct);
                    else M<Real>::sincos(u1 * TWOPI, &st, &ct);
                    const Real X = rad * ct + K.xmax, Y = rad * st + K.ymax;
                    if constexpr (MED == MED_RHOKAP) {
                        // reference medium: a pure absorber (any interaction
                        // ends the packet) launched straight down, so the
                        // azimuth only enters nx = ny = sint * (cos, sin) phi
                        // = +-0, which the walk treats alike; its sincos is skipped
                        cp = (Real)1;
                        sp = (Real)0;
                    } else {
                        if constexpr (SCAT64) turn(r.z, sp, cp);
                        else M<Real>::sincos(TWOPI * u2, &sp, &cp);
                    }
                    cpv = cp;
                    spv = sp;
                    sint = (Real)0;
                    if (!(not_negative(X) && less_pos(X, K.w2x) && not_negative(Y) && less_pos(Y, K.w2y))) {
                        atomicAdd(a.tally + T_MISSED, 1.0);
                    } else {
                        // (FP64: a product; each quotient is ten operations of its pipe)
                        ix = (int)(sizeof(Real) == 8 ? X * K.cells_x : (Real)NX * X / K.w2x);
                        iy = (int)(sizeof(Real) == 8 ? Y * K.cells_y : (Real)NY * Y / K.w2y);
                        ix = ix > NX - 1 ? NX - 1 : ix;
                        iy = iy > NY - 1 ? NY - 1 : iy;
                        iz = NZ - 1;
                        // (straight down: only after a reflection do x and y matter)
                        if (sizeof(Real) == 4 || a.fresnel || MED != MED_RHOKAP) {
                            fx = X - (Real)ix * hx;
                            fy = Y - (Real)iy * hy;
                        }
                        fz = hz - (Real)1.e-8 * hz;
                        props();
                        w = (Real)1;
                        if (a.fresnel) {
                            const Real nt = MED == MED_RHOKAP ? K.rhokap_n : lut[mid].n;
                            Real rsp = K.rhokap_spec;
                            if constexpr (sizeof(Real) == 4 || MED != MED_RHOKAP) {
                                rsp = (namb - nt) / (namb + nt);
                                rsp = rsp * rsp;
                            }
                            if constexpr (SPEC_REG) spec += (double)rsp;
                            else atomicAdd(&s_entered[MED == MED_MATERIAL ? mid : 0], 1u);
                            w = (Real)1 - rsp;
                        }
                        tau = M<Real>::neglog(u3);
                        if constexpr (DIST) tau *= inv_mut;
                        nx = sint * cp;  // direction (0, 0, -1): +-0 in x and y
                        ny = sint * sp;
                        nz = (Real)-1;
                        // the set-up of that direction, without its divisions
                        tdx = tdy = tmx = tmy = BIG;
                        sgx = sgy = sgz = -1;
                        tdz = hz;
                        tmz = fz;
                        t = (Real)0;
                        dep = (Real)0;
                        nsteps = 0;
                        alive = true;
                    }
                }
            }
            live = __ballot_sync(FULL, alive);
        }
        if (live == 0u) {
            if (exhausted) break;
            continue;
        }
        // ------------------------------------------------- flight phase --
        // voxel steps of the flying lanes until enough lanes wait for the
        // event batch or none flies
        Real tmin, ahead, gap;
        bool px = false, py = false, pz = false;  // FP64: the axis of the next face
        // whether the flight's interaction point lies beyond the next face
        // (ties between faces go z over y over x, src/inttau2.f90:116-118)
        auto look = [&]() {
            if constexpr (sizeof(Real) == 4) {
                tmin = fminf(fminf(tmx, tmy), tmz);
            } else {
                const bool yz = less_pos(tmy, tmz);
                tmin = yz ? tmy : tmz;
                px = less_pos(tmx, tmin);
                tmin = px ? tmx : tmin;
                py = yz && !px;
                pz = !yz && !px;
            }
            gap = tmin - t;
            ahead = DIST ? tmin : gap * mut;  // distance, or optical depth to the face
            return less_pos(ahead, tau);
        };
        bool go = look() && alive, capped = false;
        // one voxel step (src/inttau2.f90:37-63) of the lanes with `go`
        auto vstep = [&](auto careful) {
            if constexpr (decltype(careful)::value) {
                // a packet past its step cap ends here, before the step
                if (go && nsteps >= max_steps) {
                    nsteps += 1;
                    capped = true;
                    go = false;
                }
            }
            const Real d = dep + w * (sizeof(Real) == 8 ? gap : tmin - t) * mua;
            if (go) deposit<T32>(a, cell(), ix, iy, iz, d);
            // step into the next cell, branch-free over the axis; the
            // reference snaps the crossed coordinate to the face +- delta
            // (src/inttau2.f90:140-169), which knx/kny/knz carry.  Past an
            // outer face the lane waits for the event batch.
            if constexpr (sizeof(Real) == 4) {
                int g = go;
                fly_cross(tmx, tmy, tmz, t, dep, tmin, tau, ix, iy, iz, nsteps, g, NUDGE ? tdx * knx : tdx,
                          NUDGE ? tdy * kny : tdy, NUDGE ? tdz * knz : tdz, DIST ? 0.f : ahead, sgx, sgy, sgz, NX, NY, NZ);
                go = g != 0;
            } else {
                nsteps += go ? 1u : 0u;
                dep = go ? (Real)0 : dep;
                tau = go ? tau - ahead : tau;
                t = go ? tmin : t;
                const bool cx = go && px, cy = go && py, cz = go && pz;
                // (the crossed axis chosen first: one FP64 addition, not three)
                const Real td = px ? tdx : (py ? tdy : tdz);
                const Real next = tmin + (NUDGE ? td * (px ? knx : (py ? kny : knz)) : td);
                tmx = cx ? next : tmx;
                tmy = cy ? next : tmy;
                tmz = cz ? next : tmz;
                ix += cx ? sgx : 0;
                iy += cy ? sgy : 0;
                iz += cz ? sgz : 0;
                go = go && (unsigned)ix < (unsigned)NX && (unsigned)iy < (unsigned)NY && (unsigned)iz < (unsigned)NZ;
            }
            if constexpr (MED != MED_UNIFORM) {
                if (go) props();
            }
            go = look() && go;
        };
        {
            const int thr = sizeof(Real) == 4 ? wait_min(scat_min, __popc(live)) : scat_min;
            // a flight crosses at most NX + NY + NZ faces between two outer
            // faces, so only packets that near their cap need the test per step
            const uint32_t far = (uint32_t)NX + (uint32_t)NY + (uint32_t)NZ + 2u;
            if (max_steps >= far && !__any_sync(FULL, alive && nsteps > max_steps - far)) {
                for (;;) {
                    const unsigned fl = __ballot_sync(FULL, go);
                    if (fl == 0u || __popc(live & ~fl) >= thr) break;
                    if constexpr (DIST && !T32) {
                        int g = go;
                        fly_steps(tmx, tmy, tmz, t, dep, tmin, ix, iy, iz, nsteps, g, tdx, tdy, tdz, w, mua, tau, sgx, sgy,
                                  sgz, NX, NY, NZ, a.jmean);
                        go = g != 0;
                    } else {
#pragma unroll
                        for (int q = 0; q < (MED == MED_RHOKAP || sizeof(Real) == 8 ? 1 : VSTEPS); ++q) vstep(std::false_type{});
                    }
                }
            } else {
                for (;;) {
                    const unsigned fl = __ballot_sync(FULL, go);
                    if (fl == 0u || __popc(live & ~fl) >= thr) break;
                    vstep(std::true_type{});
                }
                // the interaction counts as a step too
                const bool in = (unsigned)ix < (unsigned)NX && (unsigned)iy < (unsigned)NY && (unsigned)iz < (unsigned)NZ;
                if (alive && !go && !capped && in && nsteps >= max_steps) {
                    nsteps += 1;
                    capped = true;
                }
                if (capped) {
                    if (dep != (Real)0) deposit<T32>(a, cell(), ix, iy, iz, dep);
                    dep = (Real)0;
                    atomicAdd(a.tally + T_OVERFLOW, 1.0);
                    atomicOr(&s_err, (unsigned)DEVERR_STEP_CAP);
                    cSteps += nsteps;
                    alive = false;
                }
            }
        }

        // ------------------------------------------------- event batch --
        // interactions (implicit capture, HG scatter, roulette) and Fresnel
        // faces, handled together once enough lanes wait; both kinds draw
        // their uniforms from one Philox block per lane
        {
            const bool cx = (unsigned)ix >= (unsigned)NX, cy = (unsigned)iy >= (unsigned)NY;
            const bool cz = (unsigned)iz >= (unsigned)NZ, face = cx || cy || cz;
            // the packet's end
            auto end = [&]() {
                if (dep != (Real)0) deposit<T32>(a, cell(), ix, iy, iz, dep);
                dep = (Real)0;
                cSteps += nsteps;
                alive = false;
            };
            // on to the interaction point inside this cell
            auto interact = [&]() {
                nsteps += 1;
                if constexpr (DIST) {
                    // tau holds the flight distance of the interaction point
                    dep += w * (tau - t) * mua;
                    t = tau;
                } else if constexpr (sizeof(Real) == 8 && MED == MED_RHOKAP) {
                    dep += w * tau;  // a pure absorber, mua = mut, and the packet ends here
                } else {
                    Real dd;
                    if constexpr (sizeof(Real) == 8) dd = div64(tau, mut);
                    else dd = M<Real>::div(tau, mut);
                    dep += w * dd * mua;
                    t += dd;
                }
                w *= MED == MED_RHOKAP ? (Real)0 : lut[mid].alb;
            };
            // an outer face: reflect or escape (without Fresnel: escape)
            auto surface = [&](uint32_t draw) {
                const Real nc = cx ? nx : (cy ? ny : nz);
                const Real nt = MED == MED_RHOKAP ? K.rhokap_n : lut[mid].n;
                if (!a.fresnel || !(Uniform<Real>::from(draw) < fresnel<Real>(nt, namb, M<Real>::abs(nc)))) {
                    atomicAdd(&s_tal[cz ? (sgz > 0 ? 1 : 2) : 3], (double)w);
                    cSteps += nsteps;  // nothing to deposit: the crossing did
                    alive = false;
                    return;
                }
                // reflect, back into the cell it came from: mirror the crossed
                // direction component; the next face along it is one cell
                // width back
                if (cx) {
                    ix -= sgx;
                    fy = axis_pos(ny, fy, hy, tmy, t);
                    fz = axis_pos(nz, fz, hz, tmz, t);
                    fx = sgx > 0 ? hx : (Real)0;
                    nx = -nx;
                    sgx = -sgx;
                    tmx = t + tdx;
                    if constexpr (SCAT64) {
                        const Azimuth p = mirror_x(Azimuth{cpv, spv});
                        cpv = p.c;
                        spv = p.s;
                    } else {
                        cpv = -cpv;  // phi -> PI - phi
                    }
                } else if (cy) {
                    iy -= sgy;
                    fx = axis_pos(nx, fx, hx, tmx, t);
                    fz = axis_pos(nz, fz, hz, tmz, t);
                    fy = sgy > 0 ? hy : (Real)0;
                    ny = -ny;
                    sgy = -sgy;
                    tmy = t + tdy;
                    if constexpr (SCAT64) {
                        const Azimuth p = mirrored(Azimuth{cpv, spv}, COS_2PI, SIN_2PI);
                        cpv = p.c;
                        spv = p.s;
                    } else {
                        spv = -spv;  // phi -> TWOPI - phi
                    }
                } else {
                    iz -= sgz;
                    fx = axis_pos(nx, fx, hx, tmx, t);
                    fy = axis_pos(ny, fy, hy, tmy, t);
                    fz = sgz > 0 ? hz : (Real)0;
                    nz = -nz;
                    sgz = -sgz;
                    tmz = t + tdz;
                }
            };
            // Russian roulette of a packet below the threshold; false: it dies
            auto roulette = [&](uint32_t draw) {
                const bool live_on = Uniform<Real>::from(draw) < inv_rm;
                atomicAdd(&s_tal[4], live_on ? (double)(w * (rm - (Real)1)) : -(double)w);
                if (live_on) w *= rm;
                return live_on;
            };
            // the same set-up for every direction
            auto setup = [&]() {
                axis_setup(nx, fx, hx, BIG, tdx, tmx, sgx);
                axis_setup(ny, fy, hy, BIG, tdy, tmy, sgy);
                axis_setup(nz, fz, hz, BIG, tdz, tmz, sgz);
            };
            if (alive && !go) {
                if constexpr (sizeof(Real) == 4 && MED != MED_RHOKAP) {
                    const U4 r = philox4x32_10_rk(ev++, plo, phi32, strm, a.rk);
                    if (face) {
                        surface(r.x);
                    } else {
                        interact();
                        cScat += 1;
                        const bool odd = scatter_f32(hgt[mid], Uniform<Real>::from(r.x), Uniform<Real>::from(r.y), hx, hy, hz,
                                                     t, fx, fy, fz, nx, ny, nz, sint, cpv, spv, tdx, tdy, tdz, tmx, tmy,
                                                     tmz, sgx, sgy, sgz);
                        t = (Real)0;
                        tau = M<Real>::neglog(Uniform<Real>::from(r.w));
                        if constexpr (DIST) tau *= inv_mut;
                        if (odd || !(w >= w_rare)) {
                            if (!(w > (Real)0)) {
                                cScat -= 1;
                                end();
                            } else if (!(nz == nz) || !(nx == nx) || !(ny == ny)) {
                                atomicOr(&s_err, (unsigned)DEVERR_NAN);
                                end();
                            } else {
                                setup();
                                if (a.roulette && w < wmin && !roulette(r.z)) end();
                            }
                        }
                    }
                } else if (face) {
                    surface(a.fresnel ? philox4x32_10_rk(ev++, plo, phi32, strm, a.rk).x : 0u);
                } else {
                    interact();
                    bool die = sizeof(Real) == 8 ? !ieee::gt_zero((double)w) : !(w > (Real)0);
                    if constexpr (SCAT64) {
                        if (!die) {
                            const U4 r = philox4x32_10_rk(ev++, plo, phi32, strm, a.rk);
                            cScat += 1;
                            fx = axis_pos(nx, fx, hx, tmx, t);
                            fy = axis_pos(ny, fy, hy, tmy, t);
                            fz = axis_pos(nz, fz, hz, tmz, t);
                            double cost = nz;
                            Azimuth p{cpv, spv};
                            if (stokes(lut[mid].g, lut[mid].g2, r.x, r.y, cost, sint, p)) {
                                cpv = p.c;
                                spv = p.s;
                                nx = sint * cpv;
                                ny = sint * spv;
                                nz = cost;
                            }
                            if (ieee::is_nan(nz) || ieee::is_nan(nx) || ieee::is_nan(ny)) {
                                atomicOr(&s_err, (unsigned)DEVERR_NAN);
                                die = true;
                            } else {
                                setup();
                                t = (Real)0;
                                die = a.roulette && less_pos(w, wmin) && !roulette(r.z);
                                tau = M<Real>::neglog(Uniform<Real>::from(r.w));
                            }
                        }
                    }
                    if (die) end();
                }
            }
        }
    }

    // ---- block reduction of the tallies ----
    const unsigned c1 = __reduce_add_sync(FULL, cScat);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cSteps += __shfl_xor_sync(FULL, cSteps, o);
    if constexpr (SPEC_REG) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) spec += __shfl_xor_sync(FULL, spec, o);
        if (lane == 0) atomicAdd(&s_tal[0], spec);
    }
    if (lane == 0) {
        atomicAdd(&s_cnt[1], (unsigned long long)c1);
        atomicAdd(&s_cnt[0], (unsigned long long)cSteps);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (!SPEC_REG && a.fresnel) {
            for (int m = 0; m < (MED == MED_MATERIAL ? a.nmat : 1); ++m) {
                const Real nt = MED == MED_RHOKAP ? K.rhokap_n : lut[MED == MED_MATERIAL ? m : mid_u].n;
                const Real r = (namb - nt) / (namb + nt);
                s_tal[0] += (double)s_entered[m] * (double)(r * r);
            }
        }
        atomicAdd(a.tally + T_SPECULAR, s_tal[0]);
        atomicAdd(a.tally + T_REFLECTED, s_tal[1]);
        atomicAdd(a.tally + T_TRANSMITTED, s_tal[2]);
        atomicAdd(a.tally + T_SIDE, s_tal[3]);
        atomicAdd(a.tally + T_ROULETTE_NET, s_tal[4]);
        atomicAdd(a.tally + T_STEPS, (double)s_cnt[0]);
        atomicAdd(a.tally + T_SCATTERS, (double)s_cnt[1]);
        if (s_err) atomicOr(a.err, s_err);
    }
}

// One warp per 8^3 brick: lane l takes the brick's x-rows l and l + 32 (of
// 64: y fastest, then z), the warp compares its smallest and largest id.
__global__ void brick_table_kernel(const uint8_t *mat, int nx, int ny, int nz, int bbx, int bby, int64_t nb,
                                   uint8_t *btab)
{
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t b = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < nb; b += nw) {
        const int bx = (int)(b % bbx);
        const int64_t rest = b / bbx;
        const int by = (int)(rest % bby), bz = (int)(rest / bby);
        int lo = 256, hi = -1;
        for (int row = lane; row < 64; row += 32) {
            const int y = by * 8 + (row & 7), z = bz * 8 + (row >> 3);
            if (y >= ny || z >= nz) continue;
            const uint8_t *p = mat + (int64_t)nx * (y + (int64_t)ny * z);
            for (int x = bx * 8; x < bx * 8 + 8 && x < nx; ++x) {
                const int v = p[x];
                lo = min(lo, v);
                hi = max(hi, v);
            }
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (lane == 0) btab[b] = (uint8_t)(lo == hi ? lo : 0xFF);
    }
}

// A lit cell of the normalisation (out of line: the compiler would otherwise
// issue the product and the sum, predicated off, for the dark cells too).
template <typename Out> __device__ __noinline__ double scale_lit(Out *out, double v, double f, double acc)
{
    *out = (Out)(v * f);
    return acc + v;
}

// out = in * f (normalisation of the tally), and with `sum` the total of
// `in` added to *sum: one FP64 atomic per block, so the grid is kept to a few
// thousand blocks.  Most cells of a tally are zero: for a finite f >= 0 their
// product is a zero too and they add nothing, so warps of zeros leave the
// narrow FP64 pipe alone (it bounded this pass; 512,000 cells, 2 % of them lit:
// 8.6 -> 6.9 us).
template <typename Out>
__global__ void scale_kernel(Out *out, double *in, double f, int64_t n, int zero_in, double *sum)
{
    const bool plain = ieee::is_finite(f) && ieee::ge_zero(f);
    double acc = 0.0;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        const double v = in[q];
        if (plain && ieee::bits(v) == 0) {
            out[q] = (Out)0;
            continue;
        }
        acc = scale_lit(out + q, v, f, acc);
        if (zero_in) in[q] = 0.0;
    }
    if (!sum) return;
    __shared__ double ws[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (__any_sync(0xffffffffu, ieee::bits(acc) != 0)) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    }
    if (lane == 0) ws[wid] = acc;
    __syncthreads();
    if (wid == 0) {
        acc = lane < (int)(blockDim.x >> 5) ? ws[lane] : 0.0;
        if (__any_sync(0xffffffffu, ieee::bits(acc) != 0)) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0) atomicAdd(sum, acc);
        }
    }
}

__global__ void flush_f32_kernel(double *acc, float *part, int nx, int ny, int bx0, int by0, int bz0, int bnx, int bny,
                                 int64_t n)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        const float v = part[q];
        if (v != 0.f) {
            const int64_t x = bx0 + q % bnx, y = by0 + (q / bnx) % bny, z = bz0 + q / ((int64_t)bnx * bny);
            acc[x + (int64_t)nx * (y + (int64_t)ny * z)] += (double)v;
            part[q] = 0.f;
        }
    }
}

__global__ void philox_selftest_kernel(const uint32_t *in, uint32_t *mine, uint32_t *ref, int64_t n)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t *p = in + 6 * q;
        const U4 r = philox4x32_10(p[0], p[1], p[2], p[3], p[4], p[5]);
        mine[4 * q + 0] = r.x;
        mine[4 * q + 1] = r.y;
        mine[4 * q + 2] = r.z;
        mine[4 * q + 3] = r.w;
        const uint4 c = make_uint4(p[0], p[1], p[2], p[3]);
        const uint2 k = make_uint2(p[4], p[5]);
        const uint4 o = curand_Philox4x32_10(c, k);
        ref[4 * q + 0] = o.x;
        ref[4 * q + 1] = o.y;
        ref[4 * q + 2] = o.z;
        ref[4 * q + 3] = o.w;
    }
}

int grid_for(int64_t n, int tpb)
{
    int64_t b = (n + tpb - 1) / tpb;
    if (b > 152 * 32) b = 152 * 32;
    return (int)(b > 0 ? b : 1);
}

template <typename Real, int MED, bool T32 = false>
cudaError_t launch_t(const TransportArgs &a, int sm_count, cudaStream_t s)
{
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, transport_kernel<Real, MED, T32>, TPB, 0);
    const int scat_min = a.scat_min > 0 ? a.scat_min : (sizeof(Real) == 8 ? SCAT_MIN64 : SCAT_MIN);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    const int per_warp = packets_per_warp(a.n, (int64_t)sm_count * (TPB / 32));
    const int64_t per_block = (int64_t)per_warp * (TPB / 32);
    const int64_t blocks = std::min((int64_t)sm_count * per_sm, (a.n + per_block - 1) / per_block);
    count_launch();
    transport_kernel<Real, MED, T32><<<(unsigned)blocks, TPB, 0, s>>>(a, scat_min, 0xffffffffu >> (32 - per_warp));
    return cudaGetLastError();
}

}  // namespace

// The per-launch constants, in the order of operations a thread used to
// evaluate them in FP64 (so the FP64 form's values are unchanged), and their
// FP32 roundings.
static void fill_consts(TransportArgs &a)
{
    TrConst<double> &d = a.cd;
    d.hx = 2.0 * a.xmax / a.nx;
    d.hy = 2.0 * a.ymax / a.ny;
    d.hz = 2.0 * a.zmax / a.nz;
    d.knx = 1.0 - a.nudge / (2.0 * a.xmax / a.nx);
    d.kny = 1.0 - a.nudge / (2.0 * a.ymax / a.ny);
    d.knz = 1.0 - a.nudge / (2.0 * a.zmax / a.nz);
    d.w2x = 2.0 * a.xmax;
    d.w2y = 2.0 * a.ymax;
    d.xmax = a.xmax;
    d.ymax = a.ymax;
    d.wmin = a.roulette_w;
    d.rm = a.roulette_m;
    d.inv_rm = 1.0 / a.roulette_m;
    d.namb = a.n_ambient;
    d.rhokap_n = a.rhokap_n;
    d.src_r = a.source_radius;
    d.cells_x = a.nx / d.w2x;
    d.cells_y = a.ny / d.w2y;
    const double r0 = (d.namb - d.rhokap_n) / (d.namb + d.rhokap_n);
    d.rhokap_spec = r0 * r0;
    for (int t = 0; t < MAX_MAT; ++t) {
        const OptMat &o = a.lut[t < a.nmat ? t : 0];
        const double mut = o.mua + o.mus, alb = mut > 0.0 ? o.mus / mut : 0.0, g2 = o.g * o.g;
        a.md[t] = MatR<double>{mut, o.mua, alb, o.g, g2, o.n};
        a.mf[t] = MatR<float>{(float)mut, (float)o.mua, (float)alb, (float)o.g, (float)g2, (float)o.n};
    }
    TrConst<float> &f = a.cf;
    f.hx = (float)d.hx, f.hy = (float)d.hy, f.hz = (float)d.hz;
    f.knx = (float)d.knx, f.kny = (float)d.kny, f.knz = (float)d.knz;
    f.w2x = (float)d.w2x, f.w2y = (float)d.w2y, f.xmax = (float)d.xmax, f.ymax = (float)d.ymax;
    f.wmin = (float)d.wmin, f.rm = (float)d.rm, f.inv_rm = (float)d.inv_rm;
    f.namb = (float)d.namb, f.rhokap_n = (float)d.rhokap_n, f.src_r = (float)d.src_r;
}

void fill_batch_inst(const TransportArgs &args, BatchTrInst &b)
{
    TransportArgs a = args;
    fill_consts(a);
    const TrConst<float> &f = a.cf;
    b.nx = a.nx, b.ny = a.ny, b.nz = a.nz;
    b.source = a.source, b.fresnel = a.fresnel, b.roulette = a.roulette;
    b.hx = f.hx, b.hy = f.hy, b.hz = f.hz, b.w2x = f.w2x, b.w2y = f.w2y, b.xmax = f.xmax, b.ymax = f.ymax;
    b.src_r = f.src_r, b.namb = f.namb, b.wmin = f.wmin, b.rm = f.rm, b.inv_rm = f.inv_rm;
    // the material's FP32 properties as the single pass's shared table holds them
    const OptMat &o = a.lut[a.uniform_id >= 0 && a.uniform_id < a.nmat ? a.uniform_id : 0];
    b.mut = (float)(o.mua + o.mus);
    b.mua = (float)o.mua;
    b.alb = (o.mua + o.mus) > 0.0 ? (float)(o.mus / (o.mua + o.mus)) : 0.f;
    b.g = (float)o.g;
    b.g2 = (float)(o.g * o.g);
    b.n = (float)o.n;
    b.inv_mut = 1.0f / b.mut;  // IEEE single division: the bits of the single pass's 1 / mut
    b.seed = a.seed;
    b.stream = a.stream;
    b.max_steps = a.max_steps > 0xfffffff0ll ? 0xfffffff0u : (uint32_t)a.max_steps;
    b.first = 0;
    b.count = a.n;
    b.jmean = a.jmean;
    b.tally = a.tally;
}

cudaError_t launch_transport(const TransportArgs &args, bool fp64, int sm_count, cudaStream_t s)
{
    if (args.n <= 0) return cudaSuccess;
    TransportArgs a = args;
    fill_consts(a);
    philox_round_keys(a.seed, a.rk);
    if (!a.work_zeroed) {
        cudaError_t e = cudaMemsetAsync(a.work, 0, sizeof(unsigned long long), s);
        if (e != cudaSuccess) return e;
    }
    if (fp64) {
        // the FP32 box tally is a config-mode form; on the FP64 transport it
        // serves its checks against the FP64 oracle on the same streams
        if (a.medium == MED_RHOKAP) {
            if (a.jmean32) return cudaErrorInvalidValue;
            return launch_t<double, MED_RHOKAP>(a, sm_count, s);
        }
        if (a.uniform_id >= 0)
            return a.jmean32 ? launch_t<double, MED_UNIFORM, true>(a, sm_count, s) : launch_t<double, MED_UNIFORM>(a, sm_count, s);
        return a.jmean32 ? launch_t<double, MED_MATERIAL, true>(a, sm_count, s) : launch_t<double, MED_MATERIAL>(a, sm_count, s);
    }
    if (a.medium == MED_RHOKAP) {
        if (a.jmean32) return cudaErrorInvalidValue;  // the FP32 tally is a config-mode form
        return launch_t<float, MED_RHOKAP>(a, sm_count, s);
    }
    // the tally's precision is a template parameter: no per-deposit branch
    if (a.uniform_id >= 0)
        return a.jmean32 ? launch_t<float, MED_UNIFORM, true>(a, sm_count, s) : launch_t<float, MED_UNIFORM>(a, sm_count, s);
    return a.jmean32 ? launch_t<float, MED_MATERIAL, true>(a, sm_count, s) : launch_t<float, MED_MATERIAL>(a, sm_count, s);
}

// at least four elements per thread, at most 152 x 16 blocks (atomics on *sum)
static int scale_grid(int64_t n)
{
    int64_t b = (n + 1023) / 1024;
    if (b > 152 * 16) b = 152 * 16;
    return (int)(b > 0 ? b : 1);
}

cudaError_t launch_scale_f64(double *out, double *in, double f, int64_t n, bool zero_in, cudaStream_t s, double *sum)
{
    if (n <= 0) return cudaSuccess;
    count_launch();
    scale_kernel<double><<<scale_grid(n), 256, 0, s>>>(out, in, f, n, zero_in ? 1 : 0, sum);
    return cudaGetLastError();
}

int64_t brick_table_size(int nx, int ny, int nz)
{
    return (int64_t)((nx + 7) / 8) * ((ny + 7) / 8) * ((nz + 7) / 8);
}

cudaError_t launch_brick_table(const uint8_t *mat, int nx, int ny, int nz, uint8_t *btab, cudaStream_t s)
{
    const int64_t nb = brick_table_size(nx, ny, nz);
    const int64_t blocks = std::min<int64_t>((nb + 7) / 8, 152 * 32);
    count_launch();
    brick_table_kernel<<<(unsigned)blocks, 256, 0, s>>>(mat, nx, ny, nz, (nx + 7) / 8, (ny + 7) / 8, nb, btab);
    return cudaGetLastError();
}

cudaError_t launch_flush_f32(double *acc, float *part, int nx, int ny, int bx0, int by0, int bz0, int bnx, int bny,
                             int bnz, cudaStream_t s)
{
    const int64_t n = (int64_t)bnx * bny * bnz;
    if (n <= 0) return cudaSuccess;
    count_launch();
    flush_f32_kernel<<<grid_for(n, 256), 256, 0, s>>>(acc, part, nx, ny, bx0, by0, bz0, bnx, bny, n);
    return cudaGetLastError();
}

cudaError_t launch_scale_to_f32(float *out, double *in, double f, int64_t n, bool zero_in, cudaStream_t s, double *sum)
{
    if (n <= 0) return cudaSuccess;
    count_launch();
    scale_kernel<float><<<scale_grid(n), 256, 0, s>>>(out, in, f, n, zero_in ? 1 : 0, sum);
    return cudaGetLastError();
}

namespace {
// Ceiling of the tally updates: `per_thread` fire-and-forget atomic adds per
// thread (red.global.add, the result unused, as the transport's deposits) at
// cells drawn from Philox inside the kernel, so no index stream is read; four
// cells per Philox block, mapped to [0, cells) by a 32 x 32 high product.
template <typename Real>
__global__ void __launch_bounds__(256) atomic_peak_kernel(Real *acc, uint32_t cells, int per_thread, uint32_t seed)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    for (int i = 0; i < per_thread; i += 4) {
        const U4 r = philox4x32_10((uint32_t)i, t, 0x7a11u, 0u, seed, 0x5eedu);
        atomicAdd(acc + __umulhi(r.x, cells), (Real)1);
        atomicAdd(acc + __umulhi(r.y, cells), (Real)1);
        atomicAdd(acc + __umulhi(r.z, cells), (Real)1);
        atomicAdd(acc + __umulhi(r.w, cells), (Real)1);
    }
}
}  // namespace

cudaError_t launch_atomic_peak(void *acc, bool fp32, uint32_t cells, int blocks, int per_thread, uint32_t seed,
                               cudaStream_t s)
{
    count_launch();
    if (fp32) atomic_peak_kernel<float><<<blocks, 256, 0, s>>>((float *)acc, cells, per_thread, seed);
    else atomic_peak_kernel<double><<<blocks, 256, 0, s>>>((double *)acc, cells, per_thread, seed);
    return cudaGetLastError();
}

cudaError_t launch_philox_selftest(const uint32_t *in, uint32_t *mine, uint32_t *ref, int64_t n, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    count_launch();
    philox_selftest_kernel<<<grid_for(n, 256), 256, 0, s>>>(in, mine, ref, n);
    return cudaGetLastError();
}

}  // namespace tam
