// heat64.cu -- the FP64 fused heat step on thermal classes.
//
// The physics of the per-voxel FP64 step (heat.cu, fused_kernel<double>):
// src/3dFD.f90:113-187 with the config-mode operator, Robin / Dirichlet ghost
// faces, the latent-heat clamp, Arrhenius damage and ablation, while k, rho
// and c are those of the voxels' material classes.
//
// What bounds it is GB300's FP64 pipe (about two lanes per clock per SM, and
// FP64 compares and conversions run on it too).  From per-voxel k, rho, c the
// step spends most of it on divisions: six face means k / (rho c) and the
// source's 1 / (rho c) per voxel, ~280 FP64 operations.  With classes, those
// are looked up (face coefficients per class pair, computed on the host with
// the same means), dt is folded into them, and screens are integer compares
// of the bit patterns: 13 FP64 operations per voxel in one class, 18 in
// several.  100^3 cube with a core in the damage window: 443 -> 47 us per step
// (FP64 pipe 76 % busy; a third of its operations are the window's).
#include <algorithm>

#include "heat_common.cuh"
#include "ieee_bits.h"

namespace tam {

namespace {

constexpr int TPB64 = 128;
constexpr int ROWS = 2;  // y-adjacent voxels of a thread
constexpr int ZMAX = 16;  // planes per block at most (the list holds every voxel of a block)

// The rare parts of a voxel's update, out of line: predicated off they would
// still be issued to the FP64 pipe for every voxel (the ghosts of the six faces
// alone were a third of its operations).
__device__ __noinline__ double robin_diff(const FusedArgs &a, const ClassLut64 &L, int f, int k, double tc)
{
    return -L.hdk[f * MAX_MAT + k] * (tc - a.dc[FC_BCTA + f]);
}
// Latent-heat clamp (src/3dFD.f90:169-175) of a voxel that was at boiling: its new temperature.
__device__ __noinline__ double boil64(const FusedArgs &a, const ClassLut64 &L, int k, int64_t q, double tc, double Tn,
                                      double PJdt, double dT)
{
    if (!(tc >= a.dc[FC_TBOIL])) return Tn;
    const double qv = a.dc[FC_LW] * L.rho[k] * a.dc[FC_VVOX];
    double *Q = (double *)a.Q;
    const double Qv = Q[q];
    if (!(Qv < qv)) return Tn;
    const double Ein = (PJdt + L.rho[k] * L.c[k] * dT) * a.dc[FC_VVOX];
    if (!(Ein > 0.0)) return Tn;
    const double qn = Qv + Ein;
    Q[q] = qn < qv ? qn : qv;
    return a.dc[FC_TBOIL];
}

// A thread marches ROWS y-adjacent columns through zchunk planes; the threads
// of a block take consecutive columns of the x-y plane (x fastest, wrapping from
// row pair to row pair), so every lane works at any nx.  Face differences are
// formed once where both voxels are the thread's: along z from plane to plane,
// along y inside the pair.  Voxels in the damage window (whose exponential and
// quotient are ~50 FP64 operations) or at ablation are listed and taken once the
// planes are done, a full warp at a time.
template <bool UNIFORM>
__global__ void __launch_bounds__(TPB64) cls64_step_kernel(const __grid_constant__ FusedArgs a,
                                                           const __grid_constant__ ClassLut64 L, const uint8_t *cls,
                                                           int zchunk)
{
    __shared__ double s_fa[UNIFORM ? 1 : MAX_MAT * MAX_MAT], s_src[UNIFORM ? 1 : MAX_MAT];
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const double Pdt = step_pdt<double>(a), t_new = step_tnew(a);
    const bool src_on = Pdt != 0.0;
    if (!UNIFORM) {
        for (int t = threadIdx.x; t < MAX_MAT * MAX_MAT; t += TPB64) s_fa[t] = L.fa[t];
        if (threadIdx.x < MAX_MAT) s_src[threadIdx.x] = Pdt * L.irc[threadIdx.x];
    }
    __shared__ unsigned short s_list[TPB64 * ROWS * ZMAX];
    __shared__ int s_cnt;
    if (threadIdx.x == 0) s_cnt = 0;
    __syncthreads();
    const int64_t col0 = blockIdx.x * (int64_t)TPB64, col = col0 + threadIdx.x;
    const int x = (int)(col % nx), y0 = (int)(col / nx) * ROWS;
    const int z0 = blockIdx.y * zchunk, z1 = min(nz, z0 + zchunk);
    const int64_t sy = nx, sz = (int64_t)nx * ny, ni = sz * nz;
    const double *T = (const double *)a.T_in;
    double *To = (double *)a.T_out;
    const double *J = (const double *)a.J;
    const double czd = a.dc[FC_DT] * a.dc[FC_CZ], cyd = a.dc[FC_DT] * a.dc[FC_CY], cxd = a.dc[FC_DT] * a.dc[FC_CX];
    const int uc = L.uniform >= 0 ? L.uniform : 0;
    const double au = L.fa[uc * MAX_MAT + uc];
    const double Cx = cxd * au, Cy = cyd * au, Cz = czd * au, Ku = Pdt * L.irc[uc];
    // screens on the bit patterns, which order like the values they are
    // compared with: at or above them lie the listed temperatures and the
    // negative and NaN ones.  That holds from +0 up: a screen below (T_lo = 0 K,
    // 0.01 K below which it lies) or NaN becomes +0, which takes every voxel, and
    // the exact tests decide
    auto word = [](double s) -> uint64_t { return ieee::gt_zero(s) ? ieee::bits(s) : 0; };
    const uint64_t screen = word(a.dc[FC_SCREEN]);
    const uint64_t boil = a.boil ? word(a.dc[FC_TBOIL]) : ~0ull;
    auto klass = [&](int64_t q) -> int { return UNIFORM ? uc : (int)__ldg(cls + q); };
    // difference towards the neighbour n across face f, or the face's ghost
    // (Dirichlet: the face's temperature; Robin: -h d / k (T - T_amb)); in a
    // grid of several classes times the face's diffusivity
    auto flux = [&](bool inside, int f, int64_t n, double tc, int k) -> double {
        double d = (inside ? __ldg(T + n) : a.dc[FC_BCT + f]) - tc;
        if (!inside && a.bc_type[f] == BC_ROBIN) d = robin_diff(a, L, f, k, tc);
        return UNIFORM ? d : s_fa[k * MAX_MAT + (inside ? klass(n) : k)] * d;
    };
    double tc[ROWS], fzm[ROWS];
    int kc[ROWS];
    bool in[ROWS];
    int64_t v = x + sy * y0 + sz * z0;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        in[r] = y0 + r < ny;  // (a column past the last has no row)
        tc[r] = in[r] ? T[v + r * sy] : 0.0;
        kc[r] = in[r] ? klass(v + r * sy) : 0;
        fzm[r] = in[r] ? flux(z0 > 0, 4, v + r * sy - sz, tc[r], kc[r]) : 0.0;
    }
    unsigned errbits = 0;
    for (int z = z0; z < z1; ++z, v += sz) {
        const bool up = z + 1 < nz;
        double tp[ROWS], fzp[ROWS], Jv[ROWS];
        int kp[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const int64_t q = v + r * sy;
            tp[r] = in[r] && up ? __ldg(T + q + sz) : 0.0;
            kp[r] = in[r] && up ? klass(q + sz) : kc[r];
            Jv[r] = in[r] && src_on ? J[q] : 0.0;
        }
        double fy = in[0] ? flux(y0 > 0, 2, v - sy, tc[0], kc[0]) : 0.0;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            if (!in[r]) continue;
            const int64_t q = v + r * sy;
            const double fym = fy;
            double fyp;
            if (r + 1 < ROWS && in[r + 1 < ROWS ? r + 1 : r]) {
                constexpr int R1 = ROWS - 1;
                const int rn = r < R1 ? r + 1 : R1;
                const double d = tc[rn] - tc[r];
                fyp = UNIFORM ? d : s_fa[kc[r] * MAX_MAT + kc[rn]] * d;
                fy = -fyp;
            } else {
                fyp = flux(y0 + r < ny - 1, 3, q + sy, tc[r], kc[r]);
            }
            const double fxm = flux(x > 0, 0, q - 1, tc[r], kc[r]), fxp = flux(x < nx - 1, 1, q + 1, tc[r], kc[r]);
            if (up) {
                const double d = tp[r] - tc[r];
                fzp[r] = UNIFORM ? d : s_fa[kc[r] * MAX_MAT + kp[r]] * d;
            } else {
                fzp[r] = flux(false, 5, 0, tc[r], kc[r]);
            }
            const double ax = UNIFORM ? Cx : cxd, ay = UNIFORM ? Cy : cyd, az = UNIFORM ? Cz : czd;
            const double dT = fma(az, fzm[r] + fzp[r], fma(ay, fym + fyp, ax * (fxm + fxp)));
            double Tn = tc[r] + (src_on ? fma(UNIFORM ? Ku : s_src[kc[r]], Jv[r], dT) : dT);
            if (ieee::bits(tc[r]) >= boil) Tn = boil64(a, L, kc[r], q, tc[r], Tn, Pdt * Jv[r], dT);
            To[q] = Tn;
            if (ieee::bits(Tn) >= screen) {
                if (ieee::is_nan(Tn)) errbits |= DEVERR_NAN;
                else if (ieee::lt_zero(Tn)) errbits |= DEVERR_NEG_T;
                else s_list[atomicAdd(&s_cnt, 1)] = (unsigned short)(((z - z0) * ROWS + r) * TPB64 + threadIdx.x);
            }
            // the next plane's z- difference
            fzm[r] = -fzp[r];
            tc[r] = tp[r];
            kc[r] = kp[r];
        }
    }
    if (errbits) atomicOr(a.err, errbits);
    __syncthreads();
    for (int n = threadIdx.x; n < s_cnt; n += TPB64) {
        const int l = s_list[n], r = l / TPB64;
        const int64_t c = col0 + l % TPB64;
        const int64_t q = c % nx + sy * ((c / nx) * ROWS + r % ROWS) + sz * (z0 + r / ROWS);
        rare_update<double>(a, q, ni, To[q], t_new);
    }
}

// The class of every voxel from its k, rho, c: the first class that has them.
__global__ void cls_from_props_kernel(const double *k, const double *rho, const double *c,
                                      const __grid_constant__ ClassLut64 L, int ncls, uint8_t *cls, int64_t n)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t kb = ieee::bits(k[q]), rb = ieee::bits(rho[q]), cb = ieee::bits(c[q]);
        int m = 0;
        for (int i = ncls - 1; i >= 0; --i)
            if (ieee::bits(L.k[i]) == kb && ieee::bits(L.rho[i]) == rb && ieee::bits(L.c[i]) == cb) m = i;
        cls[q] = (uint8_t)m;
    }
}

}  // namespace

cudaError_t launch_cls_from_props(const double *k, const double *rho, const double *c, const ClassLut64 &L, int ncls,
                                  uint8_t *cls, int64_t n, cudaStream_t s)
{
    count_launch();
    cls_from_props_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, 152 * 16), 256, 0, s>>>(k, rho, c, L, ncls, cls, n);
    return cudaGetLastError();
}

cudaError_t launch_cls64_step(const FusedArgs &a0, const ClassLut64 &L0, const uint8_t *cls, cudaStream_t s)
{
    FusedArgs a = a0;
    fill_fused_consts(a);
    ClassLut64 L = L0;
    for (int f = 0; f < 6; ++f)
        for (int k = 0; k < MAX_MAT; ++k) L.hdk[f * MAX_MAT + k] = a.dc[FC_BCHD + f] / L.k[k];
    const int64_t bx = ((int64_t)a.nx * ((a.ny + ROWS - 1) / ROWS) + TPB64 - 1) / TPB64;
    // columns of 2 to ZMAX planes, two waves of the six blocks that an SM holds:
    // blocks with many listed voxels then even out (100^3: 2 / 3 / 4 / 7 / 16
    // planes -> 46.6 / 46.3 / 56.6 / 53.1 / 78.9 us; 60 x 50 x 55: 2 / 4 / 8
    // planes -> 16.5 / 20.1 / 33.8 us)
    const int chunks = (int)std::max<int64_t>(1, 152 * 6 * 2 / bx);
    const int zchunk = a.zchunk > 0 ? std::min(ZMAX, a.zchunk) : std::min(ZMAX, std::max(2, (a.nz + chunks - 1) / chunks));
    const dim3 grid((unsigned)bx, (a.nz + zchunk - 1) / zchunk);
    count_launch();
    if (L.uniform >= 0) cls64_step_kernel<true><<<grid, TPB64, 0, s>>>(a, L, cls, zchunk);
    else cls64_step_kernel<false><<<grid, TPB64, 0, s>>>(a, L, cls, zchunk);
    return cudaGetLastError();
}

}  // namespace tam
