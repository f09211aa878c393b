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
// of the bit patterns: 14 FP64 operations per voxel in one class, 20 in
// several.  100^3 cube: 443 -> 45 us per step.
#include <algorithm>

#include "heat_common.cuh"
#include "ieee_bits.h"

namespace tam {

namespace {

constexpr int CX = 32, CY = 8;  // voxels of a block's column tile

template <bool UNIFORM>
__global__ void __launch_bounds__(CX *CY) cls64_step_kernel(const __grid_constant__ FusedArgs a,
                                                            const __grid_constant__ ClassLut64 L, const uint8_t *cls,
                                                            int zchunk)
{
    __shared__ double s_fa[UNIFORM ? 1 : MAX_MAT * MAX_MAT], s_src[UNIFORM ? 1 : MAX_MAT];
    const int x = blockIdx.x * CX + threadIdx.x, y = blockIdx.y * CY + threadIdx.y;
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const double Pdt = step_pdt<double>(a), t_new = step_tnew(a);
    const bool src_on = Pdt != 0.0;
    if (!UNIFORM) {
        const int tid = threadIdx.y * CX + threadIdx.x;
        s_fa[tid] = L.fa[tid];
        if (tid < MAX_MAT) s_src[tid] = Pdt * L.irc[tid];
        __syncthreads();
    }
    if (x >= nx || y >= ny) return;
    const int z0 = blockIdx.z * zchunk, z1 = min(nz, z0 + zchunk);
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
    // negative and NaN ones
    const uint64_t screen = ieee::bits(a.dc[FC_SCREEN]);
    const uint64_t boil = a.boil ? ieee::bits(a.dc[FC_TBOIL]) : ~0ull;
    int64_t v = x + sy * y + sz * z0;
    auto klass = [&](int64_t q) -> int { return UNIFORM ? uc : (int)__ldg(cls + q); };
    // neighbour difference across face f: towards the neighbour n, or the ghost's
    // (Dirichlet: the face's temperature; Robin: -h d / k (T - T_amb))
    auto face = [&](bool inside, int f, int64_t n, double tc, int k) -> double {
        double t = a.dc[FC_BCT + f];
        if (inside) t = __ldg(T + n);
        else if (a.bc_type[f] == BC_ROBIN) return -L.hdk[f * MAX_MAT + k] * (tc - a.dc[FC_BCTA + f]);
        return t - tc;
    };
    double tc = T[v], tm = z0 > 0 ? T[v - sz] : 0.0;
    int kc = klass(v), km = z0 > 0 ? klass(v - sz) : kc;
    unsigned errbits = 0;
    for (int z = z0; z < z1; ++z, v += sz) {
        const bool up = z + 1 < nz;
        const double tp = up ? __ldg(T + v + sz) : 0.0;
        const int kp = up ? klass(v + sz) : kc;
        const double Jv = src_on ? J[v] : 0.0;
        const double dxm = face(x > 0, 0, v - 1, tc, kc), dxp = face(x < nx - 1, 1, v + 1, tc, kc);
        const double dym = face(y > 0, 2, v - sy, tc, kc), dyp = face(y < ny - 1, 3, v + sy, tc, kc);
        const double dzm = z > 0 ? tm - tc : face(false, 4, 0, tc, kc);
        const double dzp = up ? tp - tc : face(false, 5, 0, tc, kc);
        double dT;
        if (UNIFORM) {
            dT = fma(Cz, dzm + dzp, fma(Cy, dym + dyp, Cx * (dxm + dxp)));
        } else {
            const double *f = s_fa + kc * MAX_MAT;
            const double sx = f[x > 0 ? klass(v - 1) : kc] * dxm + f[x < nx - 1 ? klass(v + 1) : kc] * dxp;
            const double sy_ = f[y > 0 ? klass(v - sy) : kc] * dym + f[y < ny - 1 ? klass(v + sy) : kc] * dyp;
            const double sz_ = f[z > 0 ? km : kc] * dzm + f[kp] * dzp;
            dT = fma(czd, sz_, fma(cyd, sy_, cxd * sx));
        }
        double Tn = tc + (src_on ? fma(UNIFORM ? Ku : s_src[kc], Jv, dT) : dT);
        if (ieee::bits(tc) >= boil && tc >= a.dc[FC_TBOIL]) {
            // latent-heat clamp (src/3dFD.f90:169-175)
            const double qv = a.dc[FC_LW] * L.rho[kc] * a.dc[FC_VVOX];
            double *Q = (double *)a.Q;
            const double Qv = Q[v];
            if (Qv < qv) {
                const double Ein = (Pdt * Jv + L.rho[kc] * L.c[kc] * dT) * a.dc[FC_VVOX];
                if (Ein > 0.0) {
                    const double qn = Qv + Ein;
                    Q[v] = qn < qv ? qn : qv;
                    Tn = a.dc[FC_TBOIL];
                }
            }
        }
        To[v] = Tn;
        if (ieee::bits(Tn) >= screen) {
            if (!(Tn == Tn)) errbits |= DEVERR_NAN;
            else if (Tn < 0.0) errbits |= DEVERR_NEG_T;
            else if (Tn >= a.dc[FC_SCREEN]) rare_update<double>(a, v, ni, Tn, t_new);
        }
        tm = tc;
        tc = tp;
        km = kc;
        kc = kp;
    }
    if (errbits) atomicOr(a.err, errbits);
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
    const int bx = (a.nx + CX - 1) / CX, by = (a.ny + CY - 1) / CY;
    // columns of up to 16 planes, short enough for eight blocks per SM where the grid allows
    const int chunks = std::max(1, std::min(a.nz, (152 * 8 + bx * by - 1) / (bx * by)));
    const int zchunk = a.zchunk > 0 ? a.zchunk : std::min(16, (a.nz + chunks - 1) / chunks);
    const dim3 grid(bx, by, (a.nz + zchunk - 1) / zchunk);
    count_launch();
    if (L.uniform >= 0) cls64_step_kernel<true><<<grid, dim3(CX, CY), 0, s>>>(a, L, cls, zchunk);
    else cls64_step_kernel<false><<<grid, dim3(CX, CY), 0, s>>>(a, L, cls, zchunk);
    return cudaGetLastError();
}

}  // namespace tam
