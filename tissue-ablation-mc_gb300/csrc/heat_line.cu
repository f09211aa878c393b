// heat_line.cu -- the FP32 + Kahan fused heat step for rows of any width.
//
// The quad form (heat_quad.cu) asks for rows of whole quads; here a block takes 256
// consecutive voxels of a plane, wrapping from row to row, two per thread and 128
// apart, so that every load is a run of words, and marches them through a few
// planes: the planes' values in registers (three buffers in rotation), x
// neighbours from the neighbouring lanes, the two voxels' arithmetic in two-wide
// FP32 instructions, latency hidden by occupancy (8 blocks per SM at 64 registers;
// 12 at 40: 7 to 20 % slower).  Launches and rare work as there, replayed from graphs.
//
// The form before it staged 32 x 8 tiles by 4-byte asynchronous copies, with a barrier
// per plane, in blocks of 8 planes, and was launched step by step.  Same arithmetic,
// operation for operation.
//
// What bounds it: instruction issue (60 % of the slots; 300 instructions per plane
// and warp of 64 voxels, 18 of them loads).  The boundary sum, which an x face
// puts into 4 of 10 warps of a 151-wide row, for the pair at once instead of per
// voxel: 5 % slower; plane pointers and 32-bit offsets: 4 % slower; scalar
// arithmetic: 5 % slower.  Per step, staged form before -> now: 151 x 150 x 149
// 53.8 -> 21.6 us, 101 x 99 x 103 30.4 -> 9.3, 33 x 34 x 35 26.6 -> 6.2; layers
// 97 x 95 x 60 29.5 -> 8.6, vessels 151 x 140 x 130 49.0 -> 24.7.
#include <algorithm>
#include <cstring>

#include "f32x2.cuh"
#include "heat_common.cuh"

namespace tam {

namespace {

constexpr int LTPB = 128;  // threads per block, two voxels each
constexpr int LV = 2 * LTPB;
constexpr int LZMAX = 8;   // planes per block at most (the list holds every voxel of a block)

// Boundary faces: the coefficient k / (rho c) of the ghost face times the axis's,
// and the Robin faces' h d / k, per face and class.
struct LineFaces {
    float g[6 * MAX_MAT], h[6 * MAX_MAT];
};
// Quotients by the row width without a division (Granlund and Montgomery, 1994).
struct LineDiv {
    unsigned m, s1, s2;
    explicit LineDiv(unsigned d)
    {
        unsigned l = 0;
        while (l < 32 && (1ull << l) < d) ++l;
        m = (unsigned)(((1ull << 32) * ((1ull << l) - d)) / d + 1);
        s1 = std::min(l, 1u);
        s2 = l ? l - 1 : 0;
    }
    __device__ __forceinline__ unsigned quot(unsigned n) const
    {
        const unsigned t = __umulhi(m, n);
        return (t + ((n - t) >> s1)) >> s2;
    }
};
struct LineClasses {
    const uint8_t *cls;  // rows of cpitch bytes
    const float *tab;    // the face table: as parameters, each lane's own entry would be read in turn
    int cpitch;
};

// Latent-heat clamp of a voxel at or above the boiling temperature
// (src/3dFD.f90:169-175): true when the voxel absorbed the step's energy.
__device__ __noinline__ bool line_boil(const FusedArgs &a, float rr, float c, int v, float sPJ, float dT)
{
    float *Q = (float *)a.Q;
    const float rc = rr * c, qv = a.fc[FC_LW] * rr * a.fc[FC_VVOX], Qv = Q[v];
    if (!(Qv < qv)) return false;
    const float Ein = (sPJ + rc * dT) * a.fc[FC_VVOX];
    if (!(Ein > 0.f)) return false;
    const float qn = Qv + Ein;
    Q[v] = qn < qv ? qn : qv;
    return true;
}

template <bool HET>
__global__ void __launch_bounds__(LTPB, 8)
    line_step_kernel(const __grid_constant__ FusedArgs a, const __grid_constant__ ClassLut L,
                     const __grid_constant__ LineClasses C, const __grid_constant__ LineFaces F, LineDiv D, int zchunk, float rare_thr)
{
    __shared__ unsigned short s_list[LV * LZMAX];
    __shared__ int s_cnt;
    __shared__ float s_fa[HET ? MAX_MAT * MAX_MAT : 1];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (threadIdx.x == 0) s_cnt = 0;
    const float Pdt = step_pdt<float>(a);
    const bool src = Pdt != 0.f;  // without a source J is not read
    if (HET)
        for (int t = threadIdx.x; t < MAX_MAT * MAX_MAT; t += LTPB) s_fa[t] = __ldg(C.tab + t);
    __syncthreads();
    const int nx = a.nx, ny = a.ny, nz = a.nz, pl = nx * ny;
    const unsigned q0 = blockIdx.x * LV;
    // runs of planes from the top face down: the beam enters there, so the
    // blocks with the longest lists start first
    const int z0 = (int)(gridDim.y - 1 - blockIdx.y) * zchunk, z1 = min(nz, z0 + zchunk);
    const float *T = (const float *)a.T_in, *E = a.Tc_in, *J = (const float *)a.J;
    float *To = (float *)a.T_out, *Eo = a.Tc_out;
    const int uc = L.uniform >= 0 ? L.uniform : 0;
    const unsigned thr = __float_as_uint(rare_thr);
    const int lane = threadIdx.x & 31;
    bool act[2], ed[2], odd[2];
    int v[2], oyl[2], oyh[2];
    unsigned gm[2];  // boundary faces of x and y
    int64_t cv[2];
    const int oe = lane == 0 ? -1 : 1;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const unsigned id = q0 + h * LTPB + threadIdx.x;
        const int y = (int)D.quot(id), x = (int)(id - (unsigned)y * (unsigned)nx);
        act[h] = y < ny;
        odd[h] = x & 1;
        v[h] = (act[h] ? (int)id : 0) + pl * z0;
        oyl[h] = act[h] && y > 0 ? -nx : 0;
        oyh[h] = act[h] && y < ny - 1 ? nx : 0;
        ed[h] = act[h] && ((lane == 0 && x > 0) || (lane == 31 && x < nx - 1));
        gm[h] = !act[h] ? 0u
                        : (unsigned)(x == 0) | (unsigned)(x == nx - 1) << 1 | (unsigned)(y == 0) << 2 | (unsigned)(y == ny - 1) << 3;
        cv[h] = act[h] ? x + C.cpitch * ((int64_t)ny * z0 + y) : 0;
    }
    const int64_t cpl = (int64_t)C.cpitch * ny;
    const float au = L.fa[uc * MAX_MAT + uc], iu = L.irc[uc];
    const float cx = a.fc[FC_CX], cy = a.fc[FC_CY], cz = a.fc[FC_CZ], dt = a.fc[FC_DT];
    int kp[2] = {uc, uc}, kc[2] = {uc, uc}, kn[2] = {uc, uc};
    if (HET)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            kp[h] = z0 > 0 ? __ldg(C.cls + cv[h] - (act[h] ? cpl : 0)) & (MAX_MAT - 1) : 0;
            kc[h] = __ldg(C.cls + cv[h]) & (MAX_MAT - 1);
        }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float2 A[3], B[3];  // T and the Kahan term of three planes, in rotation
    {
        const int o = z0 > 0 ? pl : 0;
        A[0] = make_float2(T[v[0] - o], T[v[1] - o]), B[0] = make_float2(E[v[0] - o], E[v[1] - o]);
        A[1] = make_float2(T[v[0]], T[v[1]]), B[1] = make_float2(E[v[0]], E[v[1]]);
    }
    auto step = [&](int z, const float2 &tp, const float2 &ep, const float2 &tc, const float2 &ec, float2 &tn, float2 &en) {
        // the next plane, and this plane's source and neighbours
        const int on = z + 1 < nz ? pl : 0;
        tn = make_float2(T[v[0] + on], T[v[1] + on]);
        en = make_float2(E[v[0] + on], E[v[1] + on]);
        float2 j = make_float2(0.f, 0.f);
        if (src) j = make_float2(J[v[0]], J[v[1]]);
        const float2 yl = make_float2(T[v[0] + oyl[0]], T[v[1] + oyl[1]]), yel = make_float2(E[v[0] + oyl[0]], E[v[1] + oyl[1]]);
        const float2 yh = make_float2(T[v[0] + oyh[0]], T[v[1] + oyh[1]]), yeh = make_float2(E[v[0] + oyh[0]], E[v[1] + oyh[1]]);
        float2 te = make_float2(0.f, 0.f), ee = te;
        if (ed[0]) te.x = T[v[0] + oe], ee.x = E[v[0] + oe];
        if (ed[1]) te.y = T[v[1] + oe], ee.y = E[v[1] + oe];
        int kxl[2], kxr[2], kyl[2], kyh[2];
        if (HET) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint8_t *c = C.cls + cv[h];
                kn[h] = z + 1 < nz ? __ldg(c + (act[h] ? cpl : 0)) & (MAX_MAT - 1) : 0;
                kyl[h] = __ldg(c + (oyl[h] ? -C.cpitch : 0)) & (MAX_MAT - 1);
                kyh[h] = __ldg(c + (oyh[h] ? C.cpitch : 0)) & (MAX_MAT - 1);
                const int ke = ed[h] ? __ldg(c + oe) & (MAX_MAT - 1) : 0;
                kxl[h] = __shfl_up_sync(0xffffffffu, kc[h], 1);
                kxr[h] = __shfl_down_sync(0xffffffffu, kc[h], 1);
                if (lane == 0) kxl[h] = ke;
                if (lane == 31) kxr[h] = ke;
            }
        }
        float2 xl, xr, xel, xer;
        xl.x = __shfl_up_sync(0xffffffffu, tc.x, 1), xl.y = __shfl_up_sync(0xffffffffu, tc.y, 1);
        xr.x = __shfl_down_sync(0xffffffffu, tc.x, 1), xr.y = __shfl_down_sync(0xffffffffu, tc.y, 1);
        xel.x = __shfl_up_sync(0xffffffffu, ec.x, 1), xel.y = __shfl_up_sync(0xffffffffu, ec.y, 1);
        xer.x = __shfl_down_sync(0xffffffffu, ec.x, 1), xer.y = __shfl_down_sync(0xffffffffu, ec.y, 1);
        if (lane == 0) xl = te, xel = ee;
        if (lane == 31) xr = te, xer = ee;
        const float2 tzm = sub2(sub2(tp, tc), sub2(ep, ec)), tzp = sub2(sub2(tn, tc), sub2(en, ec));
        const float2 tym = sub2(sub2(yl, tc), sub2(yel, ec)), typ = sub2(sub2(yh, tc), sub2(yeh, ec));
        const float2 txm = sub2(sub2(xl, tc), sub2(xel, ec)), txp = sub2(sub2(xr, tc), sub2(xer, ec));
        float2 azm = dup(au), azp = azm, aym = azm, ayp = azm, axm = azm, axp = azm, irc = dup(iu);
        if (HET) {
            const float *f0 = s_fa + kc[0] * MAX_MAT, *f1 = s_fa + kc[1] * MAX_MAT;
            azm = make_float2(f0[kp[0]], f1[kp[1]]), azp = make_float2(f0[kn[0]], f1[kn[1]]);
            aym = make_float2(f0[kyl[0]], f1[kyl[1]]), ayp = make_float2(f0[kyh[0]], f1[kyh[1]]);
            axm = make_float2(f0[kxl[0]], f1[kxl[1]]), axp = make_float2(f0[kxr[0]], f1[kxr[1]]);
            irc = make_float2(L.irc[kc[0]], L.irc[kc[1]]);
        }
        float2 lap = fma2(dup(cx), fma2(axm, txm, mul2(axp, txp)),
                          fma2(dup(cy), fma2(aym, tym, mul2(ayp, typ)), mul2(dup(cz), fma2(azm, tzm, mul2(azp, tzp)))));
        const unsigned gz = (unsigned)(z == 0) << 4 | (unsigned)(z == nz - 1) << 5;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const unsigned g = gm[h] | gz;
            if (!g) continue;
            // a face on the boundary: the inner faces' sum, each product rounded, and
            // the ghosts, which carry the voxel's own properties
            auto s = [&](const float2 &p) { return h ? p.y : p.x; };
            auto part = [&](unsigned lo, const float2 &am, const float2 &tm, const float2 &ap, const float2 &tp2) {
                return __fadd_rn(g & lo ? 0.f : __fmul_rn(s(am), s(tm)), g & lo << 1 ? 0.f : __fmul_rn(s(ap), s(tp2)));
            };
            // (at odd x, never the low face, the first product's rounding falls away)
            const float X = odd[h] ? __fmaf_rn(s(axm), s(txm), g & 2u ? 0.f : __fmul_rn(s(axp), s(txp))) : part(1u, axm, txm, axp, txp);
            const float l = __fmaf_rn(cx, X, __fmaf_rn(cz, part(16u, azm, tzm, azp, tzp), __fmul_rn(cy, part(4u, aym, tym, ayp, typ))));
            const float t = s(tc), e = s(ec);
            const int k = HET ? kc[h] : uc;
            float gs = 0.f;
            auto ghost = [&](int f) {
                const float d = a.bc_type[f] == BC_ROBIN ? __fmul_rn(-F.h[f * MAX_MAT + k], __fsub_rn(__fsub_rn(t, a.fc[FC_BCTA + f]), e))
                                                         : __fadd_rn(__fsub_rn(a.fc[FC_BCT + f], t), e);
                gs = __fadd_rn(gs, __fmul_rn(F.g[f * MAX_MAT + k], d));
            };
            if (g & 1u) ghost(0);
            if (g & 2u) ghost(1);
            if (g & 0x3cu) {
                if (g & 4u) ghost(2);
                if (g & 8u) ghost(3);
                if (g & 16u) ghost(4);
                if (g & 32u) ghost(5);
            }
            (h ? lap.y : lap.x) = __fadd_rn(l, gs);
        }
        const float2 sPJ = mul2(dup(Pdt), j);
        const float2 yk = sub2(fma2(dup(dt), lap, mul2(sPJ, irc)), ec);
        float2 t = add2(tc, yk), e = sub2(sub2(t, tc), yk);
        // rare: an old or new temperature at the screen, or a new one negative or
        // NaN, which as unsigned words are the large ones
        auto u = [](float f) { return __float_as_uint(f); };
        if (max(max(u(tc.x), u(tc.y)), max(u(t.x), u(t.y))) >= thr) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float c = h ? tc.y : tc.x;
                if (!act[h] || max(u(c), u(h ? t.y : t.x)) < thr) continue;
                const int k = HET ? kc[h] : uc;
                if (a.boil && c >= a.fc[FC_TBOIL] &&
                    line_boil(a, L.rho[k], L.c[k], v[h], h ? sPJ.y : sPJ.x, __fmul_rn(dt, h ? lap.y : lap.x))) {
                    (h ? t.y : t.x) = a.fc[FC_TBOIL];
                    (h ? e.y : e.x) = a.fc[FC_TBOIL_E];
                }
                s_list[atomicAdd(&s_cnt, 1)] = (unsigned short)((z - z0) * LV + h * LTPB + (int)threadIdx.x);
            }
        }
        if (act[0]) To[v[0]] = t.x, Eo[v[0]] = e.x;
        if (act[1]) To[v[1]] = t.y, Eo[v[1]] = e.y;
        v[0] += pl, v[1] += pl;
        if (HET) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                cv[h] += act[h] ? cpl : 0;
                kp[h] = kc[h];
                kc[h] = kn[h];
            }
        }
    };
    for (int z = z0;;) {
        step(z, A[0], B[0], A[1], B[1], A[2], B[2]);
        if (++z == z1) break;
        step(z, A[1], B[1], A[2], B[2], A[0], B[0]);
        if (++z == z1) break;
        step(z, A[2], B[2], A[0], B[0], A[1], B[1]);
        if (++z == z1) break;
    }
    __syncthreads();
    // damage, ablation and the error word of the listed voxels (this block's own
    // stores come first)
    const int cnt = s_cnt;
    const double t_new = step_tnew(a);
    unsigned errbits = 0;
    for (int n = threadIdx.x; n < cnt; n += LTPB) {
        const int l = s_list[n], w = (int)q0 + l % LV + pl * (z0 + l / LV);
        const float t = To[w], e = Eo[w], Ts = t - e;
        const double o = a.omega[w];
        errbits |= (Ts == Ts) ? (Ts < 0.f ? (unsigned)DEVERR_NEG_T : 0u) : (unsigned)DEVERR_NAN;
        if (Ts >= a.fc[FC_SCREEN]) rare_update_f32(a, w, (int64_t)pl * nz, t, e, t_new, true, o);
    }
    if (errbits) atomicOr(a.err, errbits);
}

}  // namespace

bool line_step_supported(int nx, int ny, int nz)
{
    return nz <= LZMAX * 65535 && (int64_t)nx * ny * nz < ((int64_t)1 << 31) - 512;
}

cudaError_t launch_line_table(const ClassLut &L, float *tab, cudaStream_t s)
{
    return cudaMemcpyAsync(tab, L.fa, LINE_TABLE * sizeof(float), cudaMemcpyHostToDevice, s);
}

cudaError_t launch_line_step(const FusedArgs &a0, const ClassLut &L, const uint8_t *cls, int cpitch, const float *tab,
                             cudaStream_t s)
{
    FusedArgs a = a0;
    fill_fused_consts(a);
    const float rare_thr = rare_screen(a);
    LineFaces F{};
    for (int f = 0; f < 6; ++f)
        for (int c = 0; c < MAX_MAT; ++c) {
            const float rc = L.rho[c] * L.c[c], q = L.k[c] / rc;
            F.g[f * MAX_MAT + c] = a.fc[f < 2 ? FC_CX : (f < 4 ? FC_CY : FC_CZ)] * q;
            F.h[f * MAX_MAT + c] = a.fc[FC_BCHD + f] / L.k[c];
        }
    const int bx = (int)(((int64_t)a.nx * a.ny + LV - 1) / LV);
    // planes per block: as many as leave 5000 blocks (four waves), at most 5, as in
    // the quad form (151 x 150 x 149 with 2500 / 4000 / 5000: 21.8 / 21.6 / 21.9 us;
    // 101 x 99 x 103: 9.9 / 9.9 / 9.6)
    int zc = a.zchunk > 0 ? std::min(LZMAX, a.zchunk) : (int)std::min<int64_t>(5, ((int64_t)bx * a.nz + 4999) / 5000);
    zc = std::max(zc, (a.nz + 65534) / 65535);
    const LineClasses C{cls, tab, cpitch};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)bx, (unsigned)((a.nz + zc - 1) / zc));
    cfg.blockDim = dim3(LTPB);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    count_launch();
    return L.uniform >= 0 ? cudaLaunchKernelEx(&cfg, line_step_kernel<false>, a, L, C, F, LineDiv((unsigned)a.nx), zc, rare_thr)
                          : cudaLaunchKernelEx(&cfg, line_step_kernel<true>, a, L, C, F, LineDiv((unsigned)a.nx), zc, rare_thr);
}

}  // namespace tam
