// heat_quad.cu -- the FP32 + Kahan fused heat step, quad form.
//
// For rows of whole 16-byte quads (nx a multiple of 4).  Each thread owns four
// x-adjacent voxels and marches them through a few planes with no staging:
// 128-bit loads straight from L1 / L2 / HBM, the planes' values in registers
// (three buffers in rotation), x neighbours from the neighbouring lanes, face
// differences along x formed once, and the rest of the arithmetic in two-wide
// FP32 instructions (add / sub / fma.f32x2, each half rounded as the scalar
// operation).  Latency is hidden by occupancy alone: 8 blocks of 128 threads per
// SM at 64 registers (32 bytes spilled; several classes, listed: 7 at 72, 132 bytes;
// in the plane: 5 at 96, none); a plane of prefetch in registers cost two blocks per
// SM and 15 % of the speed.  Threads take consecutive quads of a plane, wrapping from
// row to row, so that a block reads one run of memory (tiles 13 to 17 quads
// wide: 20 % slower).
//
// The form before it staged planes of 32 x 8 tiles in shared memory by TMA and was
// held up by its own pipeline: a barrier and two waits per plane, and blocks of 6
// planes however small the grid, so that a step had a floor of 12 us.  Same
// arithmetic, operation for operation.
//
// A step's launch is a programmatic dependent of the step before: its blocks
// are placed while the last of that one drain, and wait for its completion
// before their first load.
//
// What bounds it: HBM on large grids of one class, the latency of a block's few
// planes on small ones; with several classes the issue of the mixed runs' second
// sum and of the voxels beside another class (2 % of the quads on the vessel
// grid, 20 % of the time).  Per step with a core in the damage window, staged form
// before -> now: 64^3 12.8 -> 5.9 us, 100^3 24.0 -> 7.0, 200^3 45.4 -> 30.6 (27.6
// without a source), 256^3 70 -> 58.6, 384^3 218 -> 187; layers 96 x 96 x 48
// 22.8 -> 6.9, 256 x 256 x 128 51.2 -> 49.3; vessels 96^3 21.6 -> 9.0, 256^3
// 78.2 -> 77.6 (77.8 -> 71.8 without a source), 384^3 without a source 234 -> 214.
#include <algorithm>
#include <cstring>

#include "f32x2.cuh"
#include "heat_common.cuh"
#include "slab_common.cuh"

namespace tam {

namespace {

constexpr int QTPB = 128;  // threads per block (256: 1-3 % slower; 64: 10 %)
constexpr int QZMAX = 8;   // planes per block at most (the list holds every voxel of a block)

__device__ __forceinline__ float2 lo2(const float4 &v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4 &v) { return make_float2(v.z, v.w); }
// (plain loads: the step before may still be writing when this kernel starts,
// so the non-coherent path must not be used)
__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

constexpr int TW = 32, TR = 8;  // voxels per tile of the class flags

// The tile flags: for every (tile, plane), the class that all
// voxels of the 32 x 8 tile and of its one-voxel x / y rim (inside the grid)
// hold, or 0xFF when they differ.  One warp per (tile, plane): each lane
// takes one x column of the rim rows and of the tile rows, lanes 0 and 1 the
// rim columns, and the warp compares its lanes' smallest and largest class.
__global__ void tile_flags_kernel(const uint8_t *cls, int pitch, int nx, int ny, int nz, uint8_t *flags)
{
    const int tx = (nx + TW - 1) / TW, ty = (ny + TR - 1) / TR;
    const int64_t items = (int64_t)tx * ty * nz;
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t it = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < items; it += nw) {
        // it = (z * ty + tile row) * tx + tile column: neighbouring warps read neighbouring tiles
        const int txi = (int)(it % tx);
        const int64_t rest = it / tx;
        const int tyi = (int)(rest % ty), z = (int)(rest / ty);
        const int bx = txi * TW, by = tyi * TR;
        const uint8_t *pl = cls + (int64_t)pitch * ny * z;
        int cmin = 255, cmax = -1;
        auto take = [&](int xx, int yy) {
            if (xx < 0 || xx >= nx || yy < 0 || yy >= ny) return;
            const int c = pl[(int64_t)pitch * yy + xx] & (MAX_MAT - 1);
            cmin = min(cmin, c);
            cmax = max(cmax, c);
        };
        for (int yy = by - 1; yy <= by + TR; ++yy) take(bx + lane, yy);
        if (lane < 2)
            for (int yy = by; yy < by + TR; ++yy) take(lane ? bx + TW : bx - 1, yy);
        cmin = __reduce_min_sync(0xffffffffu, cmin);
        cmax = __reduce_max_sync(0xffffffffu, cmax);
        if (lane == 0) flags[((int64_t)tyi * tx + txi) * nz + z] = (uint8_t)(cmin == cmax ? cmin : 0xFF);
    }
}

// Per tile and run of zc planes (x tiles fastest, then y tiles, then runs from
// the top face down): the class that the tile flags of all its planes
// z0 - 1 .. z1 (inside the grid) agree on, or 0xFF.
__global__ void block_class_kernel(const uint8_t *flags, int tx, int ty, int nz, int zc, uint8_t *bclass)
{
    const int nzc = (nz + zc - 1) / zc;
    const int64_t items = (int64_t)tx * ty * nzc;
    for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < items; u += (int64_t)gridDim.x * blockDim.x) {
        const int64_t tile = u % ((int64_t)tx * ty);
        const int bz = (int)(u / ((int64_t)tx * ty));
        const int z0 = (nzc - 1 - bz) * zc, z1 = min(nz, z0 + zc);
        const int za = max(z0 - 1, 0), zb = min(z1, nz - 1);
        const uint8_t *f = flags + tile * nz;
        int c = f[za];
        for (int z = za + 1; z <= zb && c != 0xFF; ++z)
            if (f[z] != c) c = 0xFF;
        bclass[u] = (uint8_t)c;
    }
}

// The ghosts of a voxel and of a quad across face f.  A grid of several classes
// has the longer kernel, and its warps waited for instructions: there the ghosts,
// which few quads need, are functions and not 22 copies (256^3 vessels 82.5 -> 77.6
// us per step; one class: 58.6 us in place, 62.0 as functions).
struct Ghost4 {
    float4 t, e;
};
__device__ __noinline__ float2 ghost_call(bool robin, float hd, float k, float ta, float tb, float c, float e)
{
    if (!robin) return make_float2(tb, 0.f);
    const float D = -(hd / k) * ((c - ta) - e), t = c + D;
    return make_float2(t, e + ((t - c) - D));
}
__device__ __noinline__ Ghost4 ghosts_call(bool robin, float hd, float k, float ta, float tb, float4 tc, float4 ec)
{
    if (!robin) return Ghost4{make_float4(tb, tb, tb, tb), make_float4(0.f, 0.f, 0.f, 0.f)};
    const float h = -(hd / k);
    Ghost4 r;
    auto one = [&](float c, float e, float &tg, float &eg) {
        const float D = h * ((c - ta) - e);
        tg = c + D;
        eg = e + ((tg - c) - D);
    };
    one(tc.x, ec.x, r.t.x, r.e.x);
    one(tc.y, ec.y, r.t.y, r.e.y);
    one(tc.z, ec.z, r.t.z, r.e.z);
    one(tc.w, ec.w, r.t.w, r.e.w);
    return r;
}
template <bool HET>
__device__ __forceinline__ void ghost1(const FusedArgs &a, int f, float tc, float ec, float k, float &t, float &e)
{
    const float2 g = HET ? ghost_call(a.bc_type[f] == BC_ROBIN, a.fc[FC_BCHD + f], k, a.fc[FC_BCTA + f], a.fc[FC_BCT + f], tc, ec)
                         : ghost_pair(a, f, tc, ec, k);
    t = g.x, e = g.y;
}
template <bool HET>
__device__ __forceinline__ void ghost4(const FusedArgs &a, int f, const float4 &tc, const float4 &ec, float k, float4 &t,
                                       float4 &e)
{
    if (HET) {
        const Ghost4 r = ghosts_call(a.bc_type[f] == BC_ROBIN, a.fc[FC_BCHD + f], k, a.fc[FC_BCTA + f], a.fc[FC_BCT + f], tc, ec);
        t = r.t, e = r.e;
        return;
    }
    ghost1<HET>(a, f, tc.x, ec.x, k, t.x, e.x);
    ghost1<HET>(a, f, tc.y, ec.y, k, t.y, e.y);
    ghost1<HET>(a, f, tc.z, ec.z, k, t.z, e.z);
    ghost1<HET>(a, f, tc.w, ec.w, k, t.w, e.w);
}

// One class's step constants, each twice: an operand of the two-wide instructions.
struct QConst {
    float2 Cx, Cy, Cz, C6, Ku;
};
// Two voxels' coefficients, face by face.
struct Coef {
    float2 zm, zp, ym, yp, xm, xp, Ku;
};
__device__ __forceinline__ QConst qconst(const FusedArgs &a, float au, float irc, float Pdt)
{
    const float x = a.fc[FC_DT] * a.fc[FC_CX] * au, y = a.fc[FC_DT] * a.fc[FC_CY] * au, z = a.fc[FC_DT] * a.fc[FC_CZ] * au;
    return QConst{dup(x), dup(y), dup(z), dup(2.f * ((x + y) + z)), dup(Pdt * irc)};
}

// A heterogeneous grid's classes: per voxel (rows of cpitch bytes), and per quad
// what its update needs (see quad_status_kernel).
struct QClasses {
    const uint8_t *cls, *qs;
    const float *tab;  // face table and 1 / (rho c): as parameters, each lane's own entry would be read in turn
    int cpitch;
};
constexpr int QS_FACES = 16;  // status c + QS_FACES: class c throughout, summed face by face

// Status of every quad: c where the tile's run is one-class (bclass); c +
// QS_FACES where only the quad's own voxels and their neighbours are all of
// class c: the face-by-face sum of a grid of several classes, with one
// coefficient per axis; 0xFF: a coefficient per face.
__global__ void quad_status_kernel(const uint8_t *cls, int pitch, int nx, int ny, int nz, const uint8_t *bclass, int tx,
                                   int ty, int zc, uint8_t *qs, unsigned *nmixed)
{
    const int nq = nx / 4, nzc = (nz + zc - 1) / zc;
    const int64_t n = (int64_t)nq * ny * nz;
    unsigned mixed = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int x = 4 * (int)(i % nq), y = (int)(i / nq % ny), z = (int)(i / nq / ny);
        const int bc = bclass[((int64_t)(nzc - 1 - z / zc) * ty + y / TR) * tx + x / TW];
        if (bc < MAX_MAT) {
            qs[i] = (uint8_t)bc;
            continue;
        }
        const uint8_t *p = cls + (int64_t)pitch * (y + (int64_t)ny * z) + x;
        const int c = p[0] & (MAX_MAT - 1);
        bool one = true;
        auto look = [&](const uint8_t *q, int m) {
            for (int k = 0; k < m; ++k) one = one && (q[k] & (MAX_MAT - 1)) == c;
        };
        look(p, 4);
        if (x > 0) look(p - 1, 1);
        if (x + 4 < nx) look(p + 4, 1);
        if (y > 0) look(p - pitch, 4);
        if (y + 1 < ny) look(p + pitch, 4);
        if (z > 0) look(p - (int64_t)pitch * ny, 4);
        if (z + 1 < nz) look(p + (int64_t)pitch * ny, 4);
        qs[i] = (uint8_t)(one ? c + QS_FACES : 0xFF);
        mixed += one ? 0u : 1u;
    }
    mixed = __reduce_add_sync(0xffffffffu, mixed);
    if ((threadIdx.x & 31) == 0 && mixed) atomicAdd(nmixed, mixed);
}

// The kernel's forms: a grid of one class; of several, the quads beside another class
// listed and taken at the block's end; the same with those quads done in their plane.
//
// Listed, the quads beside another class cost a pass of scattered loads: on grids full of
// class boundaries that was most of the step (192^3 of random classes 113 us, of 8^3
// blocks 95, where the staged form took 47).  In their plane each voxel looks up its
// classes, a word per quad and neighbour (the next plane's is carried on, and so are the
// coefficients of the faces above), and its coefficients in shared memory: 44.5 and 44.4
// us, with the listed form's operations and bits.  5 blocks per SM at 96 registers, no
// spills (6 at 80: 192^3 46.0, 256^3 85.5 -> 95.8).
enum QForm { Q_ONE, Q_LISTED, Q_MIXED };
// Q_MIXED from this share of quads beside another class.  us per step listed / in the
// plane: 256^3 2 % 77.5 / 88.4, 9 % 104 / 91, 21 % 121 / 88; 192^3 2 % 37.4 / 44.3, 9 %
// 49.7 / 46.3; 128^3 2 % 14.0 / 15.7, 7 % 18.2 / 16.0; 256 x 256 x 128 in three layers
// (3 %) 54.7 / 57.6, 96 x 96 x 48 (8 %) 12.1 / 7.7.  (One quad in twelve beside another
// class is the worst of both: the staged form took 43.1 us there on 192^3, 90.1 on 256^3.)
constexpr int QMIX_SHARE = 20;

template <int FORM>
__global__ void __launch_bounds__(QTPB, FORM == Q_ONE ? 8 : (FORM == Q_LISTED ? 7 : 5))
    quad_step_kernel(const __grid_constant__ FusedArgs a, const __grid_constant__ ClassLut L,
                     const __grid_constant__ QClasses C, int zchunk, float rare_thr)
{
    constexpr bool HET = FORM != Q_ONE, MIX = FORM == Q_MIXED;
    __shared__ unsigned short s_list[QTPB * 4 * QZMAX];
    __shared__ int s_cnt;
    __shared__ unsigned short s_faces[FORM == Q_LISTED ? QTPB * QZMAX : 1];
    __shared__ int s_nf;
    // face coefficients (MIX: times the axis's factor, x, y, z)
    __shared__ float s_fa[HET ? (MIX ? 3 : 1) * MAX_MAT * MAX_MAT : 1];
    __shared__ QConst s_q[HET ? MAX_MAT : 1];
    __shared__ float s_k[MIX ? MAX_MAT : 1];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (threadIdx.x == 0) s_cnt = s_nf = 0;
    const float Pdt = step_pdt<float>(a);
    const bool src = Pdt != 0.f;  // without a source J is not read
    if (HET) {
        constexpr int N = MAX_MAT * MAX_MAT;
        for (int t = threadIdx.x; t < N; t += QTPB) {
            const float f = __ldg(C.tab + t);
            if (MIX) {
                s_fa[t] = a.fc[FC_DT] * a.fc[FC_CX] * f;
                s_fa[N + t] = a.fc[FC_DT] * a.fc[FC_CY] * f;
                s_fa[2 * N + t] = a.fc[FC_DT] * a.fc[FC_CZ] * f;
            } else {
                s_fa[t] = f;
            }
        }
        if (MIX && threadIdx.x < MAX_MAT) s_k[threadIdx.x] = L.k[threadIdx.x];
        if (threadIdx.x < MAX_MAT) s_q[threadIdx.x] = qconst(a, __ldg(C.tab + threadIdx.x * (MAX_MAT + 1)), __ldg(C.tab + N + threadIdx.x), Pdt);
    }
    __syncthreads();
    const int nx = a.nx, ny = a.ny, nz = a.nz, nq = nx >> 2, pl = nx * ny;
    const unsigned q0 = blockIdx.x * QTPB, qid = q0 + threadIdx.x;
    const int y = (int)(qid / (unsigned)nq), x = 4 * (int)(qid - (unsigned)y * (unsigned)nq);
    // runs of planes from the top face down: the beam enters there, so the
    // blocks with the longest lists start first
    const int nzc = (nz + zchunk - 1) / zchunk;
    const int z0 = (nzc - 1 - (int)blockIdx.y) * zchunk, z1 = min(nz, z0 + zchunk);
    const float *T = (const float *)a.T_in, *E = a.Tc_in, *J = (const float *)a.J;
    float *To = (float *)a.T_out, *Eo = a.Tc_out;
    const int uc = L.uniform >= 0 ? L.uniform : 0;
    const unsigned thr = __float_as_uint(rare_thr);
    const bool act = y < ny;
    const int lane = threadIdx.x & 31;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    {
        int v = act ? x + nx * y + pl * z0 : pl * z0;
        const int oyl = act && y > 0 ? -nx : 0, oyh = act && y < ny - 1 ? nx : 0;
        // the x neighbour that no lane of the warp holds
        const int oe = lane == 0 ? -1 : 4;
        const bool ed = act && ((lane == 0 && x > 0) || (lane == 31 && x + 4 < nx));
        const bool bnd = x == 0 || x + 4 == nx || y == 0 || y == ny - 1;
        // the class's constants: in registers, or (several classes) read where they are used
        const QConst qu = qconst(a, L.fa[uc * MAX_MAT + uc], L.irc[uc], Pdt);
        const QConst *qp = &qu;
        int st = 0;  // HET: the quad's status
        // MIX: the classes of the quad's voxels and of those in the planes around it, a byte each
        constexpr unsigned CMASK = 0x01010101u * (MAX_MAT - 1);
        const int64_t cpl = (int64_t)C.cpitch * ny;
        const uint8_t *cp = MIX ? C.cls + (act ? x + (int64_t)C.cpitch * y : 0) + cpl * z0 : nullptr;
        const int cyl = oyl ? -C.cpitch : 0, cyh = oyh ? C.cpitch : 0;
        auto word = [](const uint8_t *p) { return __ldg(reinterpret_cast<const unsigned *>(p)) & CMASK; };
        // entry of the face table: byte b of a word of index pairs
        auto fa = [&](int axis, unsigned w, int b) {
            const unsigned o = (b ? w >> (8 * b - 2) : w << 2) & 0x3FCu;
            return *reinterpret_cast<const float *>(reinterpret_cast<const char *>(s_fa + axis * MAX_MAT * MAX_MAT) + o);
        };
        unsigned kc = 0;
        float4 fzc = make_float4(0.f, 0.f, 0.f, 0.f);  // coefficients of the faces below
        if (MIX) {
            kc = word(cp);
            const unsigned w = kc << 4 | (z0 > 0 ? word(cp - cpl) : kc);
            fzc = make_float4(fa(2, w, 0), fa(2, w, 1), fa(2, w, 2), fa(2, w, 3));
        }
        float4 A[3], B[3];  // T and the Kahan term of three planes, in rotation
        {
            const int w = v - (z0 > 0 ? pl : 0);
            A[0] = ld4(T + w), B[0] = ld4(E + w);
            A[1] = ld4(T + v), B[1] = ld4(E + v);
        }
        auto step = [&](int z, float4 &tp, float4 &ep, const float4 &tc, const float4 &ec, float4 &tnx, float4 &enx) {
            // the next plane, and this plane's source and neighbours
            const int w2 = v + (z + 1 < nz ? pl : 0);
            tnx = ld4(T + w2);
            enx = ld4(E + w2);
            float4 j = make_float4(0.f, 0.f, 0.f, 0.f);
            if (src) j = ld4(J + v);
            float4 yl = ld4(T + v + oyl), yel = ld4(E + v + oyl), yh = ld4(T + v + oyh), yeh = ld4(E + v + oyh);
            float te = 0.f, ee = 0.f;
            if (ed) te = T[v + oe], ee = E[v + oe];
            float xl = __shfl_up_sync(0xffffffffu, tc.w, 1), xr = __shfl_down_sync(0xffffffffu, tc.x, 1);
            float el = __shfl_up_sync(0xffffffffu, ec.w, 1), er = __shfl_down_sync(0xffffffffu, ec.x, 1);
            if (lane == 0) xl = te, el = ee;
            if (lane == 31) xr = te, er = ee;
            if (HET) {
                st = __ldg(C.qs + (v >> 2));
                qp = s_q + (st & (QS_FACES - 1));
            }
            unsigned kn = 0, kyl = 0, kyh = 0, kxl = 0, kxr = 0;
            if (MIX) {
                // (outside the grid: the voxel's own class)
                kn = z + 1 < nz ? word(cp + cpl) : kc;
                kyl = word(cp + cyl), kyh = word(cp + cyh);
                const unsigned ke = ed ? __ldg(cp + oe) & (MAX_MAT - 1) : 0u;
                kxl = __shfl_up_sync(0xffffffffu, kc, 1) >> 24, kxr = __shfl_down_sync(0xffffffffu, kc, 1) & (MAX_MAT - 1);
                if (lane == 0) kxl = ke;
                if (lane == 31) kxr = ke;
                if (x == 0) kxl = kc & (MAX_MAT - 1);
                if (x + 4 == nx) kxr = kc >> 24;
            }
            // the next plane's faces below are this plane's faces above
            float4 fzn = make_float4(0.f, 0.f, 0.f, 0.f);
            if (MIX) {
                const unsigned w = kc << 4 | kn;
                fzn = make_float4(fa(2, w, 0), fa(2, w, 1), fa(2, w, 2), fa(2, w, 3));
            }
            const QConst &q = *qp;
            float4 tn = tnx, en = enx;
            if (MIX) {
                // ghost neighbours, each voxel of its own class
                auto ghosts = [&](int f, float4 &t, float4 &e) {
                    ghost1<true>(a, f, tc.x, ec.x, s_k[kc & 255u], t.x, e.x);
                    ghost1<true>(a, f, tc.y, ec.y, s_k[kc >> 8 & 255u], t.y, e.y);
                    ghost1<true>(a, f, tc.z, ec.z, s_k[kc >> 16 & 255u], t.z, e.z);
                    ghost1<true>(a, f, tc.w, ec.w, s_k[kc >> 24], t.w, e.w);
                };
                if (bnd) {
                    if (x == 0) ghost1<true>(a, 0, tc.x, ec.x, s_k[kc & 255u], xl, el);
                    if (x + 4 == nx) ghost1<true>(a, 1, tc.w, ec.w, s_k[kc >> 24], xr, er);
                    if (y == 0) ghosts(2, yl, yel);
                    if (y == ny - 1) ghosts(3, yh, yeh);
                }
                if (z == 0) ghosts(4, tp, ep);
                if (z == nz - 1) ghosts(5, tn, en);
            } else if (bnd) {
                // ghost neighbours
                const float k = L.k[HET ? st & (QS_FACES - 1) : uc];
                if (x == 0) ghost1<false>(a, 0, tc.x, ec.x, k, xl, el);
                if (x + 4 == nx) ghost1<false>(a, 1, tc.w, ec.w, k, xr, er);
                if (y == 0) ghost4<HET>(a, 2, tc, ec, k, yl, yel);
                if (y == ny - 1) ghost4<HET>(a, 3, tc, ec, k, yh, yeh);
            }
            if (!MIX && z == 0) ghost4<HET>(a, 4, tc, ec, L.k[HET ? st & (QS_FACES - 1) : uc], tp, ep);
            if (!MIX && z == nz - 1) ghost4<HET>(a, 5, tc, ec, L.k[HET ? st & (QS_FACES - 1) : uc], tn, en);
            float2 t0 = {}, e0 = {}, t1 = {}, e1 = {};
            if (!HET || st < QS_FACES) {
                // sum over the faces of C_f [(T_f - T_c) - (e_f - e_c)]; x: face differences once each
                const float d0 = xl - tc.x, d1 = tc.y - tc.x, d2 = tc.z - tc.y, d3 = tc.w - tc.z, d4 = xr - tc.w;
                const float2 sx0 = sub2(make_float2(d0 + d1, d2 - d1), make_float2(el + ec.y, ec.x + ec.z));
                const float2 sx1 = sub2(make_float2(d3 - d2, d4 - d3), make_float2(ec.y + ec.w, ec.z + er));
                auto half = [&](float2 c, float2 e, float2 sx, float2 ym, float2 yp, float2 em, float2 eq, float2 zm,
                                float2 zp, float2 fm, float2 fq, float2 jj, float2 &tt, float2 &ek) {
                    const float2 sy = sub2(add2(sub2(ym, c), sub2(yp, c)), add2(em, eq));
                    const float2 sz = sub2(add2(sub2(zm, c), sub2(zp, c)), add2(fm, fq));
                    const float2 dT = fma2(q.Cz, sz, fma2(q.Cy, sy, fma2(q.Cx, sx, mul2(q.C6, e))));
                    const float2 yk = sub2(fma2(q.Ku, jj, dT), e);
                    tt = add2(c, yk);
                    ek = sub2(sub2(tt, c), yk);
                };
                half(lo2(tc), lo2(ec), sx0, lo2(yl), lo2(yh), lo2(yel), lo2(yeh), lo2(tp), lo2(tn), lo2(ep), lo2(en), lo2(j), t0, e0);
                half(hi2(tc), hi2(ec), sx1, hi2(yl), hi2(yh), hi2(yel), hi2(yeh), hi2(tp), hi2(tn), hi2(ep), hi2(en), hi2(j), t1, e1);
            } else if (MIX || st < 2 * QS_FACES) {
                // face by face; one class around: with one coefficient per axis
                const float dx0 = (xl - tc.x) - (el - ec.x), dx1 = (tc.y - tc.x) - (ec.y - ec.x);
                const float dx2 = (tc.z - tc.y) - (ec.z - ec.y), dx3 = (tc.w - tc.z) - (ec.w - ec.z);
                const float dx4 = (xr - tc.w) - (er - ec.w);
                auto half = [&](float2 c, float2 e, float2 xm, float2 xp, float2 ym, float2 yp, float2 em, float2 eq,
                                float2 zm, float2 zp, float2 fm, float2 fq, float2 jj, const Coef &F, float2 &tt, float2 &ek) {
                    const float2 zM = sub2(sub2(zm, c), sub2(fm, e)), zP = sub2(sub2(zp, c), sub2(fq, e));
                    const float2 yM = sub2(sub2(ym, c), sub2(em, e)), yP = sub2(sub2(yp, c), sub2(eq, e));
                    const float2 dT = add2(add2(fma2(F.zm, zM, mul2(F.zp, zP)), fma2(F.ym, yM, mul2(F.yp, yP))), fma2(F.xm, xm, mul2(F.xp, xp)));
                    const float2 yk = sub2(fma2(F.Ku, jj, dT), e);
                    tt = add2(c, yk);
                    ek = sub2(sub2(tt, c), yk);
                };
                // the coefficients of voxels b and b + 1 of the quad; pairs of classes, own and neighbour's
                const unsigned own = kc << 4;
                auto coef = [&](int b) -> Coef {
                    if (!MIX) return Coef{q.Cz, q.Cz, q.Cy, q.Cy, q.Cx, q.Cx, q.Ku};
                    auto two = [&](int axis, unsigned w) { return make_float2(fa(axis, w, b), fa(axis, w, b + 1)); };
                    const unsigned wx = own | kc >> 8;  // with the next voxel of the quad
                    const float mid = fa(0, wx, b);
                    const float2 xm = make_float2(b ? fa(0, wx, 1) : fa(0, own | kxl, 0), mid), xp = make_float2(mid, b ? fa(0, own >> 24 | kxr, 0) : fa(0, wx, 1));
                    auto ku = [&](int i) { return s_q[kc >> (8 * i) & 255u].Ku.x; };
                    return Coef{b ? hi2(fzc) : lo2(fzc), b ? hi2(fzn) : lo2(fzn), two(1, own | kyl), two(1, own | kyh), xm, xp, make_float2(ku(b), ku(b + 1))};
                };
                half(lo2(tc), lo2(ec), make_float2(dx0, -dx1), make_float2(dx1, dx2), lo2(yl), lo2(yh), lo2(yel), lo2(yeh), lo2(tp), lo2(tn), lo2(ep), lo2(en), lo2(j), coef(0), t0, e0);
                half(hi2(tc), hi2(ec), make_float2(-dx2, -dx3), make_float2(dx3, dx4), hi2(yl), hi2(yh), hi2(yel), hi2(yeh), hi2(tp), hi2(tn), hi2(ep), hi2(en), hi2(j), coef(2), t1, e1);
            } else if (act) {
                // several classes around: after the planes, see below
                s_faces[atomicAdd(&s_nf, 1)] = (unsigned short)((z - z0) * QTPB + (int)threadIdx.x);
            }
            if (act && (FORM != Q_LISTED || st != 0xFF)) {
                *reinterpret_cast<float4 *>(To + v) = make_float4(t0.x, t0.y, t1.x, t1.y);
                *reinterpret_cast<float4 *>(Eo + v) = make_float4(e0.x, e0.y, e1.x, e1.y);
                // listed: an old or new temperature at the screen, negative or NaN
                // (rare_screen), one test for the quad first
                const unsigned m4[4] = {hot_word(tc.x, t0.x), hot_word(tc.y, t0.y), hot_word(tc.z, t1.x), hot_word(tc.w, t1.y)};
                if (max(max(m4[0], m4[1]), max(m4[2], m4[3])) >= thr) {
                    unsigned fix = 0;
#pragma unroll
                    for (int k = 0; k < 4; ++k) fix |= (m4[k] >= thr ? 1u : 0u) << k;
                    int at = atomicAdd(&s_cnt, __popc(fix));
                    const int l = ((z - z0) * QTPB + (int)threadIdx.x) * 4;
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (fix >> k & 1u) s_list[at++] = (unsigned short)(l + k);
                }
            }
            v += pl;
            if (MIX) kc = kn, fzc = fzn, cp += act ? cpl : 0;
        };
        for (int z = z0;;) {
            step(z, A[0], B[0], A[1], B[1], A[2], B[2]);
            if (++z == z1) break;
            step(z, A[1], B[1], A[2], B[2], A[0], B[0]);
            if (++z == z1) break;
            step(z, A[2], B[2], A[0], B[0], A[1], B[1]);
            if (++z == z1) break;
        }
    }
    __syncthreads();
    if (FORM == Q_LISTED) {
        // Voxels beside another class, a coefficient per face, one per thread: few lie
        // together (2.6 quads in each of 24 % of the warps on 256^3 vessels), and
        // inside the planes each holds up its warp (142 us per step against 78).  A
        // list per grid, with blocks of its own, read each neighbour row as lines
        // of its own (97 us); tiles of mixed runs in a kernel of their own: 81.
        const int nf = 4 * s_nf;
        for (int n = threadIdx.x; n < nf; n += QTPB) {
            const int l = s_faces[n >> 2];
            const int vp = 4 * (int)(q0 + l % QTPB) + (n & 3), z = z0 + l / QTPB, v = vp + pl * z, yy = vp / nx, xx = vp - yy * nx;
            const int64_t cp = C.cpitch, ci = xx + cp * (yy + (int64_t)ny * z);
            const int k = C.cls[ci] & (MAX_MAT - 1);
            const float tc = T[v], e0 = E[v], kk = L.k[k];
            const float *frow = s_fa + k * MAX_MAT;
            auto face = [&](bool in, int f, int dv, int64_t dc, float &t, float &e) -> float {
                if (in) {
                    t = T[v + dv];
                    e = E[v + dv];
                    return frow[C.cls[ci + dc] & (MAX_MAT - 1)];
                }
                ghost1<true>(a, f, tc, e0, kk, t, e);
                return frow[k];
            };
            float txm, txp, tyM, tyP, tzM, tzP, exm, exp_, eyM, eyP, ezM, ezP;
            const float cxd = a.fc[FC_DT] * a.fc[FC_CX], cyd = a.fc[FC_DT] * a.fc[FC_CY], czd = a.fc[FC_DT] * a.fc[FC_CZ];
            const float axm = cxd * face(xx > 0, 0, -1, -1, txm, exm), axp = cxd * face(xx < nx - 1, 1, 1, 1, txp, exp_);
            const float aym = cyd * face(yy > 0, 2, -nx, -cp, tyM, eyM), ayp = cyd * face(yy < ny - 1, 3, nx, cp, tyP, eyP);
            const float azm = czd * face(z > 0, 4, -pl, -cp * ny, tzM, ezM), azp = czd * face(z < nz - 1, 5, pl, cp * ny, tzP, ezP);
            const float sz = __fmaf_rn(azm, (tzM - tc) - (ezM - e0), azp * ((tzP - tc) - (ezP - e0)));
            const float sy = __fmaf_rn(aym, (tyM - tc) - (eyM - e0), ayp * ((tyP - tc) - (eyP - e0)));
            const float sx = __fmaf_rn(axm, (txm - tc) - (exm - e0), axp * ((txp - tc) - (exp_ - e0)));
            const float inc = __fmaf_rn(s_q[k].Ku.x, src ? J[v] : 0.f, (sz + sy) + sx);
            const float yk = inc - e0, t = tc + yk;
            To[v] = t;
            Eo[v] = (t - tc) - yk;
            if (hot_word(tc, t) >= thr) s_list[atomicAdd(&s_cnt, 1)] = (unsigned short)(4 * l + (n & 3));
        }
        if (nf) __syncthreads();
    }
    // the listed voxels (this block's own stores come first), four at a time so
    // that their loads overlap: the damage window's here, boiling, ablation, NaN
    // and negative ones through slab_fix
    const int cnt = s_cnt;
    const double t_new = step_tnew(a);
    const int64_t ni = (int64_t)pl * nz;
    unsigned errbits = 0;
    constexpr int NB = 4;
    for (int n = threadIdx.x; n < cnt; n += NB * QTPB) {
        int vv[NB];
        float tt[NB], ee[NB], tcv[NB];
        double oo[NB];
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            const int m = n + j * QTPB;
            vv[j] = -1;
            if (m < cnt) {
                const int l = s_list[m];
                // (rows are whole quads, so a thread's quad index is its place in the plane)
                vv[j] = 4 * (int)(q0 + (l >> 2) % QTPB) + (l & 3) + pl * (z0 + (l >> 2) / QTPB);
                tt[j] = To[vv[j]];
                ee[j] = Eo[vv[j]];
                tcv[j] = T[vv[j]];
                oo[j] = a.omega[vv[j]];
            }
        }
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            if (vv[j] < 0) continue;
            const float Ts = tt[j] - ee[j];
            const bool general = (a.boil && tcv[j] >= a.fc[FC_TBOIL]) || !(Ts >= 0.f) ||
                                 ge_ff(tt[j], ee[j], a.fc[FC_TABL], a.fc[FC_TABL_LO]);
            if (general)
                slab_fix<!HET>(a, L, C.cls, C.cpitch, vv[j] % nx, (vv[j] / nx) % ny, vv[j] / pl, Pdt, t_new, errbits, T, E, To, Eo, HET ? -1 : uc);
            else if (Ts >= a.fc[FC_SCREEN]) rare_update_f32(a, vv[j], ni, tt[j], ee[j], t_new, true, oo[j]);
        }
    }
    if (errbits) atomicOr(a.err, errbits);
}

}  // namespace

bool quad_step_supported(int nx, int ny, int nz)
{
    return nx > 0 && nx % 4 == 0 && nz <= QZMAX * 65535 && (int64_t)nx * ny * nz < ((int64_t)1 << 31) - 64;
}

static int64_t tiles_of(int nx, int ny, int nz) { return (int64_t)((nx + TW - 1) / TW) * ((ny + TR - 1) / TR) * nz; }

// face table, 1 / (rho c), the count of quads beside another class
constexpr int64_t CNT_AT = 4 * MAX_MAT * (MAX_MAT + 1), TAB_BYTES = CNT_AT + 16;

int64_t quad_class_bytes(int nx, int ny, int nz) { return TAB_BYTES + (int64_t)(nx / 4) * ny * nz + 2 * tiles_of(nx, ny, nz); }

cudaError_t launch_quad_classes(const ClassLut &L, const uint8_t *cls, int pitch, int nx, int ny, int nz, int zchunk, uint8_t *mem,
                                bool *mixed, cudaStream_t s)
{
    float tab[MAX_MAT * (MAX_MAT + 1) + 1];
    std::memcpy(tab, L.fa, 4 * MAX_MAT * MAX_MAT);
    std::memcpy(tab + MAX_MAT * MAX_MAT, L.irc, 4 * MAX_MAT);
    tab[MAX_MAT * (MAX_MAT + 1)] = 0.f;  // the count
    cudaError_t e = cudaMemcpyAsync(mem, tab, sizeof tab, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return e;
    uint8_t *qs = mem + TAB_BYTES;
    // the runs that one-class tiles are looked for in
    const int zc = std::min(std::min(zchunk > 0 ? zchunk : 6, 8), nz);
    const int tx = (nx + TW - 1) / TW, ty = (ny + TR - 1) / TR;
    const int64_t quads = (int64_t)(nx / 4) * ny * nz, tiles = tiles_of(nx, ny, nz), items = (int64_t)tx * ty * ((nz + zc - 1) / zc);
    uint8_t *tflag = qs + quads, *bclass = tflag + tiles;
    auto blocks = [](int64_t n, int per) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + per - 1) / per, 152 * 32)); };
    count_launch(3);
    tile_flags_kernel<<<blocks(tiles, 8), 256, 0, s>>>(cls, pitch, nx, ny, nz, tflag);
    block_class_kernel<<<blocks(items, 256), 256, 0, s>>>(tflag, tx, ty, nz, zc, bclass);
    quad_status_kernel<<<blocks(quads, 256), 256, 0, s>>>(cls, pitch, nx, ny, nz, bclass, tx, ty, zc, qs, (unsigned *)(mem + CNT_AT));
    unsigned n = 0;
    if ((e = cudaGetLastError()) == cudaSuccess) e = cudaMemcpyAsync(&n, mem + CNT_AT, sizeof n, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    *mixed = (int64_t)n * QMIX_SHARE > quads;
    return e;
}

cudaError_t launch_quad_step(const FusedArgs &a0, const ClassLut &L, const uint8_t *cls, int cpitch, const uint8_t *mem,
                             bool mixed, cudaStream_t s)
{
    FusedArgs a = a0;
    fill_fused_consts(a);
    const float rare_thr = rare_screen(a);
    const int bx = (int)(((int64_t)(a.nx / 4) * a.ny + QTPB - 1) / QTPB);
    // planes per block: as many as leave 5000 blocks (four waves), at most 5.
    // Per step with a core in the damage window, 1 / 2 / 3 / 4 / 6 planes: 64^3 5.7 /
    // 8.4 / 10.6 / 12.7 / 16.2 us; 128^3 9.6 / 11.1 / 12.4 / 14.9 / 19.2; 200^3 37.5 /
    // 33.2 / 32.0 / 31.9 / 36.8; 256^3 73.8 / 63.7 / 62.0 / 60.9 / 60.9 (5: 60.3)
    int zc = a.zchunk > 0 ? std::min(QZMAX, a.zchunk) : (int)std::min<int64_t>(5, ((int64_t)bx * a.nz + 4999) / 5000);
    zc = std::max(zc, (a.nz + 65534) / 65535);
    const QClasses C{cls, mem + TAB_BYTES, reinterpret_cast<const float *>(mem), cpitch};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)bx, (unsigned)((a.nz + zc - 1) / zc));
    cfg.blockDim = dim3(QTPB);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    count_launch();
    if (L.uniform >= 0) return cudaLaunchKernelEx(&cfg, quad_step_kernel<Q_ONE>, a, L, C, zc, rare_thr);
    return mixed ? cudaLaunchKernelEx(&cfg, quad_step_kernel<Q_MIXED>, a, L, C, zc, rare_thr)
                 : cudaLaunchKernelEx(&cfg, quad_step_kernel<Q_LISTED>, a, L, C, zc, rare_thr);
}

}  // namespace tam
