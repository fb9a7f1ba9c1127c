// 3D time step in two launches, the reference's pass structure (pass 1: D+ and the material sandwich
// into scratch arrays; pass 2: D- and the time update with Q), for any grid: no alignment of rows is
// needed and every pass-1 output is formed once.
//   Iso: prop3DAcoIsoDenQ_DEO2_FDTD.h:841-893, :1108-1159; VTI: prop3DAcoVTIDenQ_DEO2_FDTD.h:945-957,
//   :1372-1378 (linear :1697-1698); TTI: prop3DAcoTTIDenQ_DEO2_FDTD.h:885-976, :1420-1421.
//
// A CTA of 256 threads owns a (z,y) tile of 32 x 16 columns and marches along a chunk of x planes; a lane
// is a z column, a thread the two rows 2w and 2w+1 of its warp w, handled as one packed FP32 pair. x
// windows are register queues; the centre plane goes to shared memory (the thread's own cells from its
// registers, the y and z halos loaded one plane ahead, with the free-surface images), double buffered,
// one barrier a plane, so that the stencils' loads have constant offsets and need no address
// arithmetic. Global loads are single floats, coalesced along z; columns and rows outside the grid read
// the nearest cell and are selected away.
//
// 60 (Iso), 116 (VTI) and 132 (TTI) bytes a cell in the two passes together, TTI at 61 % of the measured 6547
// GB/s: bound by the latency of a plane's loads at 16 warps an SM. 203 x 181 x 251 a step: TTI 302 us, VTI 286
// us (one thread a cell with 64-bit index arithmetic, 428 instructions a cell and pass where these take 218:
// 403 and 321 us). Tried and slower: 3 CTAs an SM (80 registers: fewer loads in flight, TTI 433 us); every
// array through cp.async two planes ahead (LSU queues, TTI 317 us). Chunks of 8, 16 and 32 planes: 305, 302,
// 336 us. CTAs of 128 threads took 290 us there (TTI; 10 % longer at 64^3, which these kernels are not given): not
// taken up, other sizes were not measured.
#include "wfd_kernels.h"

namespace WFD_NS {
using namespace wfd;

namespace {

constexpr int TZ = 32, NW = 8, TY = 2 * NW, NT = 32 * NW;
constexpr int PZ = TZ + 8;            // pitch of a staged row
constexpr int BH = (TY + 7) * PZ;     // a staged plane with both halos

__device__ __forceinline__ float2 bc2(float s) { return make_float2(s, s); }
#if WFD_STRICT
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return make_float2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return add2(mul2(a, b), c); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return add2(neg2(b), a); }
#else
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 neg2(float2 a) { return __fmul2_rn(a, make_float2(-1.0f, -1.0f)); }
// b * -1 + a: one packed instruction, rounded once like -b + a
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
#endif
__device__ __forceinline__ float2 sqrt2(float2 a) { return make_float2(sqrtf(a.x), sqrtf(a.y)); }
__device__ __forceinline__ float2 div2(float2 a, float2 b) { return make_float2(a.x / b.x, a.y / b.y); }

// id * (c1(w4-w3) + c2(w5-w2) + c3(w6-w1) + c4(w7-w0)), summed left to right: D+ with w = f(k-3..k+4), D-
// with w = f(k-4..k+3)
template <class W>
__device__ __forceinline__ float2 st8(const Grid &g, float id, const W &w) {
    float2 s = mul2(bc2(g.c1), sub2(w(4), w(3)));
    s = fma2(bc2(g.c2), sub2(w(5), w(2)), s);
    s = fma2(bc2(g.c3), sub2(w(6), w(1)), s);
    return mul2(bc2(id), fma2(bc2(g.c4), sub2(w(7), w(0)), s));
}
__device__ __forceinline__ float2 st8q(const Grid &g, const float2 (&q)[8]) {
    return st8(g, g.idx, [&](int i) { return q[i]; });
}
__device__ __forceinline__ void shift(float2 (&q)[8]) {
#pragma unroll
    for (int i = 0; i < 7; i++) q[i] = q[i + 1];
}

// This thread's column and row pair, and what of it the reference computes.
struct Cols {
    bool ok[2];  // the rows' cells are computed where x is in [4, nx-4)
    bool in[2];  // inside the grid
    bool row0;   // kz = 0 under a free surface
    int z0, y0;  // the tile's corner
    int lane, w;
    long o, o1;  // offsets of the rows in a plane (clamped into the grid)
};

__device__ __forceinline__ Cols columns(const Grid &g) {
    Cols c;
    c.lane = threadIdx.x & 31;
    c.w = threadIdx.x >> 5;
    c.z0 = blockIdx.x * TZ;
    c.y0 = blockIdx.y * TY;
    const int z = c.z0 + c.lane, y = c.y0 + 2 * c.w, nz = (int)g.nz, ny = (int)g.ny;
    const bool zin = z < nz, zok = z < nz - 4 && (z >= 4 || g.fs);
#pragma unroll
    for (int r = 0; r < 2; r++) {
        c.in[r] = zin && y + r < ny;
        c.ok[r] = zok && y + r >= 4 && y + r < ny - 4;
    }
    c.row0 = g.fs && z == 0;
    const int zc = min(z, nz - 1);
    c.o = (long)min(y, ny - 1) * nz + zc;
    c.o1 = (long)min(y + 1, ny - 1) * nz + zc;
    return c;
}

__device__ __forceinline__ float2 ld2(const float *__restrict__ p, const Cols &c) { return make_float2(p[c.o], p[c.o1]); }
__device__ __forceinline__ void st2(float *p, const Cols &c, float2 v) {
    if (c.in[0]) p[c.o] = v.x;
    if (c.in[1]) p[c.o1] = v.y;
}
__device__ __forceinline__ float2 keep(const Cols &c, float2 v) {
    return make_float2(c.ok[0] ? v.x : 0.0f, c.ok[1] ? v.y : 0.0f);
}

// The halo values that this thread brings for the staged planes of NF fields, rows y0+B.., columns
// z0+B..: up to two of a y-halo row (7 rows a field, a warp a row) and one of the z halo (7 columns a
// field, a warp 4 rows). Offsets in a plane, where they go, and the sign of a free-surface image
// (antisymmetric for D+, B = -3; symmetric for D-, B = -4).
template <int NF, int B>
struct Halo {
    static constexpr int NY = (7 * NF + NW - 1) / NW;
    long oy[NY], oz;
    int sy[NY], sz;  // place in the staged plane, -1: none
    int fy[NY], fz;  // field
    float sign;

    __device__ __forceinline__ Halo(const Grid &g, const Cols &c) {
        const int nz = (int)g.nz, ny = (int)g.ny;
#pragma unroll
        for (int i = 0; i < NY; i++) {
            const int t = c.w + NW * i, h = t % 7, r = h < -B ? h : h + TY;
            fy[i] = t / 7;
            sy[i] = t < 7 * NF ? r * PZ - B + c.lane : -1;
            oy[i] = (long)min(max(c.y0 + B + r, 0), ny - 1) * nz + min(c.z0 + c.lane, nz - 1);
        }
        const int h = c.lane & 7, r = 4 * (c.w & 3) + (c.lane >> 3), col = h < -B ? h : h + TZ;
        fz = c.w >> 2;
        sz = h < 7 && fz < NF ? (r - B) * PZ + col : -1;
        int z = c.z0 + B + col;
        sign = 1.0f;
        if (z < 0) {
            sign = B == -3 ? -1.0f : 1.0f;
            z = B == -3 ? -z : -z - 1;
        }
        oz = (long)min(c.y0 + r, ny - 1) * nz + min(z, nz - 1);
    }
};

// Pass 1 on planes [xb, xe) of a chunk.
template <int PHYS>
__global__ void __launch_bounds__(NT, 2) k_pass1_3d(Grid g, Fields F, Scratch S, int xchunk) {
    constexpr int NF = PHYS == ISO ? 1 : 2, NO = 3 * NF;
    __shared__ float sm[2][NF][BH];
    const Cols c = columns(g);
    const int nx = (int)g.nx;
    const int xb = blockIdx.z * xchunk, xe = min(xb + xchunk, nx);
    const int x0 = max(xb, 4), x1 = min(xe, nx - 4);  // planes that the reference computes
    for (int x = xb; x < xe; x++)
        if (x < x0 || x >= x1)
            for (int i = 0; i < NO; i++) st2(S.t[i] + (long)x * g.sx, c, bc2(0.0f));
    if (x0 >= x1) return;
    const Halo<NF, -3> H(g, c);
    const float *fld[2] = {F.pcur, F.mcur};
    float2 q[NF][8];
    float hy[H.NY], hz = 0.0f;
    auto halos = [&](long k) {
#pragma unroll
        for (int i = 0; i < H.NY; i++) hy[i] = H.sy[i] >= 0 ? (H.fy[i] ? F.mcur : F.pcur)[k + H.oy[i]] : 0.0f;
        hz = H.sz >= 0 ? H.sign * (H.fz ? F.mcur : F.pcur)[k + H.oz] : 0.0f;
    };
    halos((long)x0 * g.sx);
#pragma unroll
    for (int f = 0; f < NF; f++)
#pragma unroll
        for (int i = 0; i < 7; i++) q[f][i + 1] = ld2(fld[f] + (long)(x0 - 3 + i) * g.sx, c);
    const int own = (2 * c.w + 3) * PZ + 3 + c.lane;
    for (int x = x0; x < x1; x++) {
        const long k = (long)x * g.sx;
        float(*st)[BH] = sm[x & 1];
#pragma unroll
        for (int f = 0; f < NF; f++) {
            shift(q[f]);
            q[f][7] = ld2(fld[f] + k + 4 * g.sx, c);
            st[f][own] = q[f][3].x;
            st[f][own + PZ] = q[f][3].y;
        }
#pragma unroll
        for (int i = 0; i < H.NY; i++)
            if (H.sy[i] >= 0) st[H.fy[i]][H.sy[i]] = hy[i];
        if (H.sz >= 0) st[H.fz][H.sz] = hz;
        const float2 b = ld2(F.b + k, c);
        float2 eps, eta, fv, sT, cT, sP, cP;
        if (PHYS != ISO) {
            eps = ld2(F.eps + k, c);
            eta = ld2(F.eta + k, c);
            fv = ld2(F.f + k, c);
        }
        if (PHYS == TTI) {
            sT = ld2(F.st + k, c);
            cT = ld2(F.ct + k, c);
            sP = ld2(F.sp + k, c);
            cP = ld2(F.cp + k, c);
        }
        __syncthreads();
        if (x + 1 < x1) halos(k + g.sx);
        float2 dx[NF], dy[NF], dz[NF];
#pragma unroll
        for (int f = 0; f < NF; f++) {
            const float *p = st[f] + own;
            float v[9];
#pragma unroll
            for (int i = 0; i < 9; i++) v[i] = i == 3 ? q[f][3].x : (i == 4 ? q[f][3].y : p[(i - 3) * PZ]);
            dy[f] = st8(g, g.idy, [&](int i) { return make_float2(v[i], v[i + 1]); });
            dz[f] = st8(g, g.idz, [&](int i) { return i == 3 ? q[f][3] : make_float2(p[i - 3], p[PZ + i - 3]); });
            dx[f] = st8q(g, q[f]);
            if (c.row0) dx[f] = dy[f] = bc2(0.0f);
        }
        if constexpr (PHYS == ISO) {
            st2(S.t[0] + k, c, keep(c, mul2(b, dx[0])));
            st2(S.t[1] + k, c, keep(c, mul2(b, dy[0])));
            st2(S.t[2] + k, c, keep(c, mul2(b, dz[0])));
        } else {
            const float2 one = bc2(1.0f), two = bc2(2.0f);
            float2 px, py, pz, mx, my, mz;
            if (PHYS == TTI) {
                const float2 stcp = mul2(sT, cP), stsp = mul2(sT, sP);
                const float2 eta2 = mul2(eta, eta), bvfv = mul2(b, fv);
                const float2 g3P = fma2(cT, dz[0], fma2(stsp, dy[0], mul2(stcp, dx[0])));
                const float2 g3M = fma2(cT, dz[1], fma2(stsp, dy[1], mul2(stcp, dx[1])));
                const float2 tmpFE = mul2(mul2(bvfv, eta), sqrt2(sub2(one, eta2)));
                const float2 tmpP = fma2(tmpFE, g3M, mul2(mul2(neg2(b), fma2(fv, eta2, mul2(two, eps))), g3P));
                const float2 tmpM = fma2(mul2(bvfv, eta2), g3M, mul2(tmpFE, g3P));
                const float2 tmpE = mul2(b, fma2(two, eps, one)), tmpF = mul2(b, sub2(one, fv));
                px = fma2(stcp, tmpP, mul2(tmpE, dx[0]));
                py = fma2(stsp, tmpP, mul2(tmpE, dy[0]));
                pz = fma2(cT, tmpP, mul2(tmpE, dz[0]));
                mx = fma2(stcp, tmpM, mul2(tmpF, dx[1]));
                my = fma2(stsp, tmpM, mul2(tmpF, dy[1]));
                mz = fma2(cT, tmpM, mul2(tmpF, dz[1]));
            } else {
                const float2 BE = mul2(b, fma2(two, eps, one)), BF1 = mul2(b, sub2(one, fv));
                px = mul2(BE, dx[0]);
                py = mul2(BE, dy[0]);
                mx = mul2(BF1, dx[1]);
                my = mul2(BF1, dy[1]);
                const float2 FA = mul2(fv, eta), FAA = mul2(FA, eta), SA2 = sqrt2(sub2(one, mul2(eta, eta)));
                pz = fma2(mul2(b, mul2(FA, SA2)), dz[1], mul2(mul2(b, sub2(one, FAA)), dz[0]));
                mz = fma2(mul2(b, add2(sub2(one, fv), FAA)), dz[1], mul2(mul2(mul2(mul2(b, fv), eta), SA2), dz[0]));
            }
            st2(S.t[0] + k, c, keep(c, px));
            st2(S.t[1] + k, c, keep(c, py));
            st2(S.t[2] + k, c, keep(c, pz));
            st2(S.t[3] + k, c, keep(c, mx));
            st2(S.t[4] + k, c, keep(c, my));
            st2(S.t[5] + k, c, keep(c, mz));
        }
    }
}

// Pass 2 on planes [xb, xe) of a chunk.
template <int PHYS, bool LINEAR>
__global__ void __launch_bounds__(NT, 2) k_pass2_3d(Grid g, Fields F, Scratch S, int xchunk) {
    constexpr int NF = PHYS == ISO ? 1 : 2;
    __shared__ float sm[2][NF][BH], sz_[2][NF][TY * PZ];  // staged y outputs, z outputs
    const Cols c = columns(g);
    const int nx = (int)g.nx;
    const int xb = blockIdx.z * xchunk, xe = min(xb + xchunk, nx);
    const int x0 = max(xb, 4), x1 = min(xe, nx - 4);
    if (!LINEAR)
        for (int x = xb; x < xe; x++)
            if (x < x0 || x >= x1) {
                st2(F.pspace + (long)x * g.sx, c, bc2(0.0f));
                if (PHYS != ISO) st2(F.mspace + (long)x * g.sx, c, bc2(0.0f));
            }
    if (x0 >= x1) return;
    const Halo<NF, -4> H(g, c);
    float2 q[NF][8];
    float hy[H.NY], hz = 0.0f;
    auto halos = [&](long k) {
#pragma unroll
        for (int i = 0; i < H.NY; i++) hy[i] = H.sy[i] >= 0 ? (H.fy[i] ? S.t[4] : S.t[1])[k + H.oy[i]] : 0.0f;
        hz = H.sz >= 0 ? (H.fz ? S.t[5] : S.t[2])[k + H.oz] : 0.0f;
    };
    float2 yo[NF], zo[NF];  // this thread's own y and z outputs of the next plane
    auto owns = [&](long k) {
#pragma unroll
        for (int f = 0; f < NF; f++) {
            yo[f] = ld2(S.t[3 * f + 1] + k, c);
            zo[f] = ld2(S.t[3 * f + 2] + k, c);
        }
    };
    halos((long)x0 * g.sx);
    owns((long)x0 * g.sx);
#pragma unroll
    for (int f = 0; f < NF; f++)
#pragma unroll
        for (int i = 0; i < 7; i++) q[f][i + 1] = ld2(S.t[3 * f] + (long)(x0 - 4 + i) * g.sx, c);
    const int own = (2 * c.w + 4) * PZ + 4 + c.lane, ownz = 2 * c.w * PZ + 4 + c.lane;
    for (int x = x0; x < x1; x++) {
        const long k = (long)x * g.sx;
        float(*st)[BH] = sm[x & 1];
        float(*zt)[TY * PZ] = sz_[x & 1];
#pragma unroll
        for (int f = 0; f < NF; f++) {
            shift(q[f]);
            q[f][7] = ld2(S.t[3 * f] + k + 3 * g.sx, c);
            st[f][own] = yo[f].x;
            st[f][own + PZ] = yo[f].y;
            zt[f][ownz] = zo[f].x;
            zt[f][ownz + PZ] = zo[f].y;
        }
#pragma unroll
        for (int i = 0; i < H.NY; i++)
            if (H.sy[i] >= 0) st[H.fy[i]][H.sy[i]] = hy[i];
        if (H.sz >= 0) zt[H.fz][H.sz - 4 * PZ] = hz;
        const float2 V = ld2(F.v + k, c), B = ld2(F.b + k, c), Q = ld2(F.q + k, c);
        float2 pc[NF], po[NF];
#pragma unroll
        for (int f = 0; f < NF; f++) {
            pc[f] = ld2((f == 0 ? F.pcur : F.mcur) + k, c);
            po[f] = ld2((f == 0 ? F.pold : F.mold) + k, c);
        }
        __syncthreads();
        float2 y1[NF], z1[NF];
#pragma unroll
        for (int f = 0; f < NF; f++) {
            y1[f] = yo[f];
            z1[f] = zo[f];
        }
        if (x + 1 < x1) {
            halos(k + g.sx);
            owns(k + g.sx);
        }
        const float2 k2 = div2(mul2(mul2(bc2(g.dt2), V), V), B);
#pragma unroll
        for (int f = 0; f < NF; f++) {
            const float *p = st[f] + own, *z = zt[f] + ownz;
            float v[9];
#pragma unroll
            for (int i = 0; i < 9; i++) v[i] = i == 4 ? y1[f].x : (i == 5 ? y1[f].y : p[(i - 4) * PZ]);
            const float2 dx = st8q(g, q[f]);
            const float2 dy = st8(g, g.idy, [&](int i) { return make_float2(v[i], v[i + 1]); });
            const float2 dz = st8(g, g.idz, [&](int i) { return i == 4 ? z1[f] : make_float2(z[i - 4], z[PZ + i - 4]); });
            float2 L = add2(add2(dx, dy), dz);
            if (c.row0) L = bc2(0.0f);
            const float2 t = sub2(sub2(mul2(k2, L), mul2(Q, sub2(pc[f], po[f]))), po[f]);
            const float2 np = add2(t, mul2(bc2(2.0f), pc[f]));
            st2((f == 0 ? F.pold : F.mold) + k, c,
                make_float2(c.ok[0] ? np.x : po[f].x, c.ok[1] ? np.y : po[f].y));
            if (!LINEAR) st2((f == 0 ? F.pspace : F.mspace) + k, c, keep(c, L));
        }
    }
}

// planes a CTA marches over: 16 where that leaves four CTAs an SM, else as few as do (each chunk reads 7
// planes of the x windows beside its own, but a CTA's planes follow one another at the latency of
// their loads)
int chunk_of(const Grid &g, dim3 &grid) {
    const long tiles = ((g.nz + TZ - 1) / TZ) * ((g.ny + TY - 1) / TY);
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long n = (4L * sms + tiles - 1) / tiles;  // chunks wanted
    long chunk = (g.nx + n - 1) / n;
    chunk = chunk < 2 ? 2 : (chunk > 16 ? 16 : chunk);
    while ((g.nx + chunk - 1) / chunk > 65535) chunk *= 2;
    grid = dim3((unsigned)((g.nz + TZ - 1) / TZ), (unsigned)((g.ny + TY - 1) / TY), (unsigned)((g.nx + chunk - 1) / chunk));
    return (int)chunk;
}

}  // namespace

// Grids of a million cells and more whose tiles are well filled; the others take one thread a cell
// (wfd_generic.cu). Smaller grids stay in L2 and are bound by the latency of a launch, which one thread a cell hides
// better: TTI 80 x 75 x 69 (414,000 cells) 21.2 us a step there and 23.0 here. The times cross below the line (TTI 100 x
// 110 x 90, 990,000 cells, 41.6 and 36.9); where between these two sizes was not measured, nor for VTI.
// A tile costs the same however much of it is computed, so the second rule is on a plane's tile cells per computed
// cell, r. The lines lie between those of one object stepping alone and of several in turn, whose launches fill each
// other's last waves; us a step there and here, alone; in turn, on both sides of each line:
//   VTI (r <= 1.5)   150 x 113 x 135 r 1.49 88.6, 90.0; 77.5, 77.6    300 x 300 x 50 r 1.45 172, 182; 160, 146
//                    101 x 100 x 101 r 1.61 39.8, 42.4; 35.2, 38.7    12000 x 9 x 10 r 85 33.9, 131.5 (alone)
//   TTI (r <= 1.85)  200 x 120 x 67 r 1.74 72.2, 65.7 (in turn)       101 x 100 x 101 r 1.61 46.0, 47.4; 44.4, 41.3
//                    300 x 70 x 70 r 1.88 67.7, 72.4; 64.6, 62.3      300 x 22 x 301 r 2.46 77.3, 95.9; 69.9, 82.0
//   Iso (r <= 1.5)   150 x 113 x 136 r 1.48 50.4, 45.9 (alone)        300 x 300 x 44 r 1.67 90.8, 99.6 (alone)
// Below 12 planes the zeros that each CTA writes on the planes beside the computed ones show, in TTI less than the
// gain: VTI 9 x 1000 x 301 36.5, 41.3; 35.2, 38.2, TTI 43.8, 42.3; 41.7, 39.0; VTI 14 x 310 x 319 32.4, 31.7; 31.6, 27.7.
bool pass3d_takes(const Grid &g, int phys) {
    if (g.ndim != 3 || g.n < 1000000 || (phys != TTI && g.nx < 12)) return false;
    const long nty = (g.ny + TY - 1) / TY, ntz = (g.nz + TZ - 1) / TZ;
    if (nty > 65535 || ntz >= 2147483647L) return false;
    const double staged = (double)(ntz * TZ) * (double)(nty * TY);
    const double computed = (double)(g.ny - 8) * (double)(g.nz - (g.fs ? 4 : 8));
    return staged <= (phys == TTI ? 1.85 : 1.5) * computed;
}

void pass1_3d(const Grid &g, int phys, const Fields &F, const Scratch &S, cudaStream_t s) {
    dim3 grid;
    const int chunk = chunk_of(g, grid);
    if (phys == ISO) k_pass1_3d<ISO><<<grid, NT, 0, s>>>(g, F, S, chunk);
    else if (phys == VTI) k_pass1_3d<VTI><<<grid, NT, 0, s>>>(g, F, S, chunk);
    else k_pass1_3d<TTI><<<grid, NT, 0, s>>>(g, F, S, chunk);
}

void pass2_3d(const Grid &g, int phys, int linear, const Fields &F, const Scratch &S, cudaStream_t s) {
    dim3 grid;
    const int chunk = chunk_of(g, grid);
    if (phys == ISO) k_pass2_3d<ISO, false><<<grid, NT, 0, s>>>(g, F, S, chunk);
    else if (phys == VTI && linear) k_pass2_3d<VTI, true><<<grid, NT, 0, s>>>(g, F, S, chunk);
    else if (phys == VTI) k_pass2_3d<VTI, false><<<grid, NT, 0, s>>>(g, F, S, chunk);
    else k_pass2_3d<TTI, false><<<grid, NT, 0, s>>>(g, F, S, chunk);
}

}  // namespace WFD_NS
