// A whole 2D time loop (Iso, VTI, TTI) in one cooperative launch as the reference's two passes, each cell's
// pass-1 outputs formed once: for the grids whose fused loop (wfd_fused_iso2d.cu, wfd_fused_aniso2d.cu) has
// more tiles than co-resident CTAs, and would recompute those outputs on every tile's halo and reload
// every material with it, each step. us a step, the fused loop and this one: Iso 1000 x 500 13.2 and 10.9,
// 2400 x 1200 54.8 and 33.0; VTI 26.5 and 17.3, 142 and 89; TTI 33.4 and 26.1, 185 and 115. (With a CTA per
// tile the fused loops keep their tiles in shared memory: 501 x 501 Iso 5.5 against 7.6 here, VTI 12.0 and
// 11.5, TTI 13.9 and 15.7; 250 x 201 VTI 9.9 and 10.5.)
//
// Two CTAs of 512 threads an SM; a warp's lanes are 32 z columns, a thread two consecutive x rows, whose
// derivatives are formed as packed FP32 pairs; CTAs take turns over tiles of 64 z x 16 x cells (CTAs of 256,
// 384 and 1024 threads and tiles 32 and 128 wide were within 10 %). Bound by the latency of the loads from L1 and
// L2 at 32 warps an SM: some 60 loads a cell in Iso and VTI, 113 in TTI (2400 x 1200: long-scoreboard stalls 12 of
// 21 per issue, l1tex 47 %, L2 20 %, DRAM 34 % busy). Per step: pass 1 (the derivatives and the material sandwich) into scratch
// arrays, a grid-wide barrier (bounded, 1.3 us), pass 2 (the divergence and the update) with the step's
// source injection, a barrier, the receivers. Everything stays in L2 up to about 2 M cells; stencil windows
// are plain loads whose reuse within a CTA L1 serves (the barrier's acquire drops what other CTAs may have
// rewritten).
//
// Fast build only (the strict build keeps the fused loops). The arithmetic is the fused step's with its
// contractions written out, so that the fields are the stepping calls' bit for bit. Rotating TTI's pass-1
// outputs back to the grid's axes in pass 1 (pass 2 the plain divergence) took 15.6 us at 1000 x 500, but
// every step then rounds differently, and over some hundred steps the rounding of pSpace drifts apart by
// 1e-3 of its largest values.
#include "wfd_gridbar.cuh"
#include "wfd_kernels.h"

namespace WFD_NS {
using namespace wfd;

#if !WFD_STRICT
namespace {

constexpr int NT = 512, TZ = 64, TX = 2 * NT / TZ;
constexpr int MAX_INJ = 1024;

__device__ __forceinline__ float2 bc2(float s) { return make_float2(s, s); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
__device__ __forceinline__ float2 neg2(float2 a) { return __fmul2_rn(a, make_float2(-1.0f, -1.0f)); }

// c1 d1 + c2 d2 + c3 d3 + c4 d4, rounded as the compiler contracts that sum in the fused step (the first product
// fused into the second), so that this loop's fields are the stepping calls' bit for bit
__device__ __forceinline__ float2 sum4(const Grid &g, float2 d1, float2 d2, float2 d3, float2 d4) {
    return fma2(bc2(g.c4), d4, fma2(bc2(g.c3), d3, fma2(bc2(g.c1), d1, mul2(bc2(g.c2), d2))));
}
// D+ with w(0..7) = f(k-3..k+4), D- with w(0..7) = f(k-4..k+3)
template <class W>
__device__ __forceinline__ float2 st8(const Grid &g, const W &w) {
    return sum4(g, sub2(w(4), w(3)), sub2(w(5), w(2)), sub2(w(6), w(1)), sub2(w(7), w(0)));
}
// the same of products a f (n: the negated weights), each difference with one product rounded
template <class A, class N, class W>
__device__ __forceinline__ float2 st8p(const Grid &g, const A &a, const N &n, const W &w) {
    auto d = [&](int hi, int lo) { return fma2(a(hi), w(hi), mul2(n(lo), w(lo))); };
    return sum4(g, d(4, 3), d(5, 2), d(6, 1), d(7, 0));
}

// a thread's pair of rows at (x, z), (x+1, z)
struct Pair {
    bool ok[2], in[2];  // computed by the reference; inside the grid
    bool top, row0;     // kz < 4 and kz = 0 under a free surface
    int x, z;
    unsigned o[2];      // offsets (the second row's is the first's where that one is outside)
};

__device__ __forceinline__ Pair pair_at(const Grid &g, int x, int z) {
    Pair c;
    const int nx = (int)g.nx, nz = (int)g.nz;
    c.x = x;
    c.z = z;
    const bool zin = z < nz, zok = z < nz - 4 && (z >= 4 || g.fs);
#pragma unroll
    for (int r = 0; r < 2; r++) {
        c.in[r] = zin && x + r < nx;
        c.ok[r] = zok && x + r >= 4 && x + r < nx - 4;
    }
    c.top = g.fs && z < 4;
    c.row0 = g.fs && z == 0;
    c.o[0] = (unsigned)x * (unsigned)nz + (unsigned)z;
    c.o[1] = c.in[1] ? c.o[0] + (unsigned)nz : c.o[0];
    return c;
}

// the windows of a pair (some row is ok). Along x rows x+B .. x+B+8, B = -3 (D+) or -4 (D-): row r's are the
// 8 from r on. A row outside the grid only feeds the row that is not ok and reads the nearest one.
template <int B, bool CONST>
__device__ __forceinline__ void winx(const Grid &g, const float *p, const Pair &c, float (&v)[9]) {
#pragma unroll
    for (int i = 0; i < 9; i++) {
        const float *q = p + ((unsigned)min(max(c.x + B + i, 0), (int)g.nx - 1) * (unsigned)g.nz + (unsigned)c.z);
        v[i] = CONST ? __ldg(q) : *q;
    }
}
__device__ __forceinline__ float2 rows(const float (&v)[9], int i) { return make_float2(v[i], v[i + 1]); }
// Along z columns z+B .. z+B+7; above the free surface the antisymmetric (B = -3) or symmetric image.
template <int B, bool CONST>
__device__ __forceinline__ void winz(const float *p, const Pair &c, float2 (&w)[8]) {
    if (c.top) {
        const float *a = p + (c.o[0] - (unsigned)c.z), *b = p + (c.o[1] - (unsigned)c.z);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int j = c.z + B + i, k = j >= 0 ? j : (B == -3 ? -j : -j - 1);
            const float s = j < 0 && B == -3 ? -1.0f : 1.0f;
            w[i] = make_float2(s * a[k], s * b[k]);
        }
    } else {
        const float *a = p + c.o[0], *b = p + c.o[1];
#pragma unroll
        for (int i = 0; i < 8; i++)
            w[i] = CONST ? make_float2(__ldg(a + B + i), __ldg(b + B + i)) : make_float2(a[B + i], b[B + i]);
    }
}
// D+ of field p for both rows
__device__ __forceinline__ void gradient(const Grid &g, const float *p, const Pair &c, float (&dx)[2], float (&dz)[2]) {
    float v[9];
    float2 w[8];
    winx<-3, false>(g, p, c, v);
    winz<-3, false>(p, c, w);
    float2 x = mul2(bc2(g.idx), st8(g, [&](int i) { return rows(v, i); }));
    const float2 z = mul2(bc2(g.idz), st8(g, [&](int i) { return w[i]; }));
    if (c.row0) x = bc2(0.0f);
    dx[0] = x.x, dx[1] = x.y, dz[0] = z.x, dz[1] = z.y;
}

// pass 1 of a pair: S.t[0], S.t[1] the first and second vector component of P, S.t[2], S.t[3] of M, the
// expressions of the fused step
template <int PHYS>
__device__ __forceinline__ void pass1(const Grid &g, const Fields &F, const Scratch &S, const float *pcur,
                                      const float *mcur, const Pair &c) {
    if (!c.ok[0] && !c.ok[1]) return;
    float dPx[2], dPz[2], dMx[2], dMz[2];
    gradient(g, pcur, c, dPx, dPz);
    if (PHYS != ISO) gradient(g, mcur, c, dMx, dMz);
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const unsigned k = c.o[r];
        const float B = __ldg(F.b + k);
        float o0, o2, o3 = 0.0f, o5 = 0.0f;
        if (PHYS == ISO) {
            o0 = B * dPx[r];
            o2 = B * dPz[r];
        } else {
            const float E = 1 + 2 * __ldg(F.eps + k);
            const float A = __ldg(F.eta + k);
            const float Fv = __ldg(F.f + k);
            if (PHYS == VTI) {
                // prop2DAcoVTIDenQ_DEO2_FDTD.h:771-779
                o0 = B * E * dPx[r];
                o2 = B * (1 - Fv * A * A) * dPz[r] + B * Fv * A * sqrtf(1 - A * A) * dMz[r];
                o3 = B * (1 - Fv) * dMx[r];
                o5 = B * Fv * A * sqrtf(1 - A * A) * dPz[r] + B * (1 - Fv + Fv * A * A) * dMz[r];
            } else {
                // prop2DAcoTTIDenQ_DEO2_FDTD.h:672-760
                const float cosT = __ldg(F.ct + k), sinT = __ldg(F.st + k);
                auto g1 = [&](float x, float z) { return __fmaf_rn(cosT, x, -__fmul_rn(sinT, z)); };
                auto g3 = [&](float x, float z) { return __fmaf_rn(cosT, z, __fmul_rn(sinT, x)); };
                const float dPG1 = g1(dPx[r], dPz[r]), dPG3 = g3(dPx[r], dPz[r]);
                const float dMG1 = g1(dMx[r], dMz[r]), dMG3 = g3(dMx[r], dMz[r]);
                o0 = B * E * dPG1;
                const float X = B * Fv * A * sqrtf(1 - A * A);
                o2 = __fmaf_rn(B * (1 - Fv * A * A), dPG3, __fmul_rn(X, dMG3));
                o3 = B * (1 - Fv) * dMG1;
                o5 = __fmaf_rn(X, dPG3, __fmul_rn(B * (1 - Fv + Fv * A * A), dMG3));
            }
        }
        if (!c.ok[r]) continue;
        S.t[0][k] = o0;
        S.t[1][k] = o2;
        if (PHYS != ISO) {
            S.t[2][k] = o3;
            S.t[3][k] = o5;
        }
    }
}

// the divergence of a pair's pass-1 vector (a, b), VTI and Iso: the sum's x product fused, as in the fused step
__device__ __forceinline__ void divergence(const Grid &g, const float *a, const float *b, const Pair &c, float (&L)[2]) {
    float v[9];
    float2 w[8];
    winx<-4, false>(g, a, c, v);
    winz<-4, false>(b, c, w);
    const float2 dz = mul2(bc2(g.idz), st8(g, [&](int i) { return w[i]; }));
    const float2 s = fma2(bc2(g.idx), st8(g, [&](int i) { return rows(v, i); }), dz);
    L[0] = c.row0 ? 0.0f : s.x;
    L[1] = c.row0 ? 0.0f : s.y;
}
// TTI: the back-rotation inside the stencils (prop2DAcoTTIDenQ_DEO2_FDTD.h:1055-1135), the weights at the
// tap's own cell
__device__ __forceinline__ void divergence_tti(const Grid &g, const Fields &F, const Scratch &S, const Pair &c,
                                               float (&LP)[2], float (&LM)[2]) {
    float2 x[4];  // D- along x of ct t0, st t1, ct t2, st t3
#pragma unroll
    for (int h = 0; h < 2; h++) {  // ct, st
        float a[9], v[9];
        winx<-4, true>(g, h ? F.st : F.ct, c, a);
#pragma unroll
        for (int i = h; i < 4; i += 2) {
            winx<-4, false>(g, S.t[i], c, v);
            x[i] = st8p(g, [&](int k) { return rows(a, k); }, [&](int k) { return neg2(rows(a, k)); },
                        [&](int k) { return rows(v, k); });
        }
    }
    float2 z[4];  // along z of st t0, ct t1, st t2, ct t3
#pragma unroll
    for (int h = 0; h < 2; h++) {
        float2 a[8], w[8];
        winz<-4, true>(h ? F.ct : F.st, c, a);
#pragma unroll
        for (int i = h; i < 4; i += 2) {
            winz<-4, false>(S.t[i], c, w);
            z[i] = st8p(g, [&](int k) { return a[k]; }, [&](int k) { return neg2(a[k]); }, [&](int k) { return w[k]; });
        }
    }
    auto sum = [&](int i) {
        const float2 a = fma2(bc2(g.idx), x[i], mul2(bc2(-g.idz), z[i]));
        const float2 b = fma2(bc2(g.idx), x[i + 1], mul2(bc2(g.idz), z[i + 1]));
        return __fadd2_rn(a, b);
    };
    const float2 P = sum(0), M = sum(2);
    LP[0] = c.row0 ? 0.0f : P.x;
    LP[1] = c.row0 ? 0.0f : P.y;
    LM[0] = c.row0 ? 0.0f : M.x;
    LM[1] = c.row0 ? 0.0f : M.y;
}

// pass 2 of a pair: the divergence and the update; pSpace and mSpace at the last step only
template <int PHYS>
__device__ __forceinline__ void pass2(const Grid &g, const Fields &F, const Scratch &S, const float *pcur, float *pold,
                                      const float *mcur, float *mold, const Pair &c, bool last) {
    if (!c.ok[0] && !c.ok[1]) return;
    float LP[2], LM[2];
    if (PHYS == TTI) {
        divergence_tti(g, F, S, c, LP, LM);
    } else {
        divergence(g, S.t[0], S.t[1], c, LP);
        if (PHYS == VTI) divergence(g, S.t[2], S.t[3], c, LM);
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        if (!c.ok[r]) continue;
        const unsigned k = c.o[r];
        const float V = __ldg(F.v + k);
        const float dt2V2_B = g.dt2 * V * V / __ldg(F.b + k);
        const float Q = __ldg(F.q + k);
        const float pc = pcur[k], po = pold[k];
        pold[k] = dt2V2_B * LP[r] - Q * (pc - po) - po + 2 * pc;
        if (last) F.pspace[k] = LP[r];
        if (PHYS != ISO) {
            const float mc = mcur[k], mo = mold[k];
            mold[k] = dt2V2_B * LM[r] - Q * (mc - mo) - mo + 2 * mc;
            if (last) F.mspace[k] = LM[r];
        }
    }
}

template <int PHYS>
__global__ void __launch_bounds__(NT, 2) k_loop2d(Grid g, Fields F, Scratch S, long nsteps, long it0, RunExtract ex,
                                                  unsigned *sync_words) {
    __shared__ int ok_flag, n_inj;
    __shared__ int inj[MAX_INJ];  // this CTA's source groups
    const int ntz = (int)((g.nz + TZ - 1) / TZ), ntx = (int)((g.nx + TX - 1) / TX), ntiles = ntz * ntx;
    const int zt = threadIdx.x % TZ, xt = threadIdx.x / TZ * 2;
    constexpr int NO = PHYS == ISO ? 2 : 4;
    auto each = [&](auto &&fn) {
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x)
            fn(pair_at(g, t / ntz * TX + xt, t % ntz * TZ + zt));
    };
    // what no step writes: the scratch arrays' and pSpace's cells outside the reference's range
    each([&](const Pair &c) {
        for (int r = 0; r < 2; r++) {
            if (!c.in[r] || c.ok[r]) continue;
            for (int i = 0; i < NO; i++) S.t[i][c.o[r]] = 0.0f;
            F.pspace[c.o[r]] = 0.0f;
            if (PHYS != ISO) F.mspace[c.o[r]] = 0.0f;
        }
    });
    if (threadIdx.x == 0) n_inj = 0;
    __syncthreads();
    for (int gi = threadIdx.x; gi < F.inj.ngroups; gi += NT) {
        if (F.inj.key[gi] >= g.n) continue;  // outside the grid: in no tile, as in the fused loops
        const int x = (int)(F.inj.key[gi] / g.nz), z = (int)(F.inj.key[gi] % g.nz);
        if ((x / TX * ntz + z / TZ) % (int)gridDim.x == (int)blockIdx.x) inj[atomicAdd(&n_inj, 1)] = gi;
    }
    __syncthreads();
    unsigned gen = 0;
    for (long st = 0; st < nsteps; st++) {
        float *pcur = (st & 1) ? F.pold : F.pcur, *pold = (st & 1) ? F.pcur : F.pold;
        float *mcur = (st & 1) ? F.mold : F.mcur, *mold = (st & 1) ? F.mcur : F.mold;
        const long it = it0 + st;
        each([&](const Pair &c) { pass1<PHYS>(g, F, S, pcur, mcur, c); });
        if (!grid_barrier(sync_words, gen, &ok_flag)) return;
        each([&](const Pair &c) { pass2<PHYS>(g, F, S, pcur, pold, mcur, mold, c, st == nsteps - 1); });
        if (n_inj && it >= 1 && it <= F.inj.nt) {
            // the step's source injection into the new field, each group's contributions in order, separate
            // IEEE multiply and add
            __syncthreads();
            for (int i = threadIdx.x; i < n_inj; i += NT) {
                const int gi = inj[i];
                float acc = pold[F.inj.key[gi]];
                for (long j = F.inj.start[gi]; j < F.inj.start[gi + 1]; j++)
                    acc = __fadd_rn(acc, __fmul_rn(F.inj.c[j], F.inj.wav[F.inj.other[j] * F.inj.nt + (it - 1)]));
                pold[F.inj.key[gi]] = acc;
            }
        }
        if (!grid_barrier(sync_words, gen, &ok_flag)) return;
        if (ex.ngroups && it >= 1 && it <= ex.nt) {
            // data[key*nt + it-1] += sum c * new field[other], each group in order, IEEE multiply and add
            for (long gi = (long)blockIdx.x + (long)threadIdx.x * gridDim.x; gi < ex.ngroups; gi += (long)gridDim.x * NT) {
                float *dst = ex.data + ex.key[gi] * ex.nt + (it - 1);
                float acc = *dst;
                for (long j = ex.start[gi]; j < ex.start[gi + 1]; j++)
                    acc = __fadd_rn(acc, __fmul_rn(ex.c[j], pold[ex.other[j]]));
                *dst = acc;
            }
        }
    }
}

template <int PHYS>
int launch(const Grid &g, const Fields &F, const Scratch &S, long nsteps, long it0, const RunExtract &ex,
           unsigned *sync_words, cudaStream_t s) {
    int dev = 0, sms = 0, per = 0, coop = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_loop2d<PHYS>, NT, 0);
    if (!coop || per < 1) return -1;
    const long tiles = ((g.nz + TZ - 1) / TZ) * ((g.nx + TX - 1) / TX), cap = (long)sms * per;
    Grid gg = g;
    Fields FF = F;
    Scratch SS = S;
    long ns = nsteps, i0 = it0;
    RunExtract ee = ex;
    unsigned *sw = sync_words;
    void *args[] = {&gg, &FF, &SS, &ns, &i0, &ee, &sw};
    return cudaLaunchCooperativeKernel((const void *)k_loop2d<PHYS>, dim3((unsigned)(tiles < cap ? tiles : cap)),
                                       dim3(NT), args, 0, s) == cudaSuccess
               ? 0
               : 1;
}

}  // namespace

int loop2d_run(const Grid &g, int phys, const Fields &F, const Scratch &S, long nsteps, long it0, const RunExtract &ex,
               unsigned *sync_words, cudaStream_t s) {
    if (g.ndim != 2 || F.inj.ngroups > MAX_INJ || g.n >= (1L << 31)) return -1;
    if (phys == ISO) return launch<ISO>(g, F, S, nsteps, it0, ex, sync_words, s);
    if (phys == VTI) return launch<VTI>(g, F, S, nsteps, it0, ex, sync_words, s);
    return launch<TTI>(g, F, S, nsteps, it0, ex, sync_words, s);
}
#endif

}  // namespace WFD_NS
