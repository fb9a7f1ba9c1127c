// Wavefield-separation imaging condition (prop3DAcoIsoDenQ_DEO2_FDTD.h:673-765; VTI
// prop3DAcoVTIDenQ_DEO2_FDTD.h:606-725; TTI prop3DAcoTTIDenQ_DEO2_FDTD.h:609-728; 2D Iso
// prop2DAcoIsoDenQ_DEO2_FDTD.h:584-672), with a hand-written batched column FFT.
//
// The reference, per (x,y) column and per field: zero-pad the column to n = 2nz, transform, zero half
// of the bins, transform back, and accumulate 2B/V^3 * Re(a*b), where a keeps bins 0..nz of the
// forward field and b bins 0..nz (RTM) or 0 and nz..n-1 (FWI) of the adjoint field. Summing the kept
// bins in closed form (only the first nz inputs are nonzero and only the first nz outputs are used)
// leaves, for a column x,
//   Re a_j = x_j / 2 + (1/n) sum of x_m over the m of j's parity
//   Im a_j = -(H x)_j,  (H x)_j = (1/n) sum over odd d = j - m of cot(pi d / n) x_m
// and for the FWI filter the complex conjugate of that, so
//   Re(a b) = Re a Re b - Hx Hy (RTM), + Hx Hy (FWI).
// H is a real Toeplitz operator that takes the odd cells to the even ones and back, so the column's
// even cells and its odd cells are each one circular convolution of length L = the power of two >= nz,
// and a field pair (x, y) goes through it as the complex column x + iy: 2 forward and 2 inverse
// transforms of length L a field pair, where transforming each padded column by itself took 16 of
// length >= 4nz - 1 (Bluestein's algorithm, which any nz that is not a power of two needed). x and y
// may differ by orders of magnitude (a saved V^2/B-scaled derivative against a pressure), and a
// transform rounds relative to the larger of the two it carries, so each is first brought to a maximum
// of about 1 by a power of two of its own: without that the result was 1.7e-6 off (relative L2
// against float64) at 40:1, with it 1.8e-7 at any ratio (Bluestein transforms of each column: 3.3e-7).
//
// One thread holds 8 points of both transforms (u: odd cells, v: even cells), L/8 threads a column.
// Stages are radix 8 (the last one 2 or 4 when log2 L is no multiple of 3), decimation in frequency
// forward and in time back, in place in shared memory (one padded exchange between stages), so no
// reordering is needed and the product with the transformed operator happens in registers. Each
// persistent CTA forms the twiddles and the transformed operator itself, once, in shared memory: no
// tables in global memory, so calls on any streams and of any nz share nothing.
//
// Bound by shared-memory traffic and FP32 issue (about 90 kflop a column at nz = 300), not by the
// 24 B/cell that have to move: l1tex 63 %, issue 51 % busy. A whole call (3D Iso, 160 x 128 x 300 cells, nz no power of two): 151 us;
// one CTA a column with radix-2 stages and sincospif twiddles took 5580 us.
#include "wfd_kernels.h"

namespace WFD_NS {
using namespace wfd;

namespace {

__device__ __forceinline__ float2 add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {  // a * conj(b)
    return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
// a * (S i)
template <int S>
__device__ __forceinline__ float2 muli(float2 a) {
    return S > 0 ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

// X_k = sum_r a_r e^{S 2 pi i r k / N}, natural order in and out
template <int S>
__device__ __forceinline__ void dft4(float2 &a0, float2 &a1, float2 &a2, float2 &a3) {
    const float2 s0 = add(a0, a2), d0 = sub(a0, a2), s1 = add(a1, a3), d1 = muli<S>(sub(a1, a3));
    a0 = add(s0, s1);
    a1 = add(d0, d1);
    a2 = sub(s0, s1);
    a3 = sub(d0, d1);
}
// HALF: a[4..7] are zero
template <int S, bool HALF>
__device__ __forceinline__ void dft8(float2 (&a)[8]) {
    constexpr float h = 0.70710678118654752f;
    float2 b[8];
#pragma unroll
    for (int r = 0; r < 4; r++) {
        b[r] = HALF ? a[r] : add(a[r], a[r + 4]);
        b[r + 4] = HALF ? a[r] : sub(a[r], a[r + 4]);
    }
    b[5] = make_float2(h * (b[5].x - S * b[5].y), h * (b[5].y + S * b[5].x));
    b[6] = muli<S>(b[6]);
    b[7] = make_float2(h * (-b[7].x - S * b[7].y), h * (-b[7].y + S * b[7].x));
    dft4<S>(b[0], b[1], b[2], b[3]);
    dft4<S>(b[4], b[5], b[6], b[7]);
#pragma unroll
    for (int r = 0; r < 4; r++) {
        a[2 * r] = b[r];
        a[2 * r + 1] = b[r + 4];
    }
}

template <int K>
struct Sep {
    static constexpr int L = 1 << K;           // transform length
    static constexpr int T = L / 8;            // threads of a column
    static constexpr int NT = T > 256 ? T : 256;
    static constexpr int CPB = NT / T;         // columns at a time
    static constexpr int NS = K / 3;           // radix-8 stages
    static constexpr int REM = 1 << (K % 3);   // radix of the last stage, 1: none
    static constexpr int BUF = L + T;          // floats2 of one padded transform
    static constexpr bool BIG = K == 13;       // no room for all tables: formed as they are used
    // shared memory (float2): transforms, operator (v, u), twiddles, DC values
    static constexpr int O_G = 2 * CPB * BUF;
    static constexpr int O_W = O_G + (BIG ? 1 : 2) * L;
    static constexpr int O_DC = O_W + (BIG ? 0 : L);
    static constexpr int O_MAX = O_DC + 2 * CPB;  // a warp's largest |x| and |y|
    static constexpr size_t SMEM = sizeof(float2) * (size_t)(O_MAX + NT / 32);
    static_assert(SMEM <= 227 * 1024, "shared memory of a CTA");

    // length of the sub-transforms of stage s, and where its twiddles start: w[(r-1) M/8 + q] for
    // e^{-2 pi i q r / M}
    static constexpr int M(int s) { return L >> (3 * s); }
    static constexpr int woff(int s) { return s == 0 ? 0 : woff(s - 1) + 7 * (M(s - 1) / 8); }

    static __device__ __forceinline__ int pad(int i) { return i + (i >> 3); }

    template <int ST>
    static __device__ __forceinline__ float2 twiddle(const float2 *w, int q, int r) {
        if (!BIG) return w[woff(ST) + (r - 1) * (M(ST) / 8) + q];
        float s, c;
        sincospif(-2.0f * (float)(q * r) / (float)M(ST), &s, &c);
        return make_float2(c, s);
    }

    // position of element r of this thread's butterfly in stage ST
    template <int ST>
    static __device__ __forceinline__ int pos(int t, int r) {
        constexpr int P = M(ST) / 8;
        return pad((t / P) * M(ST) + t % P + r * P);
    }

    template <bool V>
    static __device__ __forceinline__ void rem(float2 (&a)[8]) {
        constexpr int S = V ? 1 : -1;
        if (REM == 4) {
            dft4<S>(a[0], a[1], a[2], a[3]);
            dft4<S>(a[4], a[5], a[6], a[7]);
        } else if (REM == 2) {
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
                const float2 x = a[e], y = a[e + 1];
                a[e] = add(x, y);
                a[e + 1] = sub(x, y);
            }
        }
    }

    // both transforms forward from stage ST (inputs in registers); afterwards register e holds
    // position 8t + e
    template <int ST, bool HALF>
    static __device__ __forceinline__ void forward(float2 (&u)[8], float2 (&v)[8], float2 *bu, float2 *bv,
                                                   const float2 *w, int t) {
        if constexpr (ST < NS) {
            dft8<-1, HALF>(u);
            dft8<-1, HALF>(v);
            constexpr int P = M(ST) / 8;
            if constexpr (P > 1) {
                const int q = t % P;
#pragma unroll
                for (int r = 1; r < 8; r++) {
                    const float2 z = twiddle<ST>(w, q, r);
                    u[r] = cmul(u[r], z);
                    v[r] = cmul(v[r], z);
                }
                exchange<ST, ST + 1>(u, v, bu, bv, t);
                forward<ST + 1, false>(u, v, bu, bv, w, t);
            }
        } else {
            rem<false>(u);
            rem<false>(v);
        }
    }

    // back, from the registers forward() leaves to those it was given
    template <int ST>
    static __device__ __forceinline__ void inverse(float2 (&u)[8], float2 (&v)[8], float2 *bu, float2 *bv,
                                                   const float2 *w, int t) {
        if constexpr (ST == NS) {
            rem<true>(u);
            rem<true>(v);
            if constexpr (REM > 1) exchange<NS, NS - 1>(u, v, bu, bv, t);
            inverse<NS - 1>(u, v, bu, bv, w, t);
        } else {
            constexpr int P = M(ST) / 8;
            if constexpr (P > 1) {
                const int q = t % P;
#pragma unroll
                for (int r = 1; r < 8; r++) {
                    const float2 z = twiddle<ST>(w, q, r);
                    u[r] = cmulc(u[r], z);
                    v[r] = cmulc(v[r], z);
                }
            }
            dft8<1, false>(u);
            dft8<1, false>(v);
            if constexpr (ST > 0) {
                exchange<ST, ST - 1>(u, v, bu, bv, t);
                inverse<ST - 1>(u, v, bu, bv, w, t);
            }
        }
    }

    // stage FROM's outputs to the threads that need them in stage TO (in place; stage NS holds 8
    // consecutive positions a thread)
    template <int FROM, int TO>
    static __device__ __forceinline__ void exchange(float2 (&u)[8], float2 (&v)[8], float2 *bu, float2 *bv, int t) {
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const int i = slot<FROM>(t, r);
            bu[i] = u[r];
            bv[i] = v[r];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const int i = slot<TO>(t, r);
            u[r] = bu[i];
            v[r] = bv[i];
        }
    }
    template <int ST>
    static __device__ __forceinline__ int slot(int t, int r) {
        if constexpr (ST < NS) return pos<ST>(t, r);
        else return pad(8 * t + r);
    }

    // frequency that forward() leaves at position p
    static __device__ __forceinline__ int freq(int p) {
        int f = 0, mul = 1;
        for (int m = L; m > REM; m >>= 3) {
            f += (p / (m / 8)) * mul;
            p %= m / 8;
            mul *= 8;
        }
        return f + p * mul;
    }

    // biased exponents of the column's largest |x| and |y| (1..253; 127 when it is not finite)
    static __device__ __forceinline__ uint2 exponents(uint2 mx, uint2 *buf, int slot, int t) {
        if constexpr (T >= 32) {
            mx.x = __reduce_max_sync(0xffffffffu, mx.x);
            mx.y = __reduce_max_sync(0xffffffffu, mx.y);
            if constexpr (T > 32) {
                if (t % 32 == 0) buf[(slot * T + t) / 32] = mx;
                __syncthreads();
                for (int i = 0; i < T / 32; i++) {
                    const uint2 o = buf[slot * (T / 32) + i];
                    mx.x = max(mx.x, o.x);
                    mx.y = max(mx.y, o.y);
                }
            }
        } else {
            for (int o = T / 2; o > 0; o >>= 1) {
                mx.x = max(mx.x, __shfl_xor_sync(0xffffffffu, mx.x, o));
                mx.y = max(mx.y, __shfl_xor_sync(0xffffffffu, mx.y, o));
            }
        }
        auto e = [](unsigned m) { return m >= 0x7f800000u ? 127u : min(max(m >> 23, 1u), 253u); };
        return make_uint2(e(mx.x), e(mx.y));
    }

    // (1/L) cot(pi d / n) for the odd d that a column of nz cells reaches, else 0
    static __device__ __forceinline__ float tap(int d, int nz) {
        if (d >= nz || d <= -nz) return 0.0f;
        double s, c;
        sincospi((double)d / (2.0 * nz), &s, &c);
        return (float)(c / s / L);
    }
};

template <int K>
__global__ void __launch_bounds__(Sep<K>::NT, Sep<K>::NT > 256 ? 1 : 3)
    k_wavefieldsep(long ncols, int nz, int isfwi, const float *__restrict__ v_, const float *__restrict__ b_,
                   const float *__restrict__ pold, const float *__restrict__ mold, const float *__restrict__ dp,
                   const float *__restrict__ dm, float *__restrict__ dv) {
    using C = Sep<K>;
    constexpr int T = C::T, L = C::L;
    extern __shared__ float2 sm[];
    const int slot = threadIdx.x / T, t = threadIdx.x % T;
    float2 *bu = sm + (2 * slot) * C::BUF, *bv = bu + C::BUF;
    float2 *G = sm + C::O_G, *W = sm + C::O_W, *dc = sm + C::O_DC + 2 * slot;

    // Twiddles, then the operator's taps through the same transform. The taps are formed by all threads together (a
    // cotangent in double is long, and a CTA of several columns would form each one several times).
    if (!C::BIG) {
        for (int i = threadIdx.x; i < L; i += C::NT) {
            int m = L, o = i;  // stage length and offset inside the stage
            while (m >= 8 && o >= 7 * (m / 8)) {
                o -= 7 * (m / 8);
                m >>= 3;
            }
            if (m >= 8) {
                const int r = o / (m / 8) + 1, q = o % (m / 8);
                double s, c;
                sincospi(-2.0 * (q * r) / m, &s, &c);
                W[i] = make_float2((float)c, (float)s);
            }
        }
    }
    {
        float *taps = reinterpret_cast<float *>(G);
        for (int i = threadIdx.x; i < L; i += C::NT) taps[i] = C::tap(2 * (i < L / 2 ? i : i - L) + 1, nz);
        __syncthreads();
        float2 u[8], v[8];
#pragma unroll
        for (int r = 0; r < 8; r++) {  // v: distance 2i + 1 (i from -L/2 to L/2 - 1), u: 2i - 1
            const int i = t + r * T;
            v[r] = make_float2(taps[i], 0.0f);
            u[r] = make_float2(i == L / 2 ? 0.0f : taps[(i + L - 1) % L], 0.0f);
        }
        C::template forward<0, false>(u, v, bu, bv, W, t);
        if (slot == 0) {
#pragma unroll
            for (int e = 0; e < 8; e++) {
                G[e * T + t] = v[e];
                if (!C::BIG) G[L + e * T + t] = u[e];
            }
        }
        __syncthreads();
    }

    const float scale = 1.0f / (float)(2 * nz);  // the reference rounds its scaled inputs: so here
    const double sign = isfwi ? 1.0 : -1.0;
    uint2 *red = reinterpret_cast<uint2 *>(sm + C::O_MAX);
    const long ngroups = (ncols + C::CPB - 1) / C::CPB;
    for (long cg = blockIdx.x; cg < ngroups; cg += gridDim.x) {
        const long col = cg * C::CPB + slot;
        const bool live = col < ncols;
        const long base = col * nz;
        // cells 2i and 2i + 1, i = t + r T; the sum and the image's increment in double, so that only
        // the transforms' rounding is left in it
        double acc[4][2];
#pragma unroll
        for (int r = 0; r < 4; r++) acc[r][0] = acc[r][1] = 0.0;
        const int nfield = dm ? 2 : 1;
        for (int fld = 0; fld < nfield; fld++) {
            const float *x = (fld == 0 ? dp : dm) + base, *y = (fld == 0 ? pold : mold) + base;
            float2 u[8], v[8];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const int j = 2 * (t + r * T);
                const bool in0 = live && j < nz, in1 = live && j + 1 < nz;
                v[r] = make_float2(in0 ? scale * x[j] : 0.0f, in0 ? scale * y[j] : 0.0f);
                u[r] = make_float2(in1 ? scale * x[j + 1] : 0.0f, in1 ? scale * y[j + 1] : 0.0f);
                v[r + 4] = u[r + 4] = make_float2(0.0f, 0.0f);
            }
            uint2 mx = make_uint2(0u, 0u);
#pragma unroll
            for (int r = 0; r < 4; r++) {
                mx.x = max(mx.x, max(__float_as_uint(fabsf(u[r].x)), __float_as_uint(fabsf(v[r].x))));
                mx.y = max(mx.y, max(__float_as_uint(fabsf(u[r].y)), __float_as_uint(fabsf(v[r].y))));
            }
            const uint2 ex = C::exponents(mx, red, slot, t);
            const float2 norm = make_float2(__uint_as_float((254u - ex.x) << 23), __uint_as_float((254u - ex.y) << 23));
#pragma unroll
            for (int r = 0; r < 4; r++) {
                u[r] = make_float2(u[r].x * norm.x, u[r].y * norm.y);
                v[r] = make_float2(v[r].x * norm.x, v[r].y * norm.y);
            }
            C::template forward<0, true>(u, v, bu, bv, W, t);
            if (t == 0) {
                dc[0] = v[0];
                dc[1] = u[0];
            }
#pragma unroll
            for (int e = 0; e < 8; e++) {
                const float2 gv = G[e * T + t];
                float2 gu;
                if (!C::BIG) {
                    gu = G[L + e * T + t];
                } else {  // the u taps are the v taps one place on
                    float s, c;
                    sincospif(-2.0f * (float)C::freq(8 * t + e) / (float)L, &s, &c);
                    gu = cmul(gv, make_float2(c, s));
                }
                v[e] = cmul(v[e], gv);
                u[e] = cmul(u[e], gu);
            }
            C::template inverse<(C::REM > 1 ? C::NS : C::NS - 1)>(u, v, bu, bv, W, t);
            const float2 s0 = dc[0], s1 = dc[1];
            // 2^e of the two normalisations, and Re a Re b -+ Hx Hy of one cell
            const double ux = __hiloint2double((int)(ex.x + 896u) << 20, 0), uy = __hiloint2double((int)(ex.y + 896u) << 20, 0);
            auto term = [&](float x, float y, float2 sum, float2 h) {
                return ((double)nz * (scale * x) + ux * sum.x) * ((double)nz * (scale * y) + uy * sum.y) +
                       sign * (ux * h.x) * (uy * h.y);
            };
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const int j = 2 * (t + r * T);
                if (live && j < nz)  // even cells: H of the odd ones (u)
                    acc[r][0] += term(x[j], y[j], s0, u[r]);
                if (live && j + 1 < nz) acc[r][1] += term(x[j + 1], y[j + 1], s1, v[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int j = 2 * (t + r * T) + h;
                if (live && j < nz) {
                    const long k = base + j;
                    const double V = v_[k];
                    const double B = b_[k];
                    dv[k] = (float)((double)dv[k] + 2 * B / (V * V * V) * acc[r][h]);
                }
            }
    }
}

template <int K>
bool launch(const Grid &g, long isfwi, const Fields &F, const float *dp, const float *dm, float *dv, cudaStream_t s) {
    using C = Sep<K>;
    const long ncols = g.nx * g.ny;
    static PerDevice<int> caps;
    int &cap = caps.here();
    if (!cap) {
        if (cudaFuncSetAttribute(k_wavefieldsep<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM) != cudaSuccess)
            return false;
        int dev = 0, sms = 0, per = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_wavefieldsep<K>, C::NT, C::SMEM) != cudaSuccess || per < 1)
            return false;
        cap = sms * per;
    }
    const long groups = (ncols + C::CPB - 1) / C::CPB;
    k_wavefieldsep<K><<<(unsigned)(groups < cap ? groups : cap), C::NT, C::SMEM, s>>>(
        ncols, (int)g.nz, isfwi ? 1 : 0, F.v, F.b, F.pold, F.mold, dp, dm, dv);
    return true;
}

}  // namespace

bool image_wavefieldsep(const Grid &g, long isfwi, const Fields &F, const float *dp, const float *dm, float *dv,
                        cudaStream_t s) {
    int k = 4;
    while (k < 14 && (1L << k) < g.nz + (g.nz & 1)) k++;
    switch (k) {
        case 4: return launch<4>(g, isfwi, F, dp, dm, dv, s);
        case 5: return launch<5>(g, isfwi, F, dp, dm, dv, s);
        case 6: return launch<6>(g, isfwi, F, dp, dm, dv, s);
        case 7: return launch<7>(g, isfwi, F, dp, dm, dv, s);
        case 8: return launch<8>(g, isfwi, F, dp, dm, dv, s);
        case 9: return launch<9>(g, isfwi, F, dp, dm, dv, s);
        case 10: return launch<10>(g, isfwi, F, dp, dm, dv, s);
        case 11: return launch<11>(g, isfwi, F, dp, dm, dv, s);
        case 12: return launch<12>(g, isfwi, F, dp, dm, dv, s);
        case 13: return launch<13>(g, isfwi, F, dp, dm, dv, s);
        default: return false;  // deeper than 8192 cells: no CTA's shared memory holds a column
    }
}

}  // namespace WFD_NS
