// Tile staging for grids whose rows TMA cannot address (nz not a multiple of 4: row pitches that are
// no multiple of 16 bytes), for the TMA step kernel's own shared-memory layout and barriers.
//
// Every thread copies single floats with cp.async (4 bytes) and arrives on the group's mbarrier when
// its copies have landed. A warp takes whole rows: 32 columns at a time, then the columns beyond them
// of several rows together. There are no bounds checks: a box that reaches past the grid's sides
// reads whatever the flat address holds (a neighbouring row or plane, or the margin that
// propagator arrays of such grids are allocated with on both ends, field_margin()), because no cell
// that the reference computes uses a value from outside the grid and the kernels select, never
// multiply, the other cells away. With per-copy bounds tests and zero fill the 3D Iso step took 282
// us at 301 x 203 x 251, 180 us without.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "wfd_tma.cuh"

namespace wfd_dev {

__device__ __forceinline__ void cp_async4(uint32_t dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
// the barrier's arrival of this thread, once its copies so far have landed (the barrier counts every
// thread of the CTA)
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp_async_drain() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A box of W x H floats at (z0, y0) of a plane (the array at (x, 0, 0)), copied by NW warps.
template <int W, int H, int NW>
struct RaggedBox {
    static constexpr int TW = W - 32, RPT = TW ? 32 / TW : 1;  // columns beyond 32; rows of them at a time
    static_assert(TW >= 0 && TW <= 32 && (TW == 0 || 32 % TW == 0), "box width");
    static constexpr int FULL = (H + NW - 1) / NW;
    static constexpr int TAIL = TW ? ((H + RPT - 1) / RPT + NW - 1) / NW : 0;

    static __device__ __forceinline__ void load(float *dst, const float *plane, int z0, int y0, int nz, int warp,
                                                int lane) {
        const uint32_t d0 = smem_u32(dst + warp * W + lane);
        const float *s = plane + ((y0 + warp) * nz + z0 + lane);
        const long step = (long)NW * nz;
#pragma unroll
        for (int k = 0; k < FULL; k++, s += step)
            if (NW * k + NW <= H || warp + NW * k < H) cp_async4(d0 + 4u * NW * W * k, s);
        if constexpr (TAIL > 0) {
            const int r = warp * RPT + lane / TW, c = 32 + lane % TW;
            const uint32_t d1 = smem_u32(dst + r * W + c);
            const float *t = plane + ((y0 + r) * nz + z0 + c);
            const long tstep = step * RPT;
#pragma unroll
            for (int k = 0; k < TAIL; k++, t += tstep)
                if (NW * RPT * (k + 1) <= H || r + NW * RPT * k < H) cp_async4(d1 + 4u * NW * RPT * W * k, t);
        }
    }
};

}  // namespace wfd_dev
