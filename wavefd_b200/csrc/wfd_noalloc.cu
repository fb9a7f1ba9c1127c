// An entry point that allocates no memory: the wavefield-separation imaging condition
// (the AdjointBornAccumulation_wavefieldsep family) on caller-provided device arrays.
//
// Some callers cannot call cudaMalloc at all: code running under a memory pool or allocator that
// owns all device memory of the process, callers inside a region where allocation is not allowed
// (for example while other work holds the allocator), or plug-ins whose host application forbids
// device allocations by extensions. The regular entry points allocate staging buffers for host
// arrays. This variant requires every array it is given to be device or managed memory on the
// current device; the kernel itself needs no memory besides them (its tables are formed in shared
// memory), so calls on different streams are independent.
#include <math.h>
#include <stdlib.h>

#include "wfd_prop.h"

namespace {

constexpr long kMaxNz = 2048;  // largest nz accepted

int fail(const char *msg) {
    wfd::set_global_error(WFD_ERR_ARG, msg);
    return WFD_ERR_ARG;
}

}  // namespace

extern "C" int WFD_AdjointBornAccumulation_wavefieldsep_NoAlloc(long nx, long ny, long nz, long isFWI,
                                                                 const float *v, const float *b,
                                                                 const float *wavefieldDP, const float *pOld,
                                                                 const float *wavefieldDM, const float *mOld,
                                                                 float *dVel, void *stream) {
    if (nx < 1 || ny < 1 || nz < 1) return fail("wavefieldsep_NoAlloc: grid sizes must be positive");
    if (nz > kMaxNz) return fail("wavefieldsep_NoAlloc: nz exceeds the maximum of 2048");
    if (!v || !b || !wavefieldDP || !pOld || !dVel) return fail("wavefieldsep_NoAlloc: null array");
    if ((wavefieldDM == nullptr) != (mOld == nullptr))
        return fail("wavefieldsep_NoAlloc: wavefieldDM and mOld must be given together");
    const void *arrays[7] = {v, b, wavefieldDP, pOld, dVel, wavefieldDM, mOld};
    for (int i = 0; i < 7; i++)
        if (arrays[i] && !wfd::device_accessible(arrays[i]))
            return fail("wavefieldsep_NoAlloc: every array must be device or managed memory");
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) return fail("wavefieldsep_NoAlloc: no device");
    // the arrays must live on the current device
    cudaPointerAttributes attr{};
    if (cudaPointerGetAttributes(&attr, dVel) != cudaSuccess ||
        (attr.type == cudaMemoryTypeDevice && attr.device != dev))
        return fail("wavefieldsep_NoAlloc: the image is not on the current device");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    wfd::Grid g{};
    g.ndim = ny > 1 ? 3 : 2;
    g.nx = nx;
    g.ny = ny;
    g.nz = nz;
    g.sy = nz;
    g.sx = ny * nz;
    g.n = nx * ny * nz;
    wfd::Fields F{};
    F.v = const_cast<float *>(v);
    F.b = const_cast<float *>(b);
    F.pold = const_cast<float *>(pOld);
    F.mold = const_cast<float *>(mOld);
    // the bitwise-parity build when WAVEFD_B200_STRICT=1, as for new propagator objects
    const char *mode = getenv("WAVEFD_B200_STRICT");
    const bool ok = mode && mode[0] == '1'
                        ? wfd_strict::image_wavefieldsep(g, isFWI, F, wavefieldDP, wavefieldDM, dVel, s)
                        : wfd_fast::image_wavefieldsep(g, isFWI, F, wavefieldDP, wavefieldDM, dVel, s);
    const cudaError_t e = cudaGetLastError();
    if (!ok || e != cudaSuccess) {
        wfd::set_global_error(WFD_ERR_CUDA, std::string("wavefieldsep_NoAlloc launch: ") + cudaGetErrorString(e));
        return WFD_ERR_CUDA;
    }
    return WFD_OK;
}
