// Launch of the per-stage contact kernels: particles per warp and scratch.
#pragma once

#include "dem_device.cuh"

namespace sphb {

template <int PREC, int MODEL>
inline cudaError_t launch_contact_kernel(void (*fn)(DevParams, DevState, unsigned), const DevParams &P,
                                         const DevState &S, cudaStream_t st)
{
    if (P.np == 0) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    constexpr unsigned warps = SPHB_CONTACT_B / 32;   // 64 slots: below the 48 KB of a plain launch
    static_assert(warps * contact_warp_bytes<PREC, MODEL>(64) <= 48 * 1024, "contact scratch");
    const unsigned pw = contact_pw(P.np, (unsigned)sms * SPHB_CONTACT_MINB * warps);
    const unsigned per_block = warps * pw;
    fn<<<(P.np + per_block - 1) / per_block, SPHB_CONTACT_B,
         warps * contact_warp_bytes<PREC, MODEL>(P.nc), st>>>(P, S, pw);
    return cudaGetLastError();
}

}  // namespace sphb
