// Mixed-precision DEM contact kernel: the shared contact kernel template
// instantiated with FP64 overlaps, FP32 contact laws and FP64 accumulation
// (compiled with FMA contraction, unlike the FP64 kernels).
#include "dem_device.cuh"
#include "contacts_staged.cuh"
#include "contact_launch.cuh"
#include "dem_launch.h"
#include "engine_internal.h"

namespace sphb {

cudaError_t launch_contacts_mixed(const DevParams &P, const DevState &S, cudaStream_t st,
                                  int staged)
{
    if (P.np == 0) return cudaSuccess;
    if (P.contactmodel == 2 && staged) {
        size_t smem;
        unsigned cap;
        staged_contact_shape(P.nc, stage_bytes_per_particle<2>(), smem, cap);
        static size_t attr = 0;
        if (attr < smem) {
            cudaFuncSetAttribute(k_contacts_staged<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem);
            attr = smem;
        }
        dim3 grid((P.np + SPHB_STAGED_B - 1) / SPHB_STAGED_B);
        k_contacts_staged<2><<<grid, SPHB_STAGED_B, smem, st>>>(P, S, cap);
        return cudaGetLastError();
    }
    return P.contactmodel == 2 ? launch_contact_kernel<2, 2>(k_contacts<2, 2>, P, S, st)
                               : launch_contact_kernel<2, 1>(k_contacts<2, 1>, P, S, st);
}

template <int MODEL>
static cudaError_t launch_ci(const DevParams &P, const DevState &S, cudaStream_t st)
{
    return P.nb0 ? launch_contact_kernel<2, MODEL>(k_contacts_integrate<2, MODEL, true>, P, S, st)
                 : launch_contact_kernel<2, MODEL>(k_contacts_integrate<2, MODEL, false>, P, S, st);
}

cudaError_t launch_contacts_integrate_mixed(const DevParams &P, const DevState &S, cudaStream_t st)
{
    return P.contactmodel == 2 ? launch_ci<2>(P, S, st) : launch_ci<1>(P, S, st);
}

const void *step_kernel_mixed(int model)
{
    return model == 2 ? (const void *)k_step<2, 2> : (const void *)k_step<2, 1>;
}
size_t step_smem_mixed(int model, unsigned nc)
{
    return (SPHB_CONTACT_B / 32) * (model == 2 ? contact_warp_bytes<2, 2>(nc) : contact_warp_bytes<2, 1>(nc));
}

int Engine::mixed_init() { return ST_OK; }

}  // namespace sphb
