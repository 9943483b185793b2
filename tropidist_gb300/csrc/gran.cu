// The granule pass's kernel (gran.cuh) and its launch.
#include "gran.cuh"
#include "tg_capi.h"

#include <algorithm>

namespace tg {

// One block of 2^GP_TB threads per step: a loop over steps makes the compiler keep the parameters in
// registers across it and spill (23 % slower), and narrow tables spread over more SMs this way.  6
// blocks (80 registers) against 4 or 5: 20.6 / 22.0 / 21.6 ms on the 31-bit sweep.
#define GP_TB 7
template <int EB>
__global__ void __launch_bounds__(1 << GP_TB, EB == 1 ? 6 : 8)
    k_gran_pass(const __grid_constant__ GranParams P, const uint32_t *__restrict__ in, uint32_t *__restrict__ out) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    gran_step<EB, GP_TB, true>(P, blockIdx.x, in, out);
}

int launch_gran(const GranParams &P, int eb, const void *in, void *out, cudaStream_t st) {
    const uint64_t nsteps = (P.ncosets + (1u << GP_TB) - 1) >> GP_TB;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)nsteps);
    cfg.blockDim = dim3(1 << GP_TB);
    cfg.stream = st;
    // programmatic dependent launch: this pass's blocks start while the previous pass drains
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const uint32_t *src = static_cast<const uint32_t *>(in);
    uint32_t *dst = static_cast<uint32_t *>(out);
    return cuda_check(eb == 1 ? cudaLaunchKernelEx(&cfg, k_gran_pass<1>, P, src, dst)
                              : cudaLaunchKernelEx(&cfg, k_gran_pass<2>, P, src, dst), "granule pass launch");
}

}  // namespace tg
