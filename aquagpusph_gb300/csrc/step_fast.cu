// The step kernels compiled with -use_fast_math (FMA contraction,
// approximate division and square root): aqua::fast.  Same source as the
// exact kernels (step_kernels.cuh); results stay within the 1e-5 relative
// tolerance of the reference's per-step rates (tests/test_gpu_fast.py).
// The fast build also has the clustered 3-D sweep (sweep_cl.cuh).
#include "aqua_internal.cuh"
#include "kernels.cuh"

namespace aqua {
namespace fast {
#define AQUA_FAST_ARITH 1
#include "step_kernels.cuh"
#include "sweep_cl.cuh"
#undef AQUA_FAST_ARITH

// blocks of 8 warps, 3 per SM (shared memory, registers), 2,048 staged
// records per pass
constexpr int kClWarps = 8, kClRecords = 2048;

cudaError_t
launch_sweep_cl(const Consts& c, const StepArgs& a, unsigned grid,
                cudaStream_t s)
{
    if (a.N == 0)
        return cudaSuccess;
    if (a.N > kOctantMin)
        k_sweep_cl<kClWarps, kClRecords, 3, true>
            <<<grid, kClWarps * 32, sizeof(ClSmem<kClWarps, kClRecords, true>), s>>>(c, a);
    k_sweep_cl<kClWarps, kClRecords, 3, false>
        <<<grid, kClWarps * 32, sizeof(ClSmem<kClWarps, kClRecords, false>), s>>>(c, a);
    return cudaGetLastError();
}

cudaError_t
prepare_sweep_cl()
{
    const cudaError_t e =
        cudaFuncSetAttribute(k_sweep_cl<kClWarps, kClRecords, 3, true>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(ClSmem<kClWarps, kClRecords, true>));
    return e != cudaSuccess
               ? e
               : cudaFuncSetAttribute(k_sweep_cl<kClWarps, kClRecords, 3, false>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(ClSmem<kClWarps, kClRecords, false>));
}

}  // namespace fast
}  // namespace aqua
