// rsf_stencil.cu -- the stencil / update kernel instantiations.
#include "rsf_stencil_pair.cuh"

namespace rsf {

cudaError_t launch_stencil(const SubVolDev *svs, const int *pre, int blocks, const StepConst &c, int parity,
                           int arith, bool dependent, unsigned *flag, const DebugOut *dbg, cudaStream_t st) {
    if (dbg) {
        constexpr int T = ST_WARPS * 32;
        if (arith == 1) stencil_debug_kernel<Arith::Reference><<<blocks, T, 0, st>>>(svs, pre, c, parity, flag, *dbg);
        else stencil_debug_kernel<Arith::Portable><<<blocks, T, 0, st>>>(svs, pre, c, parity, flag, *dbg);
    } else {
        constexpr int T = SP_WARPS * 32;
        return launch_dependent(dependent, arith == 1 ? stencil_pair_kernel<Arith::Reference> : stencil_pair_kernel<Arith::Portable>,
                                (unsigned)blocks, T, 0, st, svs, pre, c, parity, flag);
    }
    return cudaGetLastError();
}

cudaError_t launch_box(const SubVolDev *svs, const int *pre, int blocks, const StepConst &c, const DebugOut *dbg,
                       cudaStream_t st) {
    constexpr int T = ST_WARPS * 32;
    const dim3 grid((unsigned)blocks, (unsigned)((c.zc + BOX_Z - 1) / BOX_Z));
    if (dbg) box_kernel<true><<<grid, T, 0, st>>>(svs, pre, c, *dbg);
    else box_kernel<false><<<grid, T, 0, st>>>(svs, pre, c, DebugOut{nullptr, 0});
    return cudaGetLastError();
}

}  // namespace rsf
