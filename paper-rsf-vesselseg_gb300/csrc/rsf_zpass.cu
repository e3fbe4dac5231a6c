// rsf_zpass.cu -- z-pass (local fits and data factor) for one tap count
// (compiled once per -DRSF_K value; RSF_K = 0 is the run-time-k kernel, which
// also writes the debug fields).
#include "rsf_kernels.cuh"

#ifndef RSF_K
#error "compile with -DRSF_K=<taps>"
#endif
#define RSF_CAT2(a, b) a##b
#define RSF_CAT(a, b) RSF_CAT2(a, b)

namespace rsf {

cudaError_t RSF_CAT(launch_zpass_, RSF_K)(const SubVolDev *svs, const int *pre, int blocks, const StepConst &c,
                                          const DebugOut *dbg, cudaStream_t st) {
#if RSF_K > 0
    (void)dbg;
    return launch_dependent(true, zpass_kernel<RSF_K>, (unsigned)blocks, ZP_COLS, zpass_smem(RSF_K), st, svs, pre, c);
#else
    const DebugOut d = dbg ? *dbg : DebugOut{nullptr, 0};
    return launch_dependent(true, dbg ? zpass_chunk_kernel<true> : zpass_chunk_kernel<false>, (unsigned)blocks, ZP_COLS, 0, st,
                            svs, pre, c, d);
#endif
}

cudaError_t RSF_CAT(config_zpass_, RSF_K)() {
    cudaError_t e = cudaSuccess;
#if RSF_K > 0
    e = cudaFuncSetAttribute(zpass_kernel<RSF_K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)zpass_smem(RSF_K));
    if (e == cudaSuccess) e = RSF_CAT(config_zpass_adjoint_, RSF_K)();
#endif
    return e;
}

}  // namespace rsf
