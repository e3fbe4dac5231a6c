// rsf_zadj.cu -- the z-pass with the adjoint's emit (the data-term adjoint instead
// of the data factor) for one specialised tap count (compiled once per
// -DRSF_K value, 0 for the run-time tap count; a unit of its own so that it
// compiles beside the z-pass).
#include "rsf_kernels.cuh"

#ifndef RSF_K
#error "compile with -DRSF_K=<taps>"
#endif
#define RSF_CAT2(a, b) a##b
#define RSF_CAT(a, b) RSF_CAT2(a, b)

namespace rsf {

#if RSF_K > 0
cudaError_t RSF_CAT(config_zpass_adjoint_, RSF_K)() {
    return cudaFuncSetAttribute(zpass_adjoint_kernel<RSF_K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)zpass_smem(RSF_K));
}
#endif

cudaError_t RSF_CAT(launch_zpass_adjoint_, RSF_K)(const SubVolDev *svs, const int *pre, int blocks,
                                                  const StepConst &c, const AdjVol *vols, cudaStream_t st) {
#if RSF_K > 0
    zpass_adjoint_kernel<RSF_K><<<blocks, ZP_COLS, zpass_smem(RSF_K), st>>>(svs, pre, c, vols);
#else
    zchunk_adjoint_kernel<ZG_NB><<<blocks, ZP_COLS, 0, st>>>(svs, pre, c, vols);
#endif
    return cudaGetLastError();
}

}  // namespace rsf
