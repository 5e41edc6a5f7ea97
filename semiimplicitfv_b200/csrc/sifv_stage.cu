// sifv_stage.cu -- launcher of the fused reference-ordered stage kernel.
#include "sifv_stage.cuh"

namespace sifv {

namespace {

template <int DIM, int NPH, int RS>
int launch(const StageArgs& A, cudaStream_t s) {
    using T = StageTile<DIM, NPH>;
    // per device, so set on each launch (a host-side table write)
    if (cudaFuncSetAttribute(k_stage<DIM, NPH, RS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::smem) !=
        cudaSuccess)
        return -1;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)((A.P.nx + T::TX - 1) / T::TX), (unsigned)((A.P.ny + T::TY - 1) / T::TY));
    lc.blockDim = dim3(T::threads);
    lc.dynamicSmemBytes = T::smem;
    lc.stream = s;
    lc.attrs = at;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, k_stage<DIM, NPH, RS>, A) == cudaSuccess ? 0 : -1;
}

template <int DIM, int NPH>
int launch_rs(const StageArgs& A, cudaStream_t s) {
    switch (A.P.riemann) {
        case SIFV_HLLC: return launch<DIM, NPH, SIFV_HLLC>(A, s);
        case SIFV_RUSANOV: return launch<DIM, NPH, SIFV_RUSANOV>(A, s);
        default: return launch<DIM, NPH, SIFV_LF>(A, s);
    }
}

}  // namespace

int stage_launch(const StageArgs& A, cudaStream_t s) {
    if (A.P.dim == 1) return A.P.nPh ? launch_rs<1, 2>(A, s) : launch_rs<1, 0>(A, s);
    return A.P.nPh ? launch_rs<2, 2>(A, s) : launch_rs<2, 0>(A, s);
}

}  // namespace sifv
