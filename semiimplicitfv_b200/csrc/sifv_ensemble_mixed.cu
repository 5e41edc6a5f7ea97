// sifv_ensemble_mixed.cu -- the FP32-bulk instantiation of the ensemble
// kernel, compiled with FMA contraction and the approximate single-precision
// division / square root of --use_fast_math (FP64 arithmetic is unaffected;
// mixed precision is held to an L1 error bound, not to bit equality).
#include "sifv_ensemble.cuh"
#include "sifv_ensemble_api.h"

namespace sifv {

// The mixture pressure recovery from total energy (where pInf ~ 6e8
// cancels), the carried state and the update stay FP64 inside the kernel.
namespace {
template <int NPH>
int launch_f(const EnsArgs& A, int blockSize, cudaStream_t s) {
    k_ensemble<float, NPH, false><<<A.nInst, blockSize, 0, s>>>(A);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
}  // namespace

int ensemble_launch_mixed(const EnsArgs& A, int nph, int blockSize, cudaStream_t s) {
    if (nph == 0) return launch_f<0>(A, blockSize, s);
    if (nph == 2) return launch_f<2>(A, blockSize, s);
    return launch_f<8>(A, blockSize, s);
}

}  // namespace sifv
