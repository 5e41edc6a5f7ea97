// sifv_stage_api.h -- arguments and launchers of the fused reference-ordered
// stage kernel (sifv_stage.cuh), used by the C ABI translation unit.
#pragma once

#include <cuda_runtime.h>

#include "sifv_common.cuh"

namespace sifv {

// Ghost layers the stage kernel can refresh (sifv_create takes any number;
// more than this stays on the separate kernels).
constexpr int kStageMaxGhost = 8;

// One conservative state: rho, momenta, rhoE and the phases' partial
// densities and volume fractions (ghost layers are not read).
struct StageState {
    double *rho, *mom[3], *rhoE;
    double *alphaRho[2], *alpha[2];
};

struct StageArgs {
    Params P;
    Ctl* ctl;
    StageCoef K;
    StageState in, u0, out;   // stage input, step-start state, stage output (u0 or scratch, never `in`)
    double dtFixed;           // > 0: this dt instead of the control block's, whatever its skip flag
    int last;                 // last stage: write the primitives of the new state and its PRIM ghost layers
    int dtNext;               // ... and fold its time-step limits into ctl->dtBits
    double cfl;
    double *velU, *velV, *pres, *sigma;
    const double *dx, *dy, *dz;
};

// 1D and 2D, WENO5 / UPWIND5, at most two phases.  Returns 0 on success.
int stage_launch(const StageArgs& A, cudaStream_t s);

}  // namespace sifv
