// sifv_sweep_api.h -- host entry points and argument block of the fused
// sweep path, shared by the C ABI translation unit and the sweep
// translation unit.
#pragma once

#include <cuda_runtime.h>

#include "sifv_device.cuh"

namespace sifv {

// EOS constants of the single-phase face flux.
struct FluxConsts {
    double gamma, pInf, invGm1, gPinf;
};

// Stage update of one interior cell from its complete flux divergence
// (src/ExplicitSolver.cpp:127-188) as U = a1 U + a2 U0 + a3 dt R with
// (a1, a2, a3) = (c1, c2, c3) / c4; dt is read from device memory.
struct RKUpdate {
    double a1, a2, a3;
    int save;     // stage 0 of a multi-stage scheme: back up U into U0
    int useU0;
};

struct SweepArgs {
    Params P;
    Fields F;
    const Ctl* ctl;
    FluxConsts C;
    RKUpdate K;
    double eps;
    int seg;       // cells per thread segment (line sweeps)
    int segx;      // cells per warp segment of a row (x sweep), 32 m - 2
    double* rhs[5];  // FP64 rhs buffer (rho, rhoU, rhoV, rhoW, rhoE)
    double* rhoP;    // stage primitive density: the conservative rho is updated in place by the
                     // last sweep while neighbouring stencils still need the stage-start value
    const double* inv[3];   // 1 / d per cell (ghosts included)
};

// One RK stage of the 2D explicit step as one fused kernel
// (sifv_march2d.cuh): U' = a1 in + a2 u0 + a3 dt R(in), written to `out`
// (which may be u0, never `in`); `last` also writes the primitives of U'.
struct TileArgs {
    Params P;
    FluxConsts C;
    double eps;
    Ctl* ctl;
    const double* in[4];    // stage input: rho, rhoU, rhoV, rhoE
    const double* u0[4];    // step-start state (own cells), null when a2 == 0
    double* out[4];         // stage output
    double a1, a2, a3;
    const double* inv[2];   // 1 / dx, 1 / dy per cell (ghosts included)
    int last;               // write the primitives of the new state
    double *velU, *velV, *pres;
    int strips, segs, segRows;   // work units: strips of 30 columns x segments of segRows rows (set by the launcher)
    int unitScale;               // work units per resident warp (autotuned; 0 or 1: one)
    // last stage: fold the acoustic dt of the new state (k_dt_acoustic's
    // expressions) into ctl->dtBits for the next step
    int dtNext;
    double cfl;
    const double *dx, *dy;      // cell widths (ghosts included)
};

// Planes per segment of a kernel whose blocks walk tiles of the x-y plane along
// z, `slots` blocks at a time: a segment costs its planes and about three
// planes' worth of start-up, and the blocks run in waves; the count with the
// shortest sum (down to one plane: a small mesh is one wave, as long as its
// longest walk).  Up to 64 segments are tried one by one, beyond them (a few
// tiles and many planes) the most that 1 to 16 waves hold: with 64 at most, a
// step of 4 x 4 x 4000 cells took 1050 us in FP64-fast against 340, a pressure
// iteration of 4 x 4 x 8000 59 us against 30.
inline int walk_planes(long long tiles, long long slots, int nz, long long* cost = nullptr) {
    int planes = nz;
    long long best = -1;
    auto consider = [&](long long segs) {
        if (segs < 1 || segs > nz) return;
        const int n = (int)((nz + segs - 1) / segs);
        const long long waves = (tiles * ((nz + n - 1) / n) + slots - 1) / slots;
        if (best < 0 || waves * (n + 3) < best) {
            best = waves * (n + 3);
            planes = n;
        }
    };
    for (int s = 1; s <= 64; ++s) consider(s);
    for (int w = 1; w <= 16; ++w) consider(w * slots / tiles);
    if (cost) *cost = best;
    return planes;
}

// One RK stage of the 3D explicit step as one fused kernel
// (sifv_tile3d.cuh), as TileArgs.
struct Tile3Args {
    Params P;
    FluxConsts C;
    double eps;
    Ctl* ctl;
    const double* in[5];    // stage input: rho, rhoU, rhoV, rhoW, rhoE
    const double* u0[5];    // step-start state (own cells), null when a2 == 0
    double* out[5];         // stage output (u0 or scratch, never `in`)
    double a1, a2, a3;
    const double* inv[3];   // 1 / d per cell (ghosts included)
    const double *dx, *dy, *dz;
    int last;               // write the primitives of the new state
    int dtNext;             // ... and fold its acoustic dt into ctl->dtBits
    double cfl;
    double *velU, *velV, *velW, *pres;
    int tilesX, tilesY, segs, segPlanes;   // set by the launcher
};

// Called after each kernel launch with the kernel family's name (per-kernel
// timing); may be null.
typedef void (*LaunchMark)(void* user, const char* family);

// One RK stage of the 1D or 3D explicit step on the fused sweep kernels
// (mixed: FP32 reconstruction / Riemann bulk).  Returns 0 on success.
int sweep_stage(SweepArgs A, cudaStream_t s, bool mixed, int& launches, LaunchMark mark = nullptr,
                void* user = nullptr);

int tile2d_stage(const TileArgs& A, cudaStream_t s, bool mixed, int& launches, LaunchMark mark = nullptr,
                 void* user = nullptr);
// Whether the 3D step takes less time with the sweeps than with k_tile3d.
bool sweeps_3d(const Params& P, bool mixed, int sms);
int tile3d_stage(const Tile3Args& A, cudaStream_t s, bool mixed, int& launches, LaunchMark mark = nullptr,
                 void* user = nullptr);
// out[q] = in[q] over n values (2D) or the interior cells (3D), skipped when the step is (device-side loops).
int tile2d_copy(const Ctl* ctl, const double* const in[4], double* const out[4], size_t n, cudaStream_t s,
                int& launches);
int tile3d_copy(const Params& P, const Ctl* ctl, const double* const in[5], double* const out[5], cudaStream_t s,
                int& launches);

// End-of-step conservative -> primitive on interior cells.
int sweep_finish_prim(const Params& P, const Fields& F, const Ctl* ctl, cudaStream_t s, int& launches);

}  // namespace sifv
