// sifv_ensemble.cuh -- batched ensembles of independent 1D problems of
// different sizes, advanced to a common end time in ONE kernel launch.
//
// One CTA owns one instance and runs that instance's whole time loop
// (the explicit step of ExplicitSolver::step, src/ExplicitSolver.cpp:68-203,
// with the targetDt = tEnd - t cap of the reference's time loop,
// src/RKTimeStepping.cpp:258-266): its own acoustic dt (block-wide minimum),
// then per SSP-RK stage its warps take strips of 26 cells in turn.  The 32
// lanes of a warp hold the strip and its three halo cells on either side:
// each lane converts its cell to primitives (ghosts through the PRIM ghost
// map, src/RectilinearMesh.cpp:498-524; FP64), reconstructs both face values
// of its cell from the neighbours' primitives (shuffles), solves the Riemann
// problem at its high face with the next lane's value, and updates its cell
// from its own and the previous lane's flux.  Warps of a stage share nothing:
// the block synchronises once per stage.  (Mixed precision, 400 tubes of 256
// to 4096 cells, 40 steps: 4.3 ms, where chunks of the whole block in shared
// memory took 14.7.)  With CHUNKS, FP64 only, the team that shares a halo is
// the block instead: blockDim - 6 cells at a time, values passed through
// shared memory between three barriers.  Of 32 lanes a strip leaves 6 to the
// halo, and FP64 arithmetic is the bound on long instances (20 % of it the
// halo's); the barriers are the price, and short instances leave more of a
// block idle than of a warp (ensemble_chunks, sifv_ensemble.cu).
// The stage input and output are different packed states (S[0] the state,
// S[1], S[2] scratch; the last stage writes S[0], which only the cell itself
// reads there as U0), so strips never see each other's updates.  The last
// stage also writes the primitives of the new state and folds its acoustic
// limit into the next step's dt.  Blocks never wait on each other, so
// instances of any size (and step count) retire independently; the host
// orders instances by cost (N^2) so the longest start first.  State arrays
// are packed per instance with ghosts, x fastest.
//
// T is the arithmetic of the reconstruction / Riemann bulk (double: the
// reference's operation order, bit-identical to the single-instance path;
// float: mixed precision).  Primitive recovery (including the mixture
// pressure from total energy), dt, the divergence and the update are FP64;
// in mixed precision their quotients are products with refined reciprocals
// (frcp, within 1 ulp) and with the phases' constants.
#pragma once

#include "sifv_common.cuh"
#include "sifv_fastmath.cuh"

namespace sifv {

struct EnsState {             // one packed conservative state
    double *rho, *rhoU, *rhoE;
    double* alphaRho[MAXPH];
    double* alpha[MAXPH];
};

struct EnsArgs {
    Params P;                 // per-instance values nx / nxT are set per block
    int nInst;
    const int* order;         // block -> instance (cost-sorted)
    const int* n;             // interior cells per instance
    const long long* off;     // packed cell offset per instance (ghosts included)
    EnsState S[3];            // S[0]: the state; S[1], S[2]: stage outputs
    double *velU, *pres;      // primitives of the state (rho: S[0].rho)
    const double* dx;         // packed cell widths (ghosts included)
    // per instance
    double* time;
    int* steps;
    double* lastDt;
    int* status;              // 0 ok, 1 the time step was not positive (state blew up)
    double cfl, maxDt, constDt, tEnd;
    int maxSteps;
    const int* stepLimit;     // per-instance step limit (autotuner probes), may be null
    double invGm1[MAXPH];     // 1 / (gamma - 1) and gamma pInf / (gamma - 1) of each phase
    double gPiGm1[MAXPH];
};

// std::min(dt, x) over a block, NaN ignored; result broadcast to all threads.
__device__ __forceinline__ double block_min_bcast(double v, double* sm) {
    if (!(v == v)) v = __longlong_as_double(0x7ff0000000000000LL);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = smin(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    __syncthreads();
    if (lane == 0) sm[w] = v;
    __syncthreads();
    if (w == 0) {
        v = (lane < nw) ? sm[lane] : __longlong_as_double(0x7ff0000000000000LL);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = smin(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) sm[32] = v;
    }
    __syncthreads();
    return sm[32];
}

// Largest block: 1024 threads with FP32 bulk arithmetic (fits the register
// file at <= 64 registers per thread; 608 with more than two phases), 512
// with FP64.
template <typename T, int NPH>
struct EnsMaxThreads {
    static constexpr int value = (sizeof(T) == 8) ? 512 : (NPH > 2) ? 608 : 1024;
};

// a / b of the FP64 parts: IEEE in the reference order, a refined reciprocal
// in mixed precision.
template <typename T>
__device__ __forceinline__ double ens_div(double a, double b) {
    return (sizeof(T) == 8) ? a / b : a * frcp(b);
}

// Primitives of one cell (density, velocity, pressure) from its conservative
// values.
template <typename T, int NPH>
__device__ __forceinline__ void ens_prim(const EnsArgs& A, const Params& P, double rhoC, double mom, double rhoE,
                                         const double* ar, const double* al, double& rhoP, double& u, double& p) {
    if (NPH > 0) {
        double rho = 0.0;
#pragma unroll
        for (int ph = 0; ph < NPH; ++ph)
            if (ph < P.nPh) rho += ar[ph];
        rhoP = smax(rho, 1e-14);
        u = ens_div<T>(mom, rhoP);
        const double ke = 0.5 * rhoP * u * u;
        if (sizeof(T) == 8) {
            p = mixture_pressure<NPH>(P, rhoE - ke, al);
        } else {
            double sumInv = 0.0, sumPi = 0.0;
#pragma unroll
            for (int ph = 0; ph < NPH; ++ph) {
                if (ph < P.nPh) {
                    sumInv += al[ph] * A.invGm1[ph];
                    sumPi += al[ph] * A.gPiGm1[ph];
                }
            }
            p = ens_div<T>((rhoE - ke) - sumPi, sumInv);
        }
    } else {
        const double rho = smax(rhoC, 1e-14);
        u = ens_div<T>(mom, rho);
        double ke = 0.0 + u * u;
        ke *= 0.5 * rho;
        const double e = rhoE - ke;
        p = P.eosStiffened ? (P.gamma - 1.0) * e - P.gamma * P.pInf : smax((P.gamma - 1.0) * e, 1e-14);
        rhoP = rhoC;
    }
}

// Acoustic limit of one cell (src/RKTimeStepping.cpp:43-123) from its
// primitives.  An infinite wave speed gives 0, which ends the run: frcp's
// correction would make a NaN of it, which a minimum ignores.  (A test of the
// result instead, with the IEEE quotients out of line, cost 2.5 % of a step.)
template <typename T, int NPH>
__device__ __forceinline__ double ens_limit(const EnsArgs& A, const Params& P, double dx, double rho, double u, double p,
                                            const double* ar, const double* al) {
    double cs;
    if (NPH > 0) {
        if (sizeof(T) == 8) {
            cs = mixture_sound_speed<NPH>(P, rho, p, al, ar);
        } else {
            double sumInv = 0.0;
#pragma unroll
            for (int ph = 0; ph < NPH; ++ph) {
                if (ph < P.nPh) {
                    const double rk = smax(ar[ph], 1e-14) * frcp(smax(al[ph], 1e-14));
                    const double ck2 = P.phaseGamma[ph] * (p + P.phasePInf[ph]) * frcp(rk);
                    sumInv += al[ph] * frcp(rk * smax(ck2, 1e-14));
                }
            }
            cs = sqrt(smax(frcp(rho * smax(sumInv, 1e-30)), 0.0));
        }
    } else {
        cs = single_sound_speed(P, rho, p);
    }
    const double speed = fabs(u) + cs;
    if (sizeof(T) == 8) return A.cfl * (dx / speed);
    return (__double2hiint(speed) == 0x7ff00000) ? 0.0 : A.cfl * (dx * frcp(speed));
}

constexpr int kEnsStrip = 26;   // cells per warp and strip: 32 lanes less a three-cell halo on either side

// Shared memory of a block with CHUNKS (FP64): per thread the primitives, the
// low-face values, the mass fractions and the fluxes.
template <int NPH>
__host__ __device__ constexpr size_t ens_smem(int threads) {
    return sizeof(double) * threads * (2 * (3 + NPH) + NPH + 3 + ((NPH > 0) ? 1 + 2 * NPH : 0));
}

template <typename T, int NPH, bool CHUNKS>
__global__ void __launch_bounds__(EnsMaxThreads<T, NPH>::value) k_ensemble(const __grid_constant__ EnsArgs A) {
    extern __shared__ __align__(16) unsigned char ensSmem[];   // CHUNKS: ens_smem()
    __shared__ double red[33];
    constexpr int NVR = 3 + NPH;       // reconstructed: rho, u, p, alpha[NPH]
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nWarps = blockDim.x >> 5;

    const int inst = A.order[blockIdx.x];
    const int n = A.n[inst];
    const long long base = A.off[inst];
    const Params& P = A.P;             // nx / nxT are per instance: n, n + 2 ng
    const int ng = P.ngx;
    const int RK = P.RKOrder;
    const double eps = P.wenoEps;
    const bool weno = (P.reconOrder == SIFV_WENO5);
    double t = A.time[inst];
    int steps = A.steps[inst];
    double dtLast = 0.0;
    auto at = [&](int q) -> long long { return base + ng + q; };
    const EnsState& S0 = A.S[0];
    const double kInf = __longlong_as_double(0x7ff0000000000000LL);
    bool folded = false;               // `limit` holds the acoustic limits of the current state
    double limit = kInf;

    const int stepEnd = A.stepLimit ? min(A.maxSteps, A.stepLimit[inst]) : A.maxSteps;
    while (t < A.tEnd && steps < stepEnd) {
        // ---- dt: computeAcousticTimeStep (src/RKTimeStepping.cpp:43-123) ----
        double dt;
        if (A.constDt > 0) {
            dt = A.constDt;
        } else {
            if (!folded) {             // on the stored primitives
                limit = kInf;
                for (int q = threadIdx.x; q < n; q += blockDim.x) {
                    const long long c = at(q);
                    double a[NPH > 0 ? NPH : 1], ar[NPH > 0 ? NPH : 1];
#pragma unroll
                    for (int ph = 0; ph < NPH; ++ph) {
                        a[ph] = (ph < P.nPh) ? S0.alpha[ph][c] : 0.0;
                        ar[ph] = (ph < P.nPh) ? S0.alphaRho[ph][c] : 0.0;
                    }
                    limit = smin(limit, ens_limit<T, NPH>(A, P, A.dx[c], S0.rho[c], A.velU[c], A.pres[c], ar, a));
                }
            }
            const double m = block_min_bcast(limit, red);
            dt = smin(A.maxDt, m);
        }
        limit = kInf;
        folded = RK > 1;
        const double target = A.tEnd - t;
        if (target > 0) dt = smin(dt, target);
        if (!(dt > 0.0)) {   // a non-finite wave speed: stop instead of stepping in place
            if (threadIdx.x == 0) A.status[inst] = 1;
            break;
        }

        for (int s = 0; s < RK; ++s) {
            // SSP-RK coefficients, src/ExplicitSolver.cpp:92-103
            double c1, c2, c3, c4;
            if (RK == 1) { c1 = 1.0; c2 = 0.0; c3 = 1.0; c4 = 1.0; }
            else if (RK == 2) {
                if (s == 0) { c1 = 1.0; c2 = 0.0; c3 = 1.0; c4 = 1.0; } else { c1 = 1.0; c2 = 1.0; c3 = 1.0; c4 = 2.0; }
            } else {
                if (s == 0) { c1 = 1.0; c2 = 0.0; c3 = 1.0; c4 = 1.0; }
                else if (s == 1) { c1 = 1.0; c2 = 3.0; c3 = 1.0; c4 = 4.0; }
                else { c1 = 2.0; c2 = 1.0; c3 = 2.0; c4 = 3.0; }
            }
            const double iC4 = 1.0 / c4;
            // stage input / output: S0 -> S1 (-> S2) -> S0; RK1 writes S1 and copies it back
            const EnsState& In = A.S[s];
            const bool lastStage = (s == RK - 1);
            const EnsState& Out = (lastStage && RK > 1) ? A.S[0] : A.S[s + 1];
            const bool writePrim = lastStage && RK > 1;

            // a team of consecutive threads takes its cells and a halo of three on either side: a warp, or the block
            const int team = CHUNKS ? (int)blockDim.x : 32, me = CHUNKS ? (int)threadIdx.x : lane;
            T* const sW = reinterpret_cast<T*>(ensSmem);
            T* const sLo = sW + NVR * team;
            double* const sY = reinterpret_cast<double*>(sLo + NVR * team);
            double* const sF = sY + NPH * team;
            const int first = CHUNKS ? 0 : warp * kEnsStrip, step = CHUNKS ? team - 6 : nWarps * kEnsStrip;
            for (int c0 = first; c0 < n; c0 += step) {
                // ---- primitives of position q (threads past the last ghost repeat it) ----
                const int q = c0 - 3 + me;
                // a block's warps past the last ghost have nothing to do but the barriers
                const bool live = !CHUNKS || q - lane < n + 3;
                long long c = 0;
                double mom = 0.0, rhoE = 0.0, rhoP = 0.0, ar[NPH > 0 ? NPH : 1], al[NPH > 0 ? NPH : 1];
                double y[NPH > 0 ? NPH : 1];   // mass fractions
                T w[NVR], hi[NVR], lo[NVR];
                if (live) {
                    double sn, sa, u, p;
                    const int sq = prim_src(min(q, n + 2), n, P.bc[0], P.bc[1], sn, sa);
                    c = at(sq);
#pragma unroll
                    for (int ph = 0; ph < NPH; ++ph) {
                        ar[ph] = (ph < P.nPh) ? In.alphaRho[ph][c] : 0.0;
                        al[ph] = (ph < P.nPh) ? In.alpha[ph][c] : 0.0;
                    }
                    mom = In.rhoU[c];
                    rhoE = In.rhoE[c];
                    ens_prim<T, NPH>(A, P, (NPH > 0) ? 0.0 : In.rho[c], mom, rhoE, ar, al, rhoP, u, p);
                    w[0] = T(rhoP);
                    w[1] = T((sn * sa) * u);
                    w[2] = T(p);
#pragma unroll
                    for (int ph = 0; ph < NPH; ++ph) w[3 + ph] = T(al[ph]);
                    if constexpr (CHUNKS) {
#pragma unroll
                        for (int v = 0; v < NVR; ++v) sW[v * team + me] = w[v];
                    }
                }
                if constexpr (CHUNKS) __syncthreads();
                // ---- both face values of the cell (all but the outer two threads) ----
                if (live) {
#pragma unroll
                    for (int v = 0; v < NVR; ++v) {
                        if (v >= 3 && v - 3 >= P.nPh) continue;
                        T x0, x1, x3, x4;
                        if constexpr (CHUNKS) {
                            const T* const x = sW + v * team + min(max(me, 2), team - 3);
                            x0 = x[-2]; x1 = x[-1]; x3 = x[1]; x4 = x[2];
                        } else {
                            x0 = __shfl_up_sync(kAll, w[v], 2); x1 = __shfl_up_sync(kAll, w[v], 1);
                            x3 = __shfl_down_sync(kAll, w[v], 1); x4 = __shfl_down_sync(kAll, w[v], 2);
                        }
                        if (weno) {
                            if constexpr (sizeof(T) == 4) {
                                weno5_pair(x0, x1, w[v], x3, x4, T(eps), hi[v], lo[v]);
                            } else {
                                hi[v] = weno5_high<T>(x0, x1, w[v], x3, x4, T(eps));
                                lo[v] = weno5_low<T>(x0, x1, w[v], x3, x4, T(eps));
                            }
                        } else {
                            hi[v] = upwind5L<T>(x0, x1, w[v], x3, x4);
                            lo[v] = upwind5R<T>(x0, x1, w[v], x3, x4);
                        }
                        if constexpr (CHUNKS) sLo[v * team + me] = lo[v];
                    }
                    if constexpr (CHUNKS && NPH > 0) {
#pragma unroll
                        for (int ph = 0; ph < NPH; ++ph)
                            if (ph < P.nPh) sY[ph * team + me] = y[ph] = ar[ph] / smax(rhoP, 1e-14);
                    }
                }
                if constexpr (CHUNKS) __syncthreads();
                // ---- the cell's high face: left state its own, right state the next thread's ----
                FaceFlux<NPH, T> Fx;
                double fAR[NPH > 0 ? NPH : 1];
                if (live) {
                    const int next = CHUNKS ? min(me + 1, team - 1) : 0;
                    auto above = [&](int v) -> T {
                        if constexpr (CHUNKS) return sLo[v * team + next];
                        else return __shfl_down_sync(kAll, lo[v], 1);
                    };
                    FaceState<NPH, T> L, R;
                    L.u[1] = L.u[2] = R.u[1] = R.u[2] = T(0.0);
                    L.sigma = R.sigma = T(0.0);
                    L.rho = hi[0];
                    L.u[0] = hi[1];
                    L.p = hi[2];
                    R.rho = above(0);
                    R.u[0] = above(1);
                    R.p = above(2);
#pragma unroll
                    for (int ph = 0; ph < NPH; ++ph) {
                        L.alpha[ph] = R.alpha[ph] = T(0.0);
                        if (ph < P.nPh) {
                            L.alpha[ph] = hi[3 + ph];
                            R.alpha[ph] = above(3 + ph);
                        }
                    }
                    if (NPH > 0) {
                        eff_gamma_piinf<NPH, T>(P, L.alpha, L.gEff, L.piEff);
                        eff_gamma_piinf<NPH, T>(P, R.alpha, R.gEff, R.piEff);
                    } else {
                        L.gEff = R.gEff = T(P.gamma);
                        L.piEff = R.piEff = T(P.pInf);
                    }
                    switch (P.riemann) {
                        case SIFV_HLLC: hllc_flux<0, NPH, T>(P, L, R, Fx); break;
                        case SIFV_RUSANOV: rusanov_flux<0, NPH, T>(P, L, R, Fx); break;
                        default: lf_flux<0, NPH, T>(P, L, R, Fx); break;
                    }
                    __syncwarp();
                    // upwinded partial-density flux (src/ExplicitSolver.cpp:307-326)
                    if (NPH > 0) {
                        const double iRho = (sizeof(T) == 8) ? 0.0 : frcp(smax(rhoP, 1e-14));
#pragma unroll
                        for (int ph = 0; ph < NPH; ++ph) {
                            if (ph < P.nPh) {
                                double yr;
                                if constexpr (CHUNKS) {
                                    yr = sY[ph * team + next];
                                } else {
                                    y[ph] = (sizeof(T) == 8) ? ar[ph] / smax(rhoP, 1e-14) : ar[ph] * iRho;
                                    yr = __shfl_down_sync(kAll, y[ph], 1);
                                }
                                fAR[ph] = (((double)Fx.mass >= 0) ? y[ph] : yr) * (double)Fx.mass;
                            }
                        }
                    }
                    if constexpr (CHUNKS) {
                        sF[me] = Fx.mass;
                        sF[team + me] = Fx.mom[0];
                        sF[2 * team + me] = Fx.energy;
                        if (NPH > 0) {
                            sF[3 * team + me] = Fx.fvel;
#pragma unroll
                            for (int ph = 0; ph < NPH; ++ph)
                                if (ph < P.nPh) {
                                    sF[(4 + ph) * team + me] = Fx.alpha[ph];
                                    sF[(4 + NPH + ph) * team + me] = fAR[ph];
                                }
                        }
                    }
                }
                if constexpr (CHUNKS) __syncthreads();
                // ---- the cell (all but the outer three threads): divergence (src/ExplicitSolver.cpp:294-496) and
                // update (127-188) ----
                const bool mine = me >= 3 && me < team - 3 && q < n;
                if (CHUNKS && !mine) continue;
                const double dx = A.dx[c];
                const double coeff = ens_div<T>(1.0 * 1.0, (dx * 1.0) * 1.0);
                auto below = [&](double f, int row) {   // the flux through the cell's low face
                    if constexpr (CHUNKS) return sF[row * team + me - 1];
                    else return __shfl_up_sync(kAll, f, 1);
                };
                auto div = [&](double f, int row) {
                    const double fl = below(f, row);
                    double r = 0.0;
                    r += coeff * fl;
                    r -= coeff * f;
                    return r;
                };
                const double rR = div((double)Fx.mass, 0), rU = div((double)Fx.mom[0], 1), rE = div((double)Fx.energy, 2);
                double rAR[NPH > 0 ? NPH : 1], rA[NPH > 0 ? NPH : 1];
                if (NPH > 0) {
                    const double fl = below((double)Fx.fvel, 3);
                    double divU = 0.0;
                    divU -= coeff * fl;
                    divU += coeff * (double)Fx.fvel;
#pragma unroll
                    for (int ph = 0; ph < NPH; ++ph) {
                        if (ph < P.nPh) {
                            rAR[ph] = div(fAR[ph], 4 + NPH + ph);
                            double r2 = div((double)Fx.alpha[ph], 4 + ph);
                            r2 += al[ph] * divU;
                            rA[ph] = r2;
                        }
                    }
                }
                if (!mine) continue;
                // U0 = the step-start state S0 (its density the step-start primitive; stage 0: the input itself)
                auto upd = [&](double x, double x0, double r) {
                    if (RK == 1) return x + dt * r;
                    const double y = c1 * x + c2 * x0 + c3 * dt * r;
                    return (sizeof(T) == 8) ? y / c4 : y * iC4;
                };
                const bool s0 = (s == 0);
                double nRho = upd(rhoP, s0 ? rhoP : S0.rho[c], rR);
                const double nU = upd(mom, s0 ? mom : S0.rhoU[c], rU);
                const double nE = upd(rhoE, s0 ? rhoE : S0.rhoE[c], rE);
                double nAR[NPH > 0 ? NPH : 1], nA[NPH > 0 ? NPH : 1];
                if (NPH > 0) {   // and the clamps, src/ExplicitSolver.cpp:169-185
                    double rhoSum = 0.0, aSum = 0.0;
#pragma unroll
                    for (int ph = 0; ph < NPH; ++ph) {
                        if (ph < P.nPh) {
                            nAR[ph] = smax(upd(ar[ph], s0 ? ar[ph] : S0.alphaRho[ph][c], rAR[ph]), 1e-14);
                            rhoSum += nAR[ph];
                            nA[ph] = smax(upd(al[ph], s0 ? al[ph] : S0.alpha[ph][c], rA[ph]), P.alphaMin);
                            aSum += nA[ph];
                        }
                    }
                    nRho = rhoSum;
                    const double iSum = (sizeof(T) == 8) ? 0.0 : frcp(aSum);
#pragma unroll
                    for (int ph = 0; ph < NPH; ++ph)
                        if (ph < P.nPh) nA[ph] = (sizeof(T) == 8) ? nA[ph] / aSum : nA[ph] * iSum;
                }
                Out.rho[c] = nRho;
                Out.rhoU[c] = nU;
                Out.rhoE[c] = nE;
#pragma unroll
                for (int ph = 0; ph < NPH; ++ph)
                    if (ph < P.nPh) { Out.alphaRho[ph][c] = nAR[ph]; Out.alpha[ph][c] = nA[ph]; }
                if (writePrim) {   // final cons -> prim (src/ExplicitSolver.cpp:192-200)
                    double r2, u2, p2;
                    ens_prim<T, NPH>(A, P, nRho, nU, nE, nAR, nA, r2, u2, p2);
                    if (NPH > 0) Out.rho[c] = r2;
                    A.velU[c] = u2;
                    A.pres[c] = p2;
                    if (A.constDt <= 0) limit = smin(limit, ens_limit<T, NPH>(A, P, dx, r2, u2, p2, nAR, nA));
                }
            }
            __syncthreads();
            if (lastStage && RK == 1) {   // S1 -> S0 and the primitives of the new state
                const EnsState& S1 = A.S[1];
                for (int q = threadIdx.x; q < n; q += blockDim.x) {
                    const long long c = at(q);
                    double nAR[NPH > 0 ? NPH : 1], nA[NPH > 0 ? NPH : 1], r2, u2, p2;
                    const double nRho = S1.rho[c], nU = S1.rhoU[c], nE = S1.rhoE[c];
                    S0.rhoU[c] = nU;
                    S0.rhoE[c] = nE;
#pragma unroll
                    for (int ph = 0; ph < NPH; ++ph)
                        if (ph < P.nPh) {
                            nAR[ph] = S1.alphaRho[ph][c];
                            nA[ph] = S1.alpha[ph][c];
                            S0.alphaRho[ph][c] = nAR[ph];
                            S0.alpha[ph][c] = nA[ph];
                        }
                    ens_prim<T, NPH>(A, P, nRho, nU, nE, nAR, nA, r2, u2, p2);
                    S0.rho[c] = r2;
                    A.velU[c] = u2;
                    A.pres[c] = p2;
                }
                __syncthreads();
            }
        }
        t += dt;
        ++steps;
        dtLast = dt;
    }
    // PRIM ghost fill of the state (src/RectilinearMesh.cpp:498-524), for the caller
    for (int g = threadIdx.x; g < 2 * ng; g += blockDim.x) {
        int q = (g < ng) ? -1 - g : n + (g - ng);
        double sn, sa;
        int sq = prim_src(q, n, P.bc[0], P.bc[1], sn, sa);
        long long d = at(q), sc = at(sq);
        S0.rho[d] = S0.rho[sc];
        A.velU[d] = (sn * sa) * A.velU[sc];
        A.pres[d] = A.pres[sc];
#pragma unroll
        for (int ph = 0; ph < NPH; ++ph)
            if (ph < P.nPh) { S0.alphaRho[ph][d] = S0.alphaRho[ph][sc]; S0.alpha[ph][d] = S0.alpha[ph][sc]; }
    }
    if (threadIdx.x == 0) {
        A.time[inst] = t;
        A.steps[inst] = steps;
        A.lastDt[inst] = dtLast;
    }
}

}  // namespace sifv
