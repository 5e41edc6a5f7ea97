// sifv_stage.cuh -- one SSP-RK stage of the explicit step as one kernel, in
// the reference's operation order (ExplicitSolver::step,
// src/ExplicitSolver.cpp:109-190), 1D and 2D, where it takes less time than the
// separate kernels (stage_pays; and for the fast and mixed modes on 1D meshes
// up to a size, fused_stage).
//
// A block owns a tile of cells.  It converts the tile and its three halo
// layers to primitives in shared memory (ghost cells through the PRIM ghost
// map, so no ghost layer of the input is read), then per direction
// reconstructs every cell of the tile and its two neighbours to both of its
// face values, solves the faces' Riemann problems, and finally updates the
// tile's cells, all with the expressions of k_prim_bc, k_face, k_visc_face
// and k_assemble; the results are bit-identical to theirs.  Input and output
// are different states.
//
// Why one kernel: the four kernels it stands for pass primitives and fluxes
// through memory (13 to 25 arrays in 2D) and, below about 10^5 cells, each
// costs a launch and a dependent latency chain.  The arithmetic (about 1900
// FP64 instructions per cell in 2D, a quarter of them in the 64 quotients of
// the WENO weights, sifv_rn.cuh) is the bound that remains on large meshes:
// the FP64 pipe is 61 % busy at 1024^2 (207 us per stage), held there by
// barriers and load latency at three blocks per SM.  Per RK3 step, the
// separate kernels against this one: 1D 1000 cells 82 -> 26 us; 256^2
// 134 -> 92; 1531 x 1021 viscous 1370 -> 1000; 480 x 352 two-phase 320 -> 262
// (278 with the fluxes in a buffer of their own, which leaves room for two
// two-phase blocks per SM instead of three).
#pragma once

#include "sifv_stage_api.h"

namespace sifv {

// One cell can be the source of every ghost layer of both ends of an axis.
constexpr int kStageImages = 1 + 2 * kStageMaxGhost;

// Tile and block shapes.  2D: 32 x 8 cells, 320 threads: the cells a
// direction reconstructs (34 x 8 or 32 x 10) and its faces (33 x 8 or 32 x 9)
// are one per thread.  1D: 30 cells, one warp per reconstructed variable: a
// 1D mesh has too few cells to fill the GPU, and the chain of one thread
// reconstructing every variable in turn is what it would wait for.
template <int DIM, int NPH>
struct StageTile {
    static constexpr int NV = DIM + 2 + NPH;              // reconstructed: rho, u.., p, alpha..
    static constexpr int TX = (DIM == 1) ? 30 : 32, TY = (DIM == 1) ? 1 : 8;
    static constexpr int threads = (DIM == 1) ? 32 * NV : 320;
    static constexpr int W = TX + 6, H = (DIM == 1) ? 1 : TY + 6;
    static constexpr int RX = (TX + 2) * TY, RY = TX * (TY + 2);   // reconstructed cells per direction
    static constexpr int R = (DIM == 1 || RX > RY) ? RX : RY;
    static constexpr int FX = (TX + 1) * TY, FY = (DIM == 1) ? 0 : TX * (TY + 1);
    static constexpr int NF = DIM + 2 + (NPH > 0 ? 1 + 2 * NPH : 0);   // flux slots
    static constexpr size_t smem = ((size_t)(NV + NPH) * W * H + 2 * (size_t)NV * R) * sizeof(double);
    static_assert(NF <= 2 * NV, "a face's fluxes take the place of the values it read");
    static_assert((DIM + 1) * (FX + FY) <= 2 * NV * R, "the face stresses reuse the reconstruction buffer");
};

// cons_to_prim_cell on a StageState.
template <int DIM, int NPH>
__device__ __forceinline__ void stage_prim(const Params& P, double rhoC, const double* mom, double rhoE,
                                           const double* ar, const double* al, double& rhoOut, double* u, double& p) {
    if (NPH == 0) {
        double rho = smax(rhoC, 1e-14);
#pragma unroll
        for (int d = 0; d < DIM; ++d) u[d] = mom[d] / rho;
        double ke = 0.0;
#pragma unroll
        for (int d = 0; d < DIM; ++d) ke += u[d] * u[d];
        ke *= 0.5 * rho;
        double e = rhoE - ke;
        p = P.eosStiffened ? (P.gamma - 1.0) * e - P.gamma * P.pInf : smax((P.gamma - 1.0) * e, 1e-14);
        rhoOut = rhoC;
    } else {
        double rho = 0.0;
#pragma unroll
        for (int ph = 0; ph < NPH; ++ph)
            if (ph < P.nPh) rho += ar[ph];
        double rs = smax(rho, 1e-14);
#pragma unroll
        for (int d = 0; d < DIM; ++d) u[d] = mom[d] / rs;
        double ke = 0.5 * rs * u[0] * u[0];
        if (DIM >= 2) ke += 0.5 * rs * u[1] * u[1];
        p = mixture_pressure<NPH>(P, rhoE - ke, al);
        rhoOut = rs;
    }
}

// Flux through a face normal to axis 0 of the two states.
template <int NPH, int RS>
__device__ __forceinline__ void stage_riemann(const Params& P, const FaceState<NPH>& L, const FaceState<NPH>& R,
                                              FaceFlux<NPH>& F) {
    if (RS == SIFV_HLLC) hllc_flux<0, NPH>(P, L, R, F);
    else if (RS == SIFV_RUSANOV) rusanov_flux<0, NPH>(P, L, R, F);
    else lf_flux<0, NPH>(P, L, R, F);
}

// Reconstruction of direction D: both face values of every cell from its
// five-cell stencil (recon_pair's expressions).  The loop over the variables
// stays a loop: one copy of the two reconstructions per direction.
template <int D, int DIM, int NPH>
__device__ __forceinline__ void stage_recon(const Params& P, const double* sW, double* sHi, double* sLo, int lx,
                                            int ly) {
    using T = StageTile<DIM, NPH>;
    constexpr int CX = T::TX + (D == 0 ? 2 : 0), N = (D == 0) ? T::RX : T::RY;
    constexpr int ST = (D == 0) ? 1 : T::W;
    const int nv = DIM + 2 + ((NPH > 0) ? P.nPh : 0);
    const bool weno = (P.reconOrder == SIFV_WENO5);
    const double eps = P.wenoEps;
    static_assert(DIM == 1 ? N == 32 : N <= T::threads, "one cell per thread");
    const int c = (DIM == 1) ? (int)threadIdx.x % N : (int)threadIdx.x, b = c / CX, a = c % CX;
    // tile cell (a - [D == 0], b - [D == 1]); faces past the mesh's last cell are not used
    const int i = a - (D == 0), j = b - (D == 1);
    if (c >= N || i > lx || j > ly || (D == 1 && i >= lx) || (D == 0 && DIM > 1 && j >= ly)) return;
    int v = (DIM == 1) ? (int)threadIdx.x / N : 0;
    const double* f = sW + v * (T::W * T::H) + (i + 3) + ((DIM == 1) ? 0 : (j + 3) * T::W);
    double *hi = sHi + v * T::R + c, *lo = sLo + v * T::R + c;
#pragma unroll 1
    for (; v < nv; v += (DIM == 1) ? T::NV : 1) {
        const double x0 = f[-2 * ST], x1 = f[-ST], x2 = f[0], x3 = f[ST], x4 = f[2 * ST];
        *hi = weno ? weno5_high<double>(x0, x1, x2, x3, x4, eps) : upwind5L<double>(x0, x1, x2, x3, x4);
        *lo = weno ? weno5_low<double>(x0, x1, x2, x3, x4, eps) : upwind5R<double>(x0, x1, x2, x3, x4);
        f += T::W * T::H;
        hi += T::R;
        lo += T::R;
    }
}

// Riemann problems of direction d's faces.  A face's fluxes take the place of
// the values only it reads: slots 0 .. NV - 1 of its left cell's high-face
// values, the rest of its right cell's low-face ones (stage_flux).  Both
// directions run the axis-0 solver on (normal, transverse) components: in two
// dimensions its sums over the components are commutative, so exchanging the
// components changes no bit.
template <int DIM, int NPH, int RS>
__device__ __forceinline__ void stage_faces(int d, const Params& P, const double* sW, double* sHi, double* sLo, int lx,
                                            int ly) {
    using T = StageTile<DIM, NPH>;
    const int gx = T::TX + (d == 0), nface = (d == 0) ? T::FX : T::FY;
    const int cx = T::TX + (d == 0 ? 2 : 0), R_ = T::R;
    constexpr int NV = T::NV;
    const int t = threadIdx.x;
    static_assert(T::FX <= T::threads && T::FY <= T::threads, "one face per thread");
    if (t < nface) {
        const int j = (d == 0) ? t / (T::TX + 1) : t / T::TX, i = t - j * gx;
        if (i > lx || j > ly || (d == 1 && i >= lx) || (d == 0 && DIM > 1 && j >= ly)) return;
        const int cl = i + cx * j;                      // left cell (i - 1, j) or (i, j - 1)
        const int cr = cl + ((d == 0) ? 1 : cx);
        FaceState<NPH> L, R;
        L.u[1] = L.u[2] = R.u[1] = R.u[2] = 0.0;
        L.sigma = R.sigma = 0.0;
        L.rho = sHi[cl];
        R.rho = sLo[cr];
#pragma unroll
        for (int q = 0; q < DIM; ++q) {
            const int v = (DIM == 1) ? 1 : 1 + (q ^ d);
            L.u[q] = sHi[v * R_ + cl];
            R.u[q] = sLo[v * R_ + cr];
        }
        L.p = sHi[(DIM + 1) * R_ + cl];
        R.p = sLo[(DIM + 1) * R_ + cr];
#pragma unroll
        for (int ph = 0; ph < NPH; ++ph) {
            L.alpha[ph] = R.alpha[ph] = 0.0;
            if (ph < P.nPh) {
                L.alpha[ph] = sHi[(DIM + 2 + ph) * R_ + cl];
                R.alpha[ph] = sLo[(DIM + 2 + ph) * R_ + cr];
            }
        }
        if (NPH > 0) {
            eff_gamma_piinf<NPH>(P, L.alpha, L.gEff, L.piEff);
            eff_gamma_piinf<NPH>(P, R.alpha, R.gEff, R.piEff);
        } else {
            L.gEff = R.gEff = P.gamma;
            L.piEff = R.piEff = P.pInf;
        }
        FaceFlux<NPH> Fx;
        stage_riemann<NPH, RS>(P, L, R, Fx);
        auto put = [&](int q, double x) {
            if (q < NV) sHi[q * R_ + cl] = x; else sLo[(q - NV) * R_ + cr] = x;
        };
        put(0, Fx.mass);
#pragma unroll
        for (int q = 0; q < DIM; ++q) sHi[((DIM == 1) ? 1 : 1 + (q ^ d)) * R_ + cl] = Fx.mom[q];
        put(DIM + 1, Fx.energy);
        if (NPH > 0) {
            put(DIM + 2, Fx.fvel);
            // upwinded partial-density flux (src/ExplicitSolver.cpp:307-326)
            const int right = (i + 3) + ((DIM == 1) ? 0 : (j + 3) * T::W);
            const int upw = (Fx.mass >= 0) ? right - ((d == 0) ? 1 : T::W) : right;
            const double rhoUpw = smax(sW[upw], 1e-14);
#pragma unroll
            for (int ph = 0; ph < NPH; ++ph) {
                if (ph < P.nPh) {
                    put(DIM + 3 + ph, Fx.alpha[ph]);
                    put(DIM + 3 + NPH + ph, (sW[(NV + ph) * (T::W * T::H) + upw] / rhoUpw) * Fx.mass);
                }
            }
        }
    }
}

// Flux slot q of the face whose left cell is reconstructed cell cl of
// direction D.
template <int D, int DIM, int NPH>
__device__ __forceinline__ double stage_flux(const double* sHi, const double* sLo, int q, int cl) {
    using T = StageTile<DIM, NPH>;
    return (q < T::NV) ? sHi[q * T::R + cl] : sLo[(q - T::NV) * T::R + cl + ((D == 0) ? 1 : T::TX)];
}

// One direction's share of the cell's divergence, slot by slot (div_slot's
// and div_fvel's order): r of every slot, starting from 0 along x.
template <int D, int DIM, int NPH>
__device__ __forceinline__ void stage_div(const Params& P, const double* sHi, const double* sLo, int i, int j, double c,
                                          double* r) {
    using T = StageTile<DIM, NPH>;
    const int lo = (D == 0) ? i + (T::TX + 2) * j : i + T::TX * j, hi = lo + ((D == 0) ? 1 : T::TX);
#pragma unroll
    for (int q = 0; q < T::NF; ++q) {
        if (NPH > 0 && q == 0) continue;   // the mixture density is the sum of the partial densities
        const double fl = c * stage_flux<D, DIM, NPH>(sHi, sLo, q, lo), fh = c * stage_flux<D, DIM, NPH>(sHi, sLo, q, hi);
        double x = (D == 0) ? 0.0 : r[q];
        if (NPH > 0 && q == DIM + 2) {   // the face velocity: the opposite signs
            x -= fl;
            x += fh;
        } else {
            x += fl;
            x -= fh;
        }
        r[q] = x;
    }
}

// Viscous stress and work on one direction's faces (visc_stress) into sV.
template <int D, int DIM, int NPH>
__device__ __forceinline__ void stage_visc(const StageArgs& A, const double* sW, double* sV, int i0, int j0, int lx,
                                           int ly) {
    using T = StageTile<DIM, NPH>;
    const Params& P = A.P;
    constexpr int GX = T::TX + (D == 0), GY = T::TY + (D == 1), NFACE = GX * GY, WH = T::W * T::H;
    for (int t = threadIdx.x; t < NFACE; t += T::threads) {
        const int i = t % GX, j = t / GX;
        if (i > lx || j > ly || (D == 1 && i >= lx) || (D == 0 && DIM > 1 && j >= ly)) continue;
        const int iR = (i + 3) + ((DIM == 1) ? 0 : (j + 3) * T::W);
        const int iL = iR - ((D == 0) ? 1 : T::W);
        double muF = P.mu;
        if (NPH > 0 && P.perPhaseMu) {
            double muL = 0.0, muR = 0.0;
#pragma unroll
            for (int ph = 0; ph < NPH; ++ph) {
                if (ph < P.nPh) {
                    muL += sW[(DIM + 2 + ph) * WH + iL] * P.phaseMu[ph];
                    muR += sW[(DIM + 2 + ph) * WH + iR] * P.phaseMu[ph];
                }
            }
            muF = 0.5 * (muL + muR);
        }
        double tau[3], work;
        visc_stress<D>(DIM, sW + WH, sW + ((DIM >= 2) ? 2 : 1) * WH, (const double*)nullptr, iL, iR, 1, T::W, 0,
                       A.dx + (i0 + i + P.ngx), A.dy + (j0 + j + P.ngy), A.dz, muF, tau, work);
#pragma unroll
        for (int d = 0; d < DIM; ++d) sV[d * NFACE + t] = tau[d];
        sV[DIM * NFACE + t] = work;
    }
}

// Ghost positions along one axis whose PRIM source is interior cell c, after
// c itself, with the axis's velocity signs.
__device__ __forceinline__ int stage_images(int c, int n, int ng, int bcLo, int bcHi, int* pos, double* sn, double* sa) {
    int m = 1;
    pos[0] = c;
    sn[0] = sa[0] = 1.0;
    if (c >= ng && c < n - ng) return m;
    for (int g = 1; g <= ng; ++g) {
        double a, b;
        if (m < kStageImages && prim_src(-g, n, bcLo, bcHi, a, b) == c) { pos[m] = -g; sn[m] = a; sa[m] = b; ++m; }
        if (m < kStageImages && prim_src(n - 1 + g, n, bcLo, bcHi, a, b) == c) { pos[m] = n - 1 + g; sn[m] = a; sa[m] = b; ++m; }
    }
    return m;
}

// k_bc_prim for the ghost images of one interior cell with the new state's
// primitives: a cell at the mesh's edge writes its own images, so the step
// needs no ghost pass of its own.
template <int DIM, int NPH>
__device__ __noinline__ void stage_ghosts(const StageArgs& A, int i, int j, double rho, const double* u, double p,
                                          const double* nAR, const double* nA) {
    const Params& P = A.P;
    int px[kStageImages], py[kStageImages];
    double snx[kStageImages], sax[kStageImages], sny[kStageImages], say[kStageImages];
    const int mx = stage_images(i, P.nx, P.ngx, P.bc[0], P.bc[1], px, snx, sax);
    int my = 1;
    py[0] = j;
    sny[0] = say[0] = 1.0;
    if (DIM >= 2) my = stage_images(j, P.ny, P.ngy, P.bc[2], P.bc[3], py, sny, say);
    const double sg = A.sigma[cidx(P, i, j, 0)];
    for (int b = 0; b < my; ++b)
        for (int a = (b == 0) ? 1 : 0; a < mx; ++a) {
            const size_t d = cidx(P, px[a], py[b], 0);
            A.out.rho[d] = rho;
            A.velU[d] = ((snx[a] * sax[a]) * say[b]) * u[0];
            if (DIM >= 2) A.velV[d] = (sax[a] * (sny[b] * say[b])) * u[1];
            A.pres[d] = p;
            A.sigma[d] = sg;
#pragma unroll
            for (int ph = 0; ph < NPH; ++ph) {
                if (ph < P.nPh) {
                    A.out.alphaRho[ph][d] = nAR[ph];
                    A.out.alpha[ph][d] = nA[ph];
                }
            }
        }
}

template <int DIM, int NPH, int RS>
__global__ void __launch_bounds__(StageTile<DIM, NPH>::threads, 3)
    k_stage(const __grid_constant__ StageArgs A) {
    using T = StageTile<DIM, NPH>;
    constexpr int NV = T::NV, WH = T::W * T::H;
    extern __shared__ double sm[];
    double* const sW = sm;                       // primitives, then the partial densities
    double* const sHi = sW + (NV + NPH) * WH;    // high- / low-face values of the direction at hand
    double* const sLo = sHi + NV * T::R;
    const Params& P = A.P;
    const int i0 = (int)blockIdx.x * T::TX, j0 = (int)blockIdx.y * T::TY;
    const int lx = min(T::TX, P.nx - i0), ly = (DIM == 1) ? 1 : min(T::TY, P.ny - j0);   // cells of this tile
    grid_dep_launch();
    grid_dep_wait();
    if (A.dtFixed <= 0.0 && A.ctl->skip) return;

    // ---- primitives of the tile and its halo ----
    for (int t = threadIdx.x; t < WH; t += T::threads) {
        const int a = t % T::W, b = t / T::W;
        const int i = i0 + a - 3, j = (DIM == 1) ? 0 : j0 + b - 3;
        if (i >= P.nx + 3 || (DIM >= 2 && j >= P.ny + 3)) continue;
        double sg[3];
        const size_t s = prim_source(P, i, j, 0, sg);
        double mom[2], ar[NPH > 0 ? NPH : 1], al[NPH > 0 ? NPH : 1], rho, u[2], p;
        mom[0] = A.in.mom[0][s];
        if (DIM >= 2) mom[1] = A.in.mom[1][s];
#pragma unroll
        for (int ph = 0; ph < NPH; ++ph) {
            ar[ph] = (ph < P.nPh) ? A.in.alphaRho[ph][s] : 0.0;
            al[ph] = (ph < P.nPh) ? A.in.alpha[ph][s] : 0.0;
        }
        stage_prim<DIM, NPH>(P, (NPH == 0) ? A.in.rho[s] : 0.0, mom, A.in.rhoE[s], ar, al, rho, u, p);
        const bool inside = i >= 0 && i < P.nx && (DIM == 1 || (j >= 0 && j < P.ny));
        sW[t] = rho;
        sW[WH + t] = inside ? u[0] : sg[0] * u[0];
        if (DIM >= 2) sW[2 * WH + t] = inside ? u[1] : sg[1] * u[1];
        sW[(DIM + 1) * WH + t] = p;
#pragma unroll
        for (int ph = 0; ph < NPH; ++ph) {
            sW[(DIM + 2 + ph) * WH + t] = al[ph];
            sW[(NV + ph) * WH + t] = ar[ph];
        }
    }
    __syncthreads();

    // ---- fluxes ----
    // divergence (k_assemble's accumulation order: x low face, x high face, y ...)
    const int i = (int)threadIdx.x % T::TX, j = (int)threadIdx.x / T::TX;
    const bool mine = i < lx && j < ly;
    double f[T::NF];
    stage_recon<0, DIM, NPH>(P, sW, sHi, sLo, lx, ly);
    __syncthreads();
    stage_faces<DIM, NPH, RS>(0, P, sW, sHi, sLo, lx, ly);
    __syncthreads();
    const double dxi = mine ? A.dx[i0 + i + P.ngx] : 1.0, dyj = mine ? A.dy[j0 + j + P.ngy] : 1.0, dzk = A.dz[0];
    const double vol = dxi * dyj * dzk;
    const double cx = (dyj * dzk) / vol, cy = (DIM >= 2) ? (dxi * dzk) / vol : 0.0;
    if (mine) stage_div<0, DIM, NPH>(P, sHi, sLo, i, j, cx, f);
    if (DIM >= 2) {
        constexpr int D1 = (DIM >= 2) ? 1 : 0;
        __syncthreads();
        stage_recon<D1, DIM, NPH>(P, sW, sHi, sLo, lx, ly);
        __syncthreads();
        stage_faces<DIM, NPH, RS>(1, P, sW, sHi, sLo, lx, ly);
        __syncthreads();
        if (mine) stage_div<D1, DIM, NPH>(P, sHi, sLo, i, j, cy, f);
    }
    double* const sV = sHi;   // face stresses in place of the fluxes
    if (P.visc) {
        __syncthreads();
        stage_visc<0, DIM, NPH>(A, sW, sV, i0, j0, lx, ly);
        if (DIM >= 2) stage_visc<(DIM >= 2) ? 1 : 0, DIM, NPH>(A, sW, sV + (DIM + 1) * T::FX, i0, j0, lx, ly);
        __syncthreads();
    }

    // ---- update ----
    double dtLimit = __longlong_as_double(0x7ff0000000000000LL);
    if (mine) {
        const size_t c = cidx(P, i0 + i, j0 + j, 0);
        const int w = (i + 3) + ((DIM == 1) ? 0 : (j + 3) * T::W);
        double r[DIM + 2];
#pragma unroll
        for (int q = 0; q < DIM + 2; ++q) r[q] = (NPH > 0 && q == 0) ? 0.0 : f[q];
        double rAR[NPH > 0 ? NPH : 1], rA[NPH > 0 ? NPH : 1];
        if (NPH > 0) {
            const double divU = f[DIM + 2 < T::NF ? DIM + 2 : 0];
#pragma unroll
            for (int ph = 0; ph < NPH; ++ph) {
                if (ph < P.nPh) {
                    rAR[ph] = f[DIM + 3 + NPH + ph];
                    rA[ph] = f[DIM + 3 + ph];
                    rA[ph] += sW[(DIM + 2 + ph) * WH + w] * divU;
                }
            }
        }
        const double rhoC = sW[w];
        if (A.K.hasBodyForce) {   // src/ExplicitSolver.cpp:498-521
            r[1] += rhoC * A.K.accel[0];
            if (DIM >= 2) r[DIM] += rhoC * A.K.accel[1];
            double work = sW[WH + w] * A.K.accel[0];
            if (DIM >= 2) work += sW[2 * WH + w] * A.K.accel[1];
            r[DIM + 1] += rhoC * work;
        }
        if (P.visc) {   // add_face_stress: per direction the low face, then the high face
            const double* vx = sV + i + (T::TX + 1) * j;
#pragma unroll
            for (int d = 0; d < DIM + 1; ++d) r[1 + d] -= cx * vx[d * T::FX];
#pragma unroll
            for (int d = 0; d < DIM + 1; ++d) r[1 + d] += cx * vx[d * T::FX + 1];
            if (DIM >= 2) {
                const double* vy = sV + (DIM + 1) * T::FX + i + T::TX * j;
#pragma unroll
                for (int d = 0; d < DIM + 1; ++d) r[1 + d] -= cy * vy[d * T::FY];
#pragma unroll
                for (int d = 0; d < DIM + 1; ++d) r[1 + d] += cy * vy[d * T::FY + T::TX];
            }
        }
        const double dt = (A.dtFixed > 0.0) ? A.dtFixed : A.ctl->dt;
        const double c1 = A.K.c1, c2 = A.K.c2, c3 = A.K.c3, c4 = A.K.c4;
        const bool s0 = A.K.s == 0;
        // (c1 U + c2 U0 + c3 dt R) / c4; the divisors 1 and 4 are exact as products
        auto upd = [&](double u, double u0, double rr) {
            const double v = c1 * u + c2 * u0 + c3 * dt * rr;
            return (c4 == 1.0) ? v : (c4 == 4.0) ? v * 0.25 : v / c4;
        };
        double nRho = 0.0, nMom[2], nE, nAR[NPH > 0 ? NPH : 1], nA[NPH > 0 ? NPH : 1];
        if (NPH == 0) nRho = upd(rhoC, s0 ? rhoC : A.u0.rho[c], r[0]);
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const double m = A.in.mom[d][c];
            nMom[d] = upd(m, s0 ? m : A.u0.mom[d][c], r[1 + d]);
        }
        const double e = A.in.rhoE[c];
        nE = upd(e, s0 ? e : A.u0.rhoE[c], r[DIM + 1]);
        if (NPH > 0) {   // and the clamps of mp_post
            double aSum = 0.0;
#pragma unroll
            for (int ph = 0; ph < NPH; ++ph) {
                if (ph < P.nPh) {
                    const double ar = sW[(NV + ph) * WH + w], al = sW[(DIM + 2 + ph) * WH + w];
                    nAR[ph] = smax(upd(ar, s0 ? ar : A.u0.alphaRho[ph][c], rAR[ph]), 1e-14);
                    nRho += nAR[ph];
                    nA[ph] = smax(upd(al, s0 ? al : A.u0.alpha[ph][c], rA[ph]), P.alphaMin);
                    aSum += nA[ph];
                }
            }
#pragma unroll
            for (int ph = 0; ph < NPH; ++ph)
                if (ph < P.nPh) nA[ph] = nA[ph] / aSum;
        }
        A.out.rho[c] = nRho;
#pragma unroll
        for (int d = 0; d < DIM; ++d) A.out.mom[d][c] = nMom[d];
        A.out.rhoE[c] = nE;
#pragma unroll
        for (int ph = 0; ph < NPH; ++ph) {
            if (ph < P.nPh) {
                A.out.alphaRho[ph][c] = nAR[ph];
                A.out.alpha[ph][c] = nA[ph];
            }
        }
        if (A.last) {
            double rho, u[2], p;
            stage_prim<DIM, NPH>(P, nRho, nMom, nE, nAR, nA, rho, u, p);
            if (NPH > 0) A.out.rho[c] = rho;
            A.velU[c] = u[0];
            if (DIM >= 2) A.velV[c] = u[1];
            A.pres[c] = p;
            const int gi = i0 + i, gj = j0 + j;
            if (gi < P.ngx || gi >= P.nx - P.ngx || (DIM >= 2 && (gj < P.ngy || gj >= P.ny - P.ngy)))
                stage_ghosts<DIM, NPH>(A, gi, gj, rho, u, p, nAR, nA);
            if (A.dtNext) {   // k_dt_acoustic and k_dt_viscous
                const double cs = (NPH > 0) ? mixture_sound_speed<NPH>(P, rho, p, nA, nAR) : single_sound_speed(P, rho, p);
                double dtCell = dxi / (fabs(u[0]) + cs);
                if (DIM >= 2) dtCell = smin(dtCell, dyj / (fabs(u[1]) + cs));
                dtLimit = A.cfl * dtCell;
                if (P.visc) {
                    double dxMin = dxi;
                    if (DIM >= 2) dxMin = smin(dxMin, dyj);
                    const double nu = P.mu / smax(rho, 1e-14);
                    const double dv = A.cfl * (dxMin * dxMin / (2.0 * DIM * nu));
                    // a NaN limit never wins (block_min_to)
                    if (!(dtLimit == dtLimit) || dv < dtLimit) dtLimit = dv;
                }
            }
        }
    }
    if (A.last && A.dtNext) block_min_to(dtLimit, &A.ctl->dtBits);
}

}  // namespace sifv
