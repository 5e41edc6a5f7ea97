// sifv_adjoint.cuh -- discrete adjoint (reverse) and tangent (forward) of
// the explicit single-phase step: cons -> prim, PRIM ghost fill, WENO5 /
// UPWIND5 reconstruction, Riemann flux, flux divergence and the SSP-RK stage
// update of ExplicitSolver::step (src/ExplicitSolver.cpp:68-203,
// src/Reconstruction.cpp:119-200, src/HLLCSolver.cpp:7-161,
// src/RusanovSolver.cpp:7-83, src/LFSolver.cpp:8-75), linearised about the
// forward trajectory with the time-step sequence held fixed.
//
// Reverse of one stage U' = (c1 U + c2 U0 + c3 dt R(U)) / c4, given
// lam = dJ/dU':
//   k_adj_dir   per direction: mu = coeff_R lam_R - coeff_L lam_L (dJ/dF) on
//               every face, the flux Jacobian's transpose (adj_hllc,
//               adj_central), the reconstructions' transposes (adj_recon), and
//               the sum over the stencils: dJ/dW per cell, ghost positions
//               included;
//   k_adj_cell  per interior cell: adds the directions and the cell's ghost
//               images (ghost velocity signs applied), multiplies by the
//               cons -> prim Jacobian, and updates lam <- (c1/c4) lam +
//               (c3 dt/c4) g, acc0 += (c2/c4) lam_in (dJ/dU0 through the RK
//               combination).
// The tangent runs the same linearisation forwards: k_tan_prim (dW from dU
// incl. ghosts), k_tan_face (dF with Dual<1>), k_tan_update.
#pragma once

#include "sifv_adjoint_api.h"
#include "sifv_common.cuh"
#include "sifv_dual.cuh"
#include "sifv_fastmath.cuh"

namespace sifv {

// number of primitive (rho, u.., p) and conservative variables
template <int DIM>
struct NV {
    static constexpr int n = DIM + 2;
};

// cons slot of each primitive-velocity / flux component: 0 rho, 1..DIM mom, DIM+1 energy
__device__ __forceinline__ double* cons_ptr(const Fields& F, int q, int dim) {
    if (q == 0) return F.rho;
    if (q == dim + 1) return F.rhoE;
    return (q == 1) ? F.rhoU : (q == 2) ? F.rhoV : F.rhoW;
}
__device__ __forceinline__ const double* prim_ptr(const Fields& F, int q, int dim) {
    if (q == 0) return F.rho;
    if (q == dim + 1) return F.pres;
    return (q == 1) ? F.velU : (q == 2) ? F.velV : F.velW;
}

template <int DIR>
__device__ __forceinline__ double face_coeff(const Params& P, const Fields& F, int i, int j, int k) {
    double dxi = F.dx[i + P.ngx], dyj = F.dy[j + P.ngy], dzk = F.dz[k + P.ngz];
    double vol = dxi * dyj * dzk;
    return (DIR == 0) ? (dyj * dzk) / vol : (DIR == 1) ? (dxi * dzk) / vol : (dxi * dyj) / vol;
}

template <int DIR>
__device__ __forceinline__ long long face_index(const Params& P, int i, int j, int k) {
    const long long fnx = P.nx + (DIR == 0), fny = P.ny + (DIR == 1);
    return (long long)i + fnx * ((long long)j + fny * (long long)k);
}

// Face states + Riemann flux in arithmetic T (double or Dual<N>).
template <int DIR, typename T>
__device__ __forceinline__ void riemann_T(const Params& P, const FaceState<0, T>& L, const FaceState<0, T>& R,
                                          FaceFlux<0, T>& Fx) {
    switch (P.riemann) {
        case SIFV_HLLC: hllc_flux<DIR, 0, T>(P, L, R, Fx); break;
        case SIFV_RUSANOV: rusanov_flux<DIR, 0, T>(P, L, R, Fx); break;
        default: lf_flux<DIR, 0, T>(P, L, R, Fx); break;
    }
}

template <typename T>
__device__ __forceinline__ void recon5(bool weno, double eps, const T* v, T& l, T& r) {
    if (weno) {
        l = weno5L<T>(v[0], v[1], v[2], v[3], v[4], T(eps));
        r = weno5R<T>(v[1], v[2], v[3], v[4], v[5], T(eps));
    } else {
        l = upwind5L<T>(v[0], v[1], v[2], v[3], v[4]);
        r = upwind5R<T>(v[1], v[2], v[3], v[4], v[5]);
    }
}

// flux component q (cons order) of a FaceFlux
template <typename T>
__device__ __forceinline__ const T& flux_comp(const FaceFlux<0, T>& Fx, int q, int dim) {
    if (q == 0) return Fx.mass;
    if (q == dim + 1) return Fx.energy;
    return Fx.mom[q - 1];
}

// ---------------------------------------------------------------------------
// Reverse mode of the local operators, written out by hand: the product of a
// row vector with the Jacobian costs about three evaluations, where pushing
// 2 (dim + 2) (Riemann) or 5 (WENO) partial derivatives forwards costs 6 to 11.
// Every comparison acts as in the forward pass, so the derivative is that of
// the branch it took; sqrt and fabs at 0 have the zero subgradient.
// ---------------------------------------------------------------------------

// One side of a face and the adjoint of its primitives.
template <int DIM, typename S>
struct AdjSide {
    S r, u[DIM], p, E, c, un;        // state, total energy, sound speed, normal velocity
    S gr, gu[DIM], gp, gE, gc, gun;  // adjoints
};

template <int D, int DIM, typename S>
__device__ __forceinline__ void adj_side_init(const Params& P, const S* W, AdjSide<DIM, S>& a) {
    a.r = W[0];
    S k = S(0);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        a.u[d] = W[1 + d];
        k += a.u[d] * a.u[d];
        a.gu[d] = S(0);
    }
    a.p = W[DIM + 1];
    a.un = a.u[D];
    a.E = (a.p + S(P.gamma) * S(P.pInf)) / (S(P.gamma) - S(1)) + S(0.5) * a.r * k;
    a.c = ::sqrt(S(P.gamma) * smax(a.p + S(P.pInf), S(1e-14)) / smax(a.r, S(1e-14)));
    a.gr = a.gp = a.gE = a.gc = a.gun = S(0);
}

// adjoints of the energy, the sound speed and the normal velocity folded into
// the primitives'
template <int D, int DIM, typename S>
__device__ __forceinline__ void adj_side_finish(const Params& P, AdjSide<DIM, S>& a, S* g) {
    S k = S(0);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        k += a.u[d] * a.u[d];
        a.gu[d] += a.gE * a.r * a.u[d];
    }
    a.gu[D] += a.gun;
    a.gp += a.gE / (S(P.gamma) - S(1));
    a.gr += a.gE * S(0.5) * k;
    if (a.c > S(0)) {
        const S pp = a.p + S(P.pInf), h = S(0.5) * a.gc * a.c;
        if (!(pp < S(1e-14))) a.gp += h / pp;
        if (!(a.r < S(1e-14))) a.gr -= h / a.r;
    }
    g[0] = a.gr;
#pragma unroll
    for (int d = 0; d < DIM; ++d) g[1 + d] = a.gu[d];
    g[DIM + 1] = a.gp;
}

// w times m^T dF(W), F the physical flux along D (pressure included)
template <int D, int DIM, typename S>
__device__ __forceinline__ void adj_physical(const S* m, S w, AdjSide<DIM, S>& a) {
    S mu = S(0);
#pragma unroll
    for (int d = 0; d < DIM; ++d) mu += m[1 + d] * a.u[d];
    const S mE = m[DIM + 1];
    a.gr += w * a.un * (m[0] + mu);
#pragma unroll
    for (int d = 0; d < DIM; ++d) a.gu[d] += w * m[1 + d] * a.r * a.un;
    a.gun += w * (a.r * (m[0] + mu) + mE * (a.E + a.p));
    a.gp += w * (m[1 + D] + mE * a.un);
    a.gE += w * mE * a.un;
}

// w times m^T dU(W), U the conservative state
template <int DIM, typename S>
__device__ __forceinline__ void adj_conserved(const S* m, S w, AdjSide<DIM, S>& a) {
    S mu = S(0);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        mu += m[1 + d] * a.u[d];
        a.gu[d] += w * m[1 + d] * a.r;
    }
    a.gr += w * (m[0] + mu);
    a.gE += w * m[DIM + 1];
}

template <typename S>
__device__ __forceinline__ S adj_sign(S x) { return (x > S(0)) ? S(1) : (x < S(0)) ? S(-1) : S(0); }

// m^T dF of the Rusanov (src/RusanovSolver.cpp:7-83) and LF
// (src/LFSolver.cpp:8-75) fluxes: F = (F_L + F_R) / 2 - s (U_R - U_L) / 2.
template <int D, int DIM, typename S>
__device__ __forceinline__ void adj_central(bool lf, const S* m, AdjSide<DIM, S>& L, AdjSide<DIM, S>& R) {
    S s, gs = m[0] * (R.r - L.r) + m[DIM + 1] * (R.E - L.E);
#pragma unroll
    for (int d = 0; d < DIM; ++d) gs += m[1 + d] * (R.r * R.u[d] - L.r * L.u[d]);
    gs *= S(-0.5);
    if (lf) {
        S vL = S(0), vR = S(0);
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            vL += L.u[d] * L.u[d];
            vR += R.u[d] * R.u[d];
        }
        vL = ::sqrt(vL);
        vR = ::sqrt(vR);
        s = smax(vL, vR) + smax(L.c, R.c);
        AdjSide<DIM, S>& V = (vL < vR) ? R : L;
        const S v = (vL < vR) ? vR : vL;
        if (v > S(0)) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) V.gu[d] += gs * V.u[d] / v;
        }
        if (L.c < R.c) R.gc += gs; else L.gc += gs;
    } else {
        const S sL = ::fabs(L.un) + L.c, sR = ::fabs(R.un) + R.c;
        s = smax(sL, sR);
        if (sL < sR) { R.gun += gs * adj_sign(R.un); R.gc += gs; }
        else { L.gun += gs * adj_sign(L.un); L.gc += gs; }
    }
    adj_physical<D>(m, S(0.5), L);
    adj_physical<D>(m, S(0.5), R);
    adj_conserved(m, S(0.5) * s, L);
    adj_conserved(m, S(-0.5) * s, R);
}

// m^T dF of the HLLC flux (src/HLLCSolver.cpp:7-161).
template <int D, int DIM, typename S>
__device__ __forceinline__ void adj_hllc(const S* m, AdjSide<DIM, S>& L, AdjSide<DIM, S>& R) {
    const S aL = L.un - L.c, bL = R.un - R.c, aR = L.un + L.c, bR = R.un + R.c;
    const S sL = smin(aL, bL), sR = smax(aR, bR);
    if (sL >= S(0)) { adj_physical<D>(m, S(1), L); return; }
    const S dL = sL - L.un, dR = sR - R.un;
    const S den = L.r * dL - R.r * dR;
    const S sS = (R.p - L.p + L.r * L.un * dL - R.r * R.un * dR) / den;
    if (sR <= S(0)) { adj_physical<D>(m, S(1), R); return; }
    const bool left = sS >= S(0);
    // star state of side K with wave speed s
    S gs = S(0), gS = S(0);
    auto star = [&](AdjSide<DIM, S>& K, S s) {
        const S u = K.un, a = s - u, ib = S(1) / (s - sS), rS = K.r * a * ib, mE = m[DIM + 1];
        const S ir = S(1) / K.r, ia = S(1) / a;
        const S h = sS + K.p * ir * ia, e = K.E * ir, q = sS - u;
        const S ES = rS * (e + q * h);
        // mass
        S grS = m[0] * s;
        K.gr += m[0] * (u - s);
        K.gun += m[0] * K.r;
        gs += m[0] * (rS - K.r);
        // momentum
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const S md = m[1 + d], w = (d == D) ? K.u[d] + q : K.u[d];
            K.gr += md * K.u[d] * (u - s);
            K.gu[d] += md * (K.r * (u - s) + s * rS);
            K.gun += md * K.r * K.u[d];
            gs += md * (rS * w - K.r * K.u[d]);
            grS += md * s * w;
        }
        K.gp += m[1 + D];
        gS += m[1 + D] * s * rS;
        K.gun -= m[1 + D] * s * rS;
        // energy
        const S gES = mE * s;
        K.gE += mE * (u - s);
        K.gp += mE * u;
        K.gun += mE * (K.E + K.p);
        gs += mE * (ES - K.E);
        grS += gES * (e + q * h);
        const S t = gES * rS;
        gS += t * (h + q);
        K.gun -= t * h;
        const S gh = t * q * ir * ia;
        K.gp += gh;
        K.gr -= gh * K.p * ir;
        S ga = -gh * K.p * ia;
        K.gE += t * ir;
        K.gr -= t * e * ir;
        // r* = r a / b
        K.gr += grS * a * ib;
        ga += grS * K.r * ib;
        const S gb = -grS * rS * ib;
        gs += ga + gb;
        K.gun -= ga;
        gS -= gb;
    };
    if (left) star(L, sL); else star(R, sR);
    // contact speed s* = num / den
    const S gn = gS / den, gd = -gn * sS;
    L.gp -= gn;
    R.gp += gn;
    L.gr += dL * (gn * L.un + gd);
    R.gr -= dR * (gn * R.un + gd);
    const S hL = L.r * (gn * L.un + gd), hR = -R.r * (gn * R.un + gd);   // adjoints of s_L - u_L, s_R - u_R
    L.gun += gn * L.r * dL - hL;
    R.gun -= gn * R.r * dR + hR;
    const S gsL = hL + (left ? gs : S(0)), gsR = hR + (left ? S(0) : gs);
    if (bL < aL) { R.gun += gsL; R.gc -= gsL; } else { L.gun += gsL; L.gc -= gsL; }
    if (aR < bR) { R.gun += gsR; R.gc += gsR; } else { L.gun += gsR; L.gc += gsR; }
}

// Both face values of the cell v[2] (hi: its high face, weno5Left; lo: its low
// face, weno5Right).  The smoothness indicators of the two are the same three
// numbers in mirror order.
template <typename S>
struct AdjRecon {
    S t[3], s[3], ie[3], w[3];   // differences, 1 / (eps + b), its square
};

template <typename S>
__device__ __forceinline__ void adj_indicators(const S* v, S eps, AdjRecon<S>& q) {
    q.t[0] = v[0] - S(2) * v[1] + v[2];
    q.s[0] = v[0] - S(4) * v[1] + S(3) * v[2];
    q.t[1] = v[1] - S(2) * v[2] + v[3];
    q.s[1] = v[1] - v[3];
    q.t[2] = v[2] - S(2) * v[3] + v[4];
    q.s[2] = S(3) * v[2] - S(4) * v[3] + v[4];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const S b = S(13.0 / 12.0) * q.t[k] * q.t[k] + S(0.25) * q.s[k] * q.s[k];
        q.ie[k] = frcp(eps + b);
        q.w[k] = q.ie[k] * q.ie[k];
    }
}

// the three candidates of the high-face value; of the low-face value for the
// reversed stencil
template <typename S>
__device__ __forceinline__ void adj_candidates(S a, S b, S c, S d, S e, S* p) {
    const S k = S(1.0 / 6.0);
    p[0] = k * (S(2) * a - S(7) * b + S(11) * c);
    p[1] = k * (S(5) * c - b + S(2) * d);
    p[2] = k * (S(2) * c + S(5) * d - e);
}

template <typename S>
__device__ __forceinline__ void adj_values(bool weno, S eps, const S* v, S& hi, S& lo) {
    S p[3], q[3];
    adj_candidates(v[0], v[1], v[2], v[3], v[4], p);
    adj_candidates(v[4], v[3], v[2], v[1], v[0], q);
    if (!weno) {
        hi = S(0.1) * p[0] + S(0.6) * p[1] + S(0.3) * p[2];
        lo = S(0.1) * q[0] + S(0.6) * q[1] + S(0.3) * q[2];
        return;
    }
    AdjRecon<S> R;
    adj_indicators(v, eps, R);
    const S h0 = S(0.1) * R.w[0], m1 = S(0.6) * R.w[1], h2 = S(0.3) * R.w[2];
    const S l0 = S(0.1) * R.w[2], l2 = S(0.3) * R.w[0];
    hi = (h0 * p[0] + m1 * p[1] + h2 * p[2]) * frcp(h0 + m1 + h2);
    lo = (l0 * q[0] + m1 * q[1] + l2 * q[2]) * frcp(l0 + m1 + l2);
}

// g[k]: share of stencil cell k in gh d(hi) + gl d(lo)
template <typename S>
__device__ __forceinline__ void adj_recon(bool weno, S eps, const S* v, S gh, S gl, S* g) {
    S p[3], q[3], cp[3], cq[3], gb[3] = {S(0), S(0), S(0)};
    AdjRecon<S> R;
    if (weno) {
        adj_candidates(v[0], v[1], v[2], v[3], v[4], p);
        adj_candidates(v[4], v[3], v[2], v[1], v[0], q);
        adj_indicators(v, eps, R);
        const S h[3] = {S(0.1) * R.w[0], S(0.6) * R.w[1], S(0.3) * R.w[2]};
        const S l[3] = {S(0.1) * R.w[2], h[1], S(0.3) * R.w[0]};
        const S ih = frcp(h[0] + h[1] + h[2]), il = frcp(l[0] + l[1] + l[2]);
        const S hi = (h[0] * p[0] + h[1] * p[1] + h[2] * p[2]) * ih;
        const S lo = (l[0] * q[0] + l[1] * q[1] + l[2] * q[2]) * il;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            cp[k] = gh * h[k] * ih;
            cq[k] = gl * l[k] * il;
            gb[k] -= S(2) * cp[k] * (p[k] - hi) * R.ie[k];
            gb[2 - k] -= S(2) * cq[k] * (q[k] - lo) * R.ie[2 - k];
        }
    } else {
        cp[0] = S(0.1) * gh; cp[1] = S(0.6) * gh; cp[2] = S(0.3) * gh;
        cq[0] = S(0.1) * gl; cq[1] = S(0.6) * gl; cq[2] = S(0.3) * gl;
    }
    const S k6 = S(1.0 / 6.0);
    g[0] = k6 * (S(2) * cp[0] - cq[2]);
    g[1] = k6 * (S(-7) * cp[0] - cp[1] + S(2) * cq[1] + S(5) * cq[2]);
    g[2] = k6 * (S(11) * (cp[0] + cq[0]) + S(5) * (cp[1] + cq[1]) + S(2) * (cp[2] + cq[2]));
    g[3] = k6 * (S(-7) * cq[0] - cq[1] + S(2) * cp[1] + S(5) * cp[2]);
    g[4] = k6 * (S(2) * cq[0] - cp[2]);
    if (weno) {
        const S t0 = gb[0] * S(13.0 / 6.0) * R.t[0], s0 = gb[0] * S(0.5) * R.s[0];
        const S t1 = gb[1] * S(13.0 / 6.0) * R.t[1], s1 = gb[1] * S(0.5) * R.s[1];
        const S t2 = gb[2] * S(13.0 / 6.0) * R.t[2], s2 = gb[2] * S(0.5) * R.s[2];
        g[0] += t0 + s0;
        g[1] += t1 + s1 - S(2) * t0 - S(4) * s0;
        g[2] += t0 + t2 - S(2) * t1 + S(3) * (s0 + s2);
        g[3] += t1 - s1 - S(2) * t2 - S(4) * s2;
        g[4] += t2 + s2;
    }
}

// ---------------------------------------------------------------------------
// Reverse of one direction: dJ/dW of every cell of a grid line, ghost
// positions -3 .. n + 2 included, from the faces of that direction.
//
// A block owns four grid lines and 58 positions along them: it converts the
// positions and five more on either side to primitives, reconstructs 64 cells
// per line, turns dJ/dF into dJ/d(face values) on the 63 faces between them,
// and gathers the reconstructions' transposes; everything between the stage
// input and dJ/dW stays in shared memory.  Against two kernels that write each
// face's ten stencil shares per variable out and gather them again, with the
// Jacobians by forward duals and a device allocation per checkpoint: value
// and gradient of 12 steps at 256^2, 8.9 -> 3.75 ms.
// S: the arithmetic of the local Jacobians (double, or float for the FP32
// reverse sweep, whose sums over the stencils are still formed in FP64).
// ---------------------------------------------------------------------------
constexpr int kAdjLines = 4, kAdjLen = 64, kAdjOut = kAdjLen - 6, kAdjStride = 72;

template <int DIM, typename S>
__host__ __device__ constexpr size_t adj_dir_smem() {
    return ((size_t)3 * NV<DIM>::n * sizeof(S) + 2 * 5 * sizeof(double)) * kAdjLines * kAdjStride;
}

template <int D, int DIM, typename S>
__device__ __forceinline__ void adj_dir(const AdjArgs& A, unsigned char* smem) {
    constexpr int NVN = NV<DIM>::n, LS = kAdjLines * kAdjStride;
    const Params& P = A.P;
    const int n = (D == 0) ? P.nx : (D == 1) ? P.ny : P.nz;
    const unsigned block = blockIdx.x - A.adjFirst[D];
    const int p0 = -3 + (int)(block % A.adjTiles[D]) * kAdjOut;
    double* const sSh = reinterpret_cast<double*>(smem);       // two buffers of five shares per cell
    S* const sW = reinterpret_cast<S*>(sSh + 2 * 5 * LS);      // primitives at p0 - 5 + index
    S* const sHi = sW + NVN * LS;                              // face values of cell p0 - 3 + index, then
    S* const sLo = sHi + NVN * LS;                             // their adjoints
    // grid line of each thread: consecutive lines are consecutive in memory for D > 0
    const int nt0 = (D == 0) ? P.ny : P.nx;                                    // faster transverse axis
    const long long nLines = (long long)nt0 * ((D == 2) ? P.ny : P.nz);
    const int l = (D == 0) ? (int)threadIdx.x / kAdjLen : (int)threadIdx.x % kAdjLines;
    const int a = (D == 0) ? (int)threadIdx.x % kAdjLen : (int)threadIdx.x / kAdjLines;
    const long long line = (long long)(block / A.adjTiles[D]) * kAdjLines + l;
    const bool on = line < nLines;
    const int q0 = on ? (int)(line % nt0) : 0, q1 = on ? (int)(line / nt0) : 0;
    auto cell = [&](int c, int& i, int& j, int& k) {
        i = (D == 0) ? c : q0;
        j = (D == 0) ? q0 : (D == 1) ? c : q1;
        k = (D == 2) ? c : q1;
    };
    const int row = l * kAdjStride;

    // ---- primitives (cons_to_prim_cell, PRIM ghost map) ----
    for (int x = a; x < kAdjLen + 4; x += kAdjLen) {
        const int e = p0 - 5 + x;
        if (!on || e < -3 || e >= n + 3) continue;
        int i, j, k;
        cell(e, i, j, k);
        double sg[3], rho, u[3], p;
        const size_t s = prim_source(P, i, j, k, sg);
        cons_to_prim_cell<0>(P, A.F, s, rho, u, p);
        sW[row + x] = (S)rho;
#pragma unroll
        for (int d = 0; d < DIM; ++d) sW[(1 + d) * LS + row + x] = (S)(sg[d] * u[d]);
        sW[(DIM + 1) * LS + row + x] = (S)p;
    }
    __syncthreads();

    // ---- face values of cell c = p0 - 3 + a ----
    const int c = p0 - 3 + a;
    const bool rec = on && c >= -1 && c <= n;
    const bool weno = (P.reconOrder == SIFV_WENO5);
    const S eps = (S)P.wenoEps;
    if (rec) {
#pragma unroll 1
        for (int v = 0; v < NVN; ++v) {
            const S* w = sW + v * LS + row + a;
            S x[5] = {w[0], w[1], w[2], w[3], w[4]};
            adj_values(weno, eps, x, sHi[v * LS + row + a], sLo[v * LS + row + a]);
        }
    }
    __syncthreads();

    // ---- the face below cell c: adjoints in place of the two values it read ----
    if (a >= 1) {
        S gl[NVN], gr[NVN];
        if (on && c >= 0 && c <= n) {
            S mu[NVN], WL[NVN], WR[NVN];
            {
                const bool rIn = c < n, lIn = c >= 1;
                int i, j, k, li, lj, lk;
                cell(c, i, j, k);
                cell(c - 1, li, lj, lk);
                const size_t cr = cidx(P, i, j, k), cl = cidx(P, li, lj, lk);
                const double fR = rIn ? face_coeff<D>(P, A.F, i, j, k) : 0.0;
                const double fL = lIn ? face_coeff<D>(P, A.F, li, lj, lk) : 0.0;
#pragma unroll
                for (int q = 0; q < NVN; ++q) {
                    const double lr = rIn ? A.lam[q][cr] : 0.0, ll = lIn ? A.lam[q][cl] : 0.0;
                    mu[q] = (S)(fR * lr - fL * ll);
                    WL[q] = sHi[q * LS + row + a - 1];
                    WR[q] = sLo[q * LS + row + a];
                }
            }
            AdjSide<DIM, S> L, R;
            adj_side_init<D>(P, WL, L);
            adj_side_init<D>(P, WR, R);
            if (P.riemann == SIFV_HLLC) adj_hllc<D>(mu, L, R);
            else adj_central<D>(P.riemann == SIFV_LF, mu, L, R);
            adj_side_finish<D>(P, L, gl);
            adj_side_finish<D>(P, R, gr);
        } else {
#pragma unroll
            for (int q = 0; q < NVN; ++q) gl[q] = gr[q] = S(0);
        }
#pragma unroll
        for (int q = 0; q < NVN; ++q) {
            sHi[q * LS + row + a - 1] = gl[q];
            sLo[q * LS + row + a] = gr[q];
        }
    }
    __syncthreads();

    // ---- transposed reconstructions, gathered per position ----
    const bool out = on && a >= 3 && a < kAdjLen - 3 && c < n + 3;
    size_t dst = 0;
    if (out) {
        int i, j, k;
        cell(c, i, j, k);
        dst = cidx(P, i, j, k);
    }
#pragma unroll 1
    for (int v = 0; v < NVN; ++v) {
        double* const sh = sSh + (v & 1) * 5 * LS + row + a;
        if (a >= 1 && a < kAdjLen - 1) {
            S g[5] = {S(0), S(0), S(0), S(0), S(0)};
            if (rec) {
                const S* w = sW + v * LS + row + a;
                const S x[5] = {w[0], w[1], w[2], w[3], w[4]};
                adj_recon(weno, eps, x, sHi[v * LS + row + a], sLo[v * LS + row + a], g);
            }
#pragma unroll
            for (int q = 0; q < 5; ++q) sh[q * LS] = (double)g[q];
        }
        __syncthreads();
        if (out) {
            double sum = 0.0;
#pragma unroll
            for (int q = 0; q < 5; ++q) sum += sh[q * LS + 2 - q];   // stencil entry q of cell c + 2 - q is c
            A.gdir[D][v][dst] = sum;
        }
    }
}

template <int DIM, typename S>
__global__ void __launch_bounds__(kAdjLines * kAdjLen, 2) k_adj_dir(const __grid_constant__ AdjArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    if (DIM == 1 || blockIdx.x < A.adjFirst[1]) adj_dir<0, DIM, S>(A, smem);
    else if (DIM == 2 || blockIdx.x < A.adjFirst[2]) adj_dir<(DIM >= 2) ? 1 : 0, DIM, S>(A, smem);
    else adj_dir<(DIM >= 3) ? 2 : 0, DIM, S>(A, smem);
}

// ghost images of interior index c along one axis: positions g in the
// three ghost layers the stencils reach whose PRIM source is c (with the
// axis's sn, sa), after c itself
__device__ __forceinline__ int axis_images(int c, int n, int bcLo, int bcHi, int* pos, double* sn, double* sa) {
    int m = 0;
    pos[m] = c; sn[m] = 1.0; sa[m] = 1.0; ++m;
    if (c >= 3 && c < n - 3) return m;
    for (int g = -3; g < 0; ++g) {
        double a, b;
        if (prim_src(g, n, bcLo, bcHi, a, b) == c) { pos[m] = g; sn[m] = a; sa[m] = b; ++m; }
    }
    for (int g = n; g < n + 3; ++g) {
        double a, b;
        if (prim_src(g, n, bcLo, bcHi, a, b) == c) { pos[m] = g; sn[m] = a; sa[m] = b; ++m; }
    }
    return m;
}

// dJ/dW of an interior cell from direction D: its own entry and those of its
// ghost images along D (faces exist only at interior transverse positions)
template <int D, int DIM>
__device__ __forceinline__ void gather_dir(const AdjArgs& A, int i, int j, int k, double* gW) {
    const Params& P = A.P;
    int pos[7];
    double sn[7], sa[7];
    const int m = (D == 0) ? axis_images(i, P.nx, P.bc[0], P.bc[1], pos, sn, sa)
                : (D == 1) ? axis_images(j, P.ny, P.bc[2], P.bc[3], pos, sn, sa)
                           : axis_images(k, P.nz, P.bc[4], P.bc[5], pos, sn, sa);
    for (int q = 0; q < m; ++q) {
        const size_t s = cidx(P, (D == 0) ? pos[q] : i, (D == 1) ? pos[q] : j, (D == 2) ? pos[q] : k);
        double* const* g = A.gdir[D];
        gW[0] += g[0][s];
#pragma unroll
        for (int d = 0; d < DIM; ++d) gW[1 + d] += ((d == D) ? sn[q] * sa[q] : sa[q]) * g[1 + d][s];
        gW[DIM + 1] += g[DIM + 1][s];
    }
}

template <int DIM>
__global__ void __launch_bounds__(128) k_adj_cell(const __grid_constant__ AdjArgs A) {
    constexpr int NVN = NV<DIM>::n;
    const Params& P = A.P;
    const Fields& F = A.F;
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int i, j, k;
    if (!int_coords(P, t, i, j, k)) return;
    const size_t c = cidx(P, i, j, k);
    double gW[NVN];
#pragma unroll
    for (int v = 0; v < NVN; ++v) gW[v] = 0.0;
    gather_dir<0, DIM>(A, i, j, k, gW);
    if (DIM >= 2) gather_dir<(DIM >= 2) ? 1 : 0, DIM>(A, i, j, k, gW);
    if (DIM >= 3) gather_dir<(DIM >= 3) ? 2 : 0, DIM>(A, i, j, k, gW);
    // cons -> prim Jacobian (IdealGasEOS / StiffenedGasEOS::toPrimitive):
    // rho_W = rho; u = m / max(rho, 1e-14); ke = 0.5 r sum u^2;
    // p = (g - 1)(E - ke) [- g pInf]  (ideal: max(., 1e-14))
    const double rho = F.rho[c];
    const bool rAct = rho > 1e-14;
    const double r = rAct ? rho : 1e-14;
    double u[3] = {0.0, 0.0, 0.0}, u2 = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        u[d] = cons_ptr(F, 1 + d, DIM)[c] / r;
        u2 += u[d] * u[d];
    }
    const double gm1 = P.gamma - 1.0;
    bool pAct = true;
    if (!P.eosStiffened) {
        double e = F.rhoE[c] - 0.5 * r * u2;
        pAct = gm1 * e > 1e-14;
    }
    const double gp = pAct ? gW[DIM + 1] : 0.0;
    double g[NVN];
    g[0] = gW[0] + (rAct ? gp * gm1 * 0.5 * u2 : 0.0);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        if (rAct) g[0] -= gW[1 + d] * u[d] / r;
        g[1 + d] = gW[1 + d] / r - gp * gm1 * u[d];
    }
    g[DIM + 1] = gp * gm1;
    // RK combination
#pragma unroll
    for (int q = 0; q < NVN; ++q) {
        const double lin = A.lam[q][c];
        double ln = A.a1 * lin + A.a3 * A.dt * g[q];
        double a0 = A.acc0[q][c] + A.a2 * lin;
        if (A.stage0) {
            ln += a0;
            a0 = 0.0;
        }
        A.lam[q][c] = ln;
        A.acc0[q][c] = a0;
    }
}

// ---------------------------------------------------------------------------
// Tangent (forward mode).  A device-resident run queues steps past its end
// time that the state kernels skip; so do these (A.skip).
// ---------------------------------------------------------------------------
// dW of every cell (ghosts: the source cell's dW with the velocity signs)
template <int DIM>
__global__ void __launch_bounds__(256) k_tan_prim(AdjArgs A) {
    if (A.skip && *A.skip) return;
    const Params& P = A.P;
    const Fields& F = A.F;
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int i, j, k;
    if (!ext_coords(P, t, i, j, k)) return;
    const size_t d = cidx(P, i, j, k);
    double sg[3] = {1.0, 1.0, 1.0};
    const size_t s = is_interior(P, i, j, k) ? d : prim_source(P, i, j, k, sg);
    const double rho = F.rho[s];
    const bool rAct = rho > 1e-14;
    const double r = rAct ? rho : 1e-14;
    double u[3] = {0.0, 0.0, 0.0}, u2 = 0.0;
#pragma unroll
    for (int q = 0; q < DIM; ++q) {
        u[q] = cons_ptr(F, 1 + q, DIM)[s] / r;
        u2 += u[q] * u[q];
    }
    const double gm1 = P.gamma - 1.0;
    bool pAct = true;
    if (!P.eosStiffened) pAct = gm1 * (F.rhoE[s] - 0.5 * r * u2) > 1e-14;
    const double dr = A.tan[0][s];
    double dp = A.tan[DIM + 1][s] + (rAct ? 0.5 * u2 * dr : 0.0);
    A.tanW[0][d] = dr;
#pragma unroll
    for (int q = 0; q < DIM; ++q) {
        const double dm = A.tan[1 + q][s];
        double du = dm / r - (rAct ? u[q] * dr / r : 0.0);
        dp -= u[q] * dm;
        A.tanW[1 + q][d] = sg[q] * du;
    }
    A.tanW[DIM + 1][d] = pAct ? gm1 * dp : 0.0;
}

template <int DIR, int DIM>
__global__ void __launch_bounds__(128) k_tan_face(AdjArgs A) {
    if (A.skip && *A.skip) return;
    constexpr int NVN = NV<DIM>::n;
    const Params& P = A.P;
    const Fields& F = A.F;
    const int fnx = P.nx + (DIR == 0), fny = P.ny + (DIR == 1), fnz = P.nz + (DIR == 2);
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long tot = (long long)fnx * fny * fnz;
    if (t >= tot) return;
    int i, j, k;
    split3(t, fnx, fny, i, j, k);
    const size_t base = cidx(P, i, j, k);
    const long st = (DIR == 0) ? 1L : (DIR == 1) ? (long)P.nxT : (long)P.nxT * P.nyT;
    const bool weno = (P.reconOrder == SIFV_WENO5);
    const int dim = DIM;
    Dual<1> WL[NVN], WR[NVN];
#pragma unroll
    for (int v = 0; v < NVN; ++v) {
        const double* f = prim_ptr(F, v, dim);
        const double* df = A.tanW[v];
        Dual<1> s[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            s[q].v = f[base + (q - 3) * st];
            s[q].d[0] = df[base + (q - 3) * st];
        }
        recon5<Dual<1>>(weno, P.wenoEps, s, WL[v], WR[v]);
    }
    FaceState<0, Dual<1>> L, R;
    L.rho = WL[0];
    R.rho = WR[0];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        L.u[d] = (d < DIM) ? WL[1 + d] : Dual<1>(0.0);
        R.u[d] = (d < DIM) ? WR[1 + d] : Dual<1>(0.0);
    }
    L.p = WL[DIM + 1];
    R.p = WR[DIM + 1];
    L.sigma = R.sigma = Dual<1>(0.0);
    L.gEff = R.gEff = Dual<1>(P.gamma);
    L.piEff = R.piEff = Dual<1>(P.pInf);
    FaceFlux<0, Dual<1>> Fx;
    riemann_T<DIR, Dual<1>>(P, L, R, Fx);
#pragma unroll
    for (int q = 0; q < NVN; ++q) A.tanF[DIR][q][t] = flux_comp(Fx, q, dim).d[0];
}

template <int DIM>
__global__ void __launch_bounds__(256) k_tan_update(AdjArgs A, int save) {
    if (A.skip && *A.skip) return;
    constexpr int NVN = NV<DIM>::n;
    const Params& P = A.P;
    const Fields& F = A.F;
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int i, j, k;
    if (!int_coords(P, t, i, j, k)) return;
    const size_t c = cidx(P, i, j, k);
    const double dt = A.dtDev ? *A.dtDev : A.dt;
    double dR[NVN];
#pragma unroll
    for (int q = 0; q < NVN; ++q) dR[q] = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        const double co = (d == 0) ? face_coeff<0>(P, F, i, j, k)
                          : (d == 1) ? face_coeff<1>(P, F, i, j, k) : face_coeff<2>(P, F, i, j, k);
        const long long lo = (d == 0) ? face_index<0>(P, i, j, k)
                             : (d == 1) ? face_index<1>(P, i, j, k) : face_index<2>(P, i, j, k);
        const long long hi = (d == 0) ? face_index<0>(P, i + 1, j, k)
                             : (d == 1) ? face_index<1>(P, i, j + 1, k) : face_index<2>(P, i, j, k + 1);
#pragma unroll
        for (int q = 0; q < NVN; ++q) dR[q] += co * A.tanF[d][q][lo] - co * A.tanF[d][q][hi];
    }
#pragma unroll
    for (int q = 0; q < NVN; ++q) {
        const double du = A.tan[q][c];
        if (save) A.tan0[q][c] = du;
        const double du0 = (A.a2 != 0.0) ? A.tan0[q][c] : 0.0;
        A.tan[q][c] = A.a1 * du + A.a2 * du0 + A.a3 * dt * dR[q];
    }
}

}  // namespace sifv
