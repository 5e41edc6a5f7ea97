// sifv_mg.cuh -- conjugate gradients preconditioned by one geometric
// multigrid V-cycle for the semi-implicit pressure system, the solver the
// reference offers through Hypre (HyprePressureSolver: PCG with one PFMG
// V-cycle of weighted-Jacobi relaxation as preconditioner, two-norm
// relative-residual stopping, src/HyprePressureSolver.cpp:124-139, 360-381).
//
// System (HyprePressureSolver::assembleSystem, src/HyprePressureSolver.cpp:154-279):
//   (1 + c_i sum_f k_f) p_i - c_i sum_f k_f p_nb(f) = rhs_i,
//   c_i = rhoc2_i dt^2,  k_f = 1 / (max(rho_f, 1e-14) d_f w_i),
// with k_f = 0 on physical (non-periodic) boundary faces.  Row i multiplied
// by m_i = vol_i / c_i gives a symmetric positive definite form
//   (m_i + sum_f T_f) p_i - sum_f T_f p_nb = m_i rhs_i,
//   T_f = A_f / (max(rho_f, 1e-14) d_f)  (one value per face),
// on which CG runs; convergence is tested on the unscaled residual
// (r_i / m_i), as Hypre tests its own system.
//
// Level layout: compact x-fastest arrays without ghosts.  tx[c] is T of the
// low-x face of cell c (the face to c - 1, wrapped on periodic axes, 0 on a
// physical boundary); the high-x face of c is tx of c + 1 (wrapped: for a
// physical boundary that is tx of cell 0, which is 0).  Coarse levels halve
// every axis longer than 1 (ceil), aggregate 2^dim cells, and take the
// Galerkin operator of piecewise-constant transfer: summed masses, summed
// face T across each coarse face.
//
// Launches.  On the meshes this solver is for, the levels below the first two
// or three are launch latency, not work.  A V-cycle is therefore one kernel
// down and one up per large level (relaxation from zero, residual and
// restriction; prolongation and relaxation: what they pass between their
// steps is recomputed at the neighbours from b and omega / diag instead of
// being stored), and one single-block kernel for every level of at most
// kMgTail cells.  The conjugate-gradient step is two kernels (direction +
// product, update); their dot products, and the V-cycle's r.z, are summed by
// the last block to finish, in a fixed order.  Convergence is decided on the
// device: kernels queued past it return at once, so the host looks once per
// batch of iterations.  150 x 96 x 77, 13 iterations: 4.05 -> 2.2 ms against
// one launch per operation with the host looking at every iteration.
#pragma once

#include "sifv_common.cuh"

namespace sifv {

struct MgLevel {
    int nx, ny, nz;
    int n;
    double *m, *tx, *ty, *tz, *diag;
    double* iw;          // omega / diag
    double *x, *b;
};

constexpr double kMgOmega = 0.8;       // weighted-Jacobi relaxation
constexpr int kMgCoarsestSweeps = 60;  // relaxation sweeps on the coarsest level
constexpr int kMgCoarsest = 256;       // cells of the coarsest level, at most (or 2 per axis)
constexpr int kMgTail = 4096;          // levels up to this size run in one block
constexpr int kMgMaxLevels = 24;

// Scalars of a solve on the device.
struct CgState {
    double rz[2];        // r.z of this iteration and the next (by parity)
    double pq, rr, bb;   // p.q, |r/m|^2, |rhs|^2
    double eps;          // tol^2
    int done;            // converged (or NaN): every kernel returns
    int iters;
    unsigned count, count2;   // blocks finished (grid_sum)
};

__device__ __forceinline__ void mg_split(const MgLevel& L, int c, int& i, int& j, int& k) {
    const unsigned q = (unsigned)c / (unsigned)L.nx;
    i = c - (int)q * L.nx;
    k = (int)(q / (unsigned)L.ny);
    j = (int)q - k * L.ny;
}

// Sum of v over the grid in a fixed order: the block's sum to partial, and in
// the block that finishes last the sum of the partials.  True in that block's
// thread 0, with the total in *total.
__device__ __forceinline__ bool grid_sum(double v, double* partial, unsigned* count, double* total) {
    __shared__ double sm[32];
    __shared__ bool lastBlock;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    auto block_sum = [&](double x) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        __syncthreads();
        if (lane == 0) sm[w] = x;
        __syncthreads();
        x = (lane < nw) ? sm[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        return x;
    };
    v = block_sum(v);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = v;
        __threadfence();
        lastBlock = atomicAdd(count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!lastBlock) return false;
    __threadfence();
    double s = 0.0;
    for (unsigned q = threadIdx.x; q < gridDim.x; q += blockDim.x) s += __ldcg(partial + q);
    s = block_sum(s);
    if (threadIdx.x != 0) return false;
    *count = 0;
    *total = s;
    return true;
}

// Fine level from the context's state: masses, face T, diagonal, the scaled
// right-hand side b = m rhs, the initial guess x = p (interior).  dt from the
// control block.
__global__ void __launch_bounds__(256) k_mg_fine(Params P, Fields F, const double* __restrict__ rho,
                                                 const double* __restrict__ rhoc2, const double* __restrict__ rhs,
                                                 const double* __restrict__ p0, const Ctl* __restrict__ ctl, MgLevel L,
                                                 double* __restrict__ wInv) {
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (t >= L.n) return;
    int i, j, k;
    mg_split(L, t, i, j, k);
    const int dim = P.dim;
    const size_t c = cidx(P, i, j, k);
    const double dt = ctl->dt;
    const double dxi = F.dx[i + P.ngx], dyj = F.dy[j + P.ngy], dzk = F.dz[k + P.ngz];
    const double vol = dxi * dyj * dzk;
    const double coeff = rhoc2[c] * (dt * dt);
    const double m = vol / coeff;
    L.m[t] = m;
    wInv[t] = 1.0 / m;
    L.b[t] = m * rhs[c];
    L.x[t] = p0[c];
    // T of the face between the cells q - 1 and q of one axis, area A, widths w, cell stride st
    auto face = [&](int q, int n, int bcLo, size_t cell, size_t st, double A, const double* w) {
        if ((q == 0 || q == n) && bcLo != SIFV_BC_PERIODIC) return 0.0;
        const double rf = 0.5 * (rho[cell] + rho[cell - st]);
        const double d = 0.5 * (w[q - 1] + w[q]);
        return A / (smax(rf, 1e-14) * d);
    };
    // a periodic axis' high boundary face is its low one (one value per face)
    const size_t sx = 1, sy = (size_t)P.nxT, sz = (size_t)P.nxT * P.nyT;
    double lo = face(i, P.nx, P.bc[0], c, sx, dyj * dzk, F.dx + P.ngx);
    double hi = (i + 1 == P.nx) ? face(0, P.nx, P.bc[0], c - (size_t)i, sx, dyj * dzk, F.dx + P.ngx)
                                : face(i + 1, P.nx, P.bc[0], c + sx, sx, dyj * dzk, F.dx + P.ngx);
    L.tx[t] = lo;
    double diag = m + lo + hi;
    if (dim >= 2) {
        lo = face(j, P.ny, P.bc[2], c, sy, dxi * dzk, F.dy + P.ngy);
        hi = (j + 1 == P.ny) ? face(0, P.ny, P.bc[2], c - (size_t)j * sy, sy, dxi * dzk, F.dy + P.ngy)
                             : face(j + 1, P.ny, P.bc[2], c + sy, sy, dxi * dzk, F.dy + P.ngy);
        L.ty[t] = lo;
        diag = diag + lo + hi;
    }
    if (dim >= 3) {
        lo = face(k, P.nz, P.bc[4], c, sz, dxi * dyj, F.dz + P.ngz);
        hi = (k + 1 == P.nz) ? face(0, P.nz, P.bc[4], c - (size_t)k * sz, sz, dxi * dyj, F.dz + P.ngz)
                             : face(k + 1, P.nz, P.bc[4], c + sz, sz, dxi * dyj, F.dz + P.ngz);
        L.tz[t] = lo;
        diag = diag + lo + hi;
    }
    L.diag[t] = diag;
    L.iw[t] = kMgOmega / diag;
}

// Galerkin coarsening of piecewise-constant aggregates, cell t of Cs.
__device__ __forceinline__ void mg_coarsen(const MgLevel& Fn, const MgLevel& Cs, int dim, int t) {
    int I, J, K;
    mg_split(Cs, t, I, J, K);
    const int fx = (Fn.nx > 1) ? 2 : 1, fy = (Fn.ny > 1) ? 2 : 1, fz = (Fn.nz > 1) ? 2 : 1;
    auto at = [&](int i, int j, int k) { return i + Fn.nx * (j + Fn.ny * k); };
    double m = 0.0;
    // faces of the aggregate: low and high (the next aggregate's low face, wrapped)
    double xl = 0.0, xh = 0.0, yl = 0.0, yh = 0.0, zl = 0.0, zh = 0.0;
    const int In = (I + 1 == Cs.nx) ? 0 : I + 1, Jn = (J + 1 == Cs.ny) ? 0 : J + 1, Kn = (K + 1 == Cs.nz) ? 0 : K + 1;
    for (int c = 0; c < fz; ++c)
        for (int b = 0; b < fy; ++b)
            for (int a = 0; a < fx; ++a) {
                const int i = I * fx + a, j = J * fy + b, k = K * fz + c;
                if (i >= Fn.nx || j >= Fn.ny || k >= Fn.nz) continue;
                m += Fn.m[at(i, j, k)];
                if (a == 0) {
                    xl += Fn.tx[at(i, j, k)];
                    xh += Fn.tx[at(In * fx, j, k)];
                }
                if (dim >= 2 && b == 0) {
                    yl += Fn.ty[at(i, j, k)];
                    yh += Fn.ty[at(i, Jn * fy, k)];
                }
                if (dim >= 3 && c == 0) {
                    zl += Fn.tz[at(i, j, k)];
                    zh += Fn.tz[at(i, j, Kn * fz)];
                }
            }
    Cs.m[t] = m;
    Cs.tx[t] = xl;
    if (dim >= 2) Cs.ty[t] = yl;
    if (dim >= 3) Cs.tz[t] = zl;
    const double diag = m + xl + xh + yl + yh + zl + zh;
    Cs.diag[t] = diag;
    Cs.iw[t] = kMgOmega / diag;
}

__global__ void __launch_bounds__(256) k_mg_coarsen(MgLevel Fn, MgLevel Cs, int dim) {
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (t < Cs.n) mg_coarsen(Fn, Cs, dim, t);
}

// The neighbours of cell c and the T of its faces.
struct MgNb {
    int xm, xp, ym, yp, zm, zp;
};
__device__ __forceinline__ MgNb mg_nb(const MgLevel& L, int c, int i, int j, int k) {
    const int sy = L.nx, sz = L.nx * L.ny;
    MgNb q;
    q.xm = c + ((i == 0) ? (L.nx - 1) : -1);
    q.xp = c + ((i == L.nx - 1) ? -(L.nx - 1) : 1);
    q.ym = c + ((j == 0) ? (L.ny - 1) * sy : -sy);
    q.yp = c + ((j == L.ny - 1) ? -(L.ny - 1) * sy : sy);
    q.zm = c + ((k == 0) ? (L.nz - 1) * sz : -sz);
    q.zp = c + ((k == L.nz - 1) ? -(L.nz - 1) * sz : sz);
    return q;
}

// (M x)_c with x given by a function of the cell index.
template <typename X>
__device__ __forceinline__ double mg_apply(const MgLevel& L, int dim, int c, const MgNb& q, double xc, X x) {
    double off = L.tx[c] * x(q.xm) + L.tx[q.xp] * x(q.xp);
    if (dim >= 2) off += L.ty[c] * x(q.ym) + L.ty[q.yp] * x(q.yp);
    if (dim >= 3) off += L.tz[c] * x(q.zm) + L.tz[q.zp] * x(q.zp);
    return L.diag[c] * xc - off;
}

// Down: relaxation from zero (x = omega b / diag), residual, restriction into
// cell t of Cs.b.
__device__ __forceinline__ void mg_down(const MgLevel& L, const MgLevel& Cs, int dim, int t) {
    int I, J, K;
    mg_split(Cs, t, I, J, K);
    const int fx = (L.nx > 1) ? 2 : 1, fy = (L.ny > 1) ? 2 : 1, fz = (L.nz > 1) ? 2 : 1;
    auto x0 = [&](int c) { return L.iw[c] * L.b[c]; };
    double s = 0.0;
    for (int c = 0; c < fz; ++c)
        for (int b = 0; b < fy; ++b)
            for (int a = 0; a < fx; ++a) {
                const int i = I * fx + a, j = J * fy + b, k = K * fz + c;
                if (i >= L.nx || j >= L.ny || k >= L.nz) continue;
                const int f = i + L.nx * (j + L.ny * k);
                s += L.b[f] - mg_apply(L, dim, f, mg_nb(L, f, i, j, k), x0(f), x0);
            }
    Cs.b[t] = s;
}

// Up: prolongation onto the relaxed iterate and one relaxation of cell t.
__device__ __forceinline__ double mg_up(const MgLevel& L, const MgLevel& Cs, int dim, int t) {
    int i, j, k;
    mg_split(L, t, i, j, k);
    const int sx = (L.nx > 1) ? 1 : 0, sy = (L.ny > 1) ? 1 : 0, sz = (L.nz > 1) ? 1 : 0;
    auto parent = [&](int a, int b, int c) { return (a >> sx) + Cs.nx * ((b >> sy) + Cs.ny * (c >> sz)); };
    auto x1 = [&](int c, int a, int b, int d) { return L.iw[c] * L.b[c] + Cs.x[parent(a, b, d)]; };
    const MgNb q = mg_nb(L, t, i, j, k);
    const int im = (i == 0) ? L.nx - 1 : i - 1, ip = (i == L.nx - 1) ? 0 : i + 1;
    const double xc = x1(t, i, j, k);
    double off = L.tx[t] * x1(q.xm, im, j, k) + L.tx[q.xp] * x1(q.xp, ip, j, k);
    if (dim >= 2) {
        const int jm = (j == 0) ? L.ny - 1 : j - 1, jp = (j == L.ny - 1) ? 0 : j + 1;
        off += L.ty[t] * x1(q.ym, i, jm, k) + L.ty[q.yp] * x1(q.yp, i, jp, k);
    }
    if (dim >= 3) {
        const int km = (k == 0) ? L.nz - 1 : k - 1, kp = (k == L.nz - 1) ? 0 : k + 1;
        off += L.tz[t] * x1(q.zm, i, j, km) + L.tz[q.zp] * x1(q.zp, i, j, kp);
    }
    const double x = xc + L.iw[t] * (L.b[t] - (L.diag[t] * xc - off));
    L.x[t] = x;
    return x;
}

__global__ void __launch_bounds__(256) k_mg_down(MgLevel L, MgLevel Cs, int dim, const CgState* S) {
    grid_dep_launch();
    grid_dep_wait();
    if (S->done) return;
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (t < Cs.n) mg_down(L, Cs, dim, t);
}

// dot: level 0, whose r.z (b.x) goes to S->rz[slot].
__global__ void __launch_bounds__(256) k_mg_up(MgLevel L, MgLevel Cs, int dim, CgState* S, double* partial, int dot,
                                               int slot) {
    grid_dep_launch();
    grid_dep_wait();
    if (S->done) return;
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    double v = 0.0;
    if (t < L.n) {
        const double x = mg_up(L, Cs, dim, t);
        if (dot) v = L.b[t] * x;
    }
    if (dot) {
        double total;
        if (grid_sum(v, partial, &S->count, &total)) S->rz[slot] = total;
    }
}

struct MgTail {
    MgLevel l[kMgMaxLevels];
    int first, n;        // levels first .. n - 1 run in the block; n levels in all
};

// The operator of the tail's levels below its first.
__global__ void __launch_bounds__(1024) k_mg_tail_setup(const __grid_constant__ MgTail T, int dim) {
    for (int l = T.first; l + 1 < T.n; ++l) {
        for (int t = threadIdx.x; t < T.l[l + 1].n; t += blockDim.x) mg_coarsen(T.l[l], T.l[l + 1], dim, t);
        __syncthreads();
    }
}

// The V-cycle's levels first .. n - 1 in one block: down, weighted-Jacobi
// sweeps on the coarsest (one cell per thread, its row in registers and the
// iterate in shared memory), up.
__global__ void __launch_bounds__(1024) k_mg_tail(const __grid_constant__ MgTail T, int dim, CgState* S,
                                                  double* partial, int slot) {
    __shared__ double xs[2][1024];
    grid_dep_launch();
    grid_dep_wait();
    if (S->done) return;
    const int last = T.n - 1;
    for (int l = T.first; l < last; ++l) {
        for (int t = threadIdx.x; t < T.l[l + 1].n; t += blockDim.x) mg_down(T.l[l], T.l[l + 1], dim, t);
        __syncthreads();
    }
    {
        const MgLevel& L = T.l[last];
        const int t = threadIdx.x;
        const bool on = t < L.n;   // at most kMgCoarsest cells
        double w[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, diag = 0.0, iw = 0.0, b = 0.0, x = 0.0;
        int nb[6] = {0, 0, 0, 0, 0, 0};
        if (on) {
            int i, j, k;
            mg_split(L, t, i, j, k);
            const MgNb q = mg_nb(L, t, i, j, k);
            nb[0] = q.xm; nb[1] = q.xp; nb[2] = q.ym; nb[3] = q.yp; nb[4] = q.zm; nb[5] = q.zp;
            w[0] = L.tx[t];
            w[1] = L.tx[q.xp];
            if (dim >= 2) { w[2] = L.ty[t]; w[3] = L.ty[q.yp]; }
            if (dim >= 3) { w[4] = L.tz[t]; w[5] = L.tz[q.zp]; }
            diag = L.diag[t];
            iw = L.iw[t];
            b = L.b[t];
            x = iw * b;
            xs[0][t] = x;
        }
        __syncthreads();
        for (int s = 0; s < kMgCoarsestSweeps; ++s) {
            const double* xi = xs[s & 1];
            if (on) {
                double off = w[0] * xi[nb[0]] + w[1] * xi[nb[1]];
                if (dim >= 2) off += w[2] * xi[nb[2]] + w[3] * xi[nb[3]];
                if (dim >= 3) off += w[4] * xi[nb[4]] + w[5] * xi[nb[5]];
                x = x + iw * (b - (diag * x - off));
                xs[(s & 1) ^ 1][t] = x;
            }
            __syncthreads();
        }
        if (on) L.x[t] = x;
        __syncthreads();
    }
    double v = 0.0;
    for (int l = last - 1; l >= T.first; --l) {
        for (int t = threadIdx.x; t < T.l[l].n; t += blockDim.x) {
            const double x = mg_up(T.l[l], T.l[l + 1], dim, t);
            if (l == 0) v += T.l[l].b[t] * x;
        }
        __syncthreads();
    }
    if (T.first == 0) {   // the whole hierarchy: r.z here
        if (last == 0 && (int)threadIdx.x < T.l[0].n) v = T.l[0].b[threadIdx.x] * T.l[0].x[threadIdx.x];
        double total;
        if (grid_sum(v, partial, &S->count, &total)) S->rz[slot] = total;
    }
}

// r = b - M x; |r/m|^2 and |b/m|^2 (the unscaled residual and right-hand
// side), and whether there is anything to solve.
__global__ void __launch_bounds__(256) k_cg_start(MgLevel L, int dim, const double* __restrict__ wInv,
                                                  double* __restrict__ r, CgState* S, double* partial) {
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    double v = 0.0, u = 0.0;
    if (t < L.n) {
        int i, j, k;
        mg_split(L, t, i, j, k);
        const double* x = L.x;
        const double b = L.b[t];
        const double rr = b - mg_apply(L, dim, t, mg_nb(L, t, i, j, k), x[t], [&](int c) { return x[c]; });
        r[t] = rr;
        v = rr * wInv[t];
        v *= v;
        u = b * wInv[t];
        u *= u;
    }
    double total;
    if (grid_sum(u, partial, &S->count, &total)) S->bb = total;
    if (grid_sum(v, partial + gridDim.x, &S->count2, &total)) {
        S->rr = total;
    }
}

// After k_cg_start: the stopping rule on the initial residual.
__global__ void k_cg_test(CgState* S, double tol) {
    S->eps = tol * tol;
    S->iters = 0;
    S->done = (S->bb == 0.0 || S->rr <= S->eps * S->bb) ? 1 : 0;
}

// p = z + beta p (beta = rz / previous rz; first: p = z), q = M p, p.q.
__global__ void __launch_bounds__(256) k_cg_product(MgLevel L, int dim, const double* __restrict__ z,
                                                    const double* __restrict__ pOld, double* __restrict__ p,
                                                    double* __restrict__ q, CgState* S, double* partial, int slot,
                                                    int first) {
    grid_dep_launch();
    grid_dep_wait();
    if (S->done) return;
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    const double beta = first ? 0.0 : S->rz[slot] / S->rz[slot ^ 1];
    double v = 0.0;
    if (t < L.n) {
        int i, j, k;
        mg_split(L, t, i, j, k);
        auto dir = [&](int c) { return first ? z[c] : z[c] + beta * pOld[c]; };
        const double pc = dir(t);
        const double a = mg_apply(L, dim, t, mg_nb(L, t, i, j, k), pc, dir);
        p[t] = pc;
        q[t] = a;
        v = pc * a;
    }
    double total;
    if (grid_sum(v, partial, &S->count, &total)) S->pq = total;
}

// x += alpha p; r -= alpha q, alpha = rz / p.q; |r/m|^2 and the stopping rule.
__global__ void __launch_bounds__(256) k_cg_update(int n, double* __restrict__ x, double* __restrict__ r,
                                                   const double* __restrict__ p, const double* __restrict__ q,
                                                   const double* __restrict__ wInv, CgState* S, double* partial,
                                                   int slot) {
    grid_dep_launch();
    grid_dep_wait();
    if (S->done) return;
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    const double alpha = S->rz[slot] / S->pq;
    double v = 0.0;
    if (t < n) {
        x[t] += alpha * p[t];
        const double rr = r[t] - alpha * q[t];
        r[t] = rr;
        const double u = rr * wInv[t];
        v = u * u;
    }
    double total;
    if (grid_sum(v, partial, &S->count, &total)) {
        S->rr = total;
        S->iters += 1;
        if (total <= S->eps * S->bb || !(total == total)) S->done = 1;
    }
}

// Solution back into the context's pressure array (interior cells only, as
// HyprePressureSolver copies back, src/HyprePressureSolver.cpp:388-396).
__global__ void __launch_bounds__(256) k_mg_scatter(Params P, MgLevel L, double* __restrict__ p, const CgState* S) {
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (t >= L.n) return;
    int i, j, k;
    mg_split(L, t, i, j, k);
    p[cidx(P, i, j, k)] = (S->bb == 0.0) ? 0.0 : L.x[t];   // Hypre: zero right-hand side -> zero solution
}

}  // namespace sifv
