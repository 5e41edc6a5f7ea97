// sifv_tile3d.cuh -- one SSP-RK stage of the 3D explicit step as one kernel,
// fast FP64 and mixed precision (included by sifv_fast.cu).
//
// A block of 320 threads owns 32 x 8 columns of cells and walks them along z.
// Per plane k:
//   A  the conservative values of plane k + 3 become primitives in a ring of
//      five planes (k - 1 .. k + 3), those of plane k's three-cell halo in x
//      and y go with the plane itself into a 38 x 14 tile;
//   B  z: both face values of every cell of plane k + 1 from the ring (each
//      thread its own column, no exchange), the flux between planes k and
//      k + 1 with the value carried from the step before; x: both face values
//      of the 34 x 8 cells;
//   C  x fluxes (33 x 8 faces);
//   D  x divergence; y: both face values of the 32 x 10 cells;
//   E  y fluxes (32 x 9 faces);
//   F  y divergence, and the update of plane k in FP64.
// Every z face is solved once, x faces 33/32 and y faces 9/8 times, and a
// cell's state is read once as a cell (and from L2 as another block's halo)
// and written once; three dimension sweeps pass primitives and an FP64 rhs
// through memory (56 arrays per stage) and read the mesh again for the dt.
// Per step, RK3, sweeps -> this, FP64 / mixed: 160^3 2.42 -> 2.07 / 1.79 ->
// 1.41 ms; 64^3 393 -> 180 / 334 -> 127 us; 8^3 153 -> 62 / 139 -> 51 us;
// 203 x 160 x 131 2.19 -> 2.28 / 1.78 -> 1.50 ms.  It is bound by its chains
// between the barriers: the FP64 pipe is busy 48 % of the time at two blocks
// per SM (shared memory), and a tile costs much the same however few of its
// rows lie in the mesh, so meshes that fit the tiles badly keep the sweeps
// (sweeps_3d).
#pragma once

#include "sifv_sweep.cuh"

namespace sifv {

struct Tile3 {
    static constexpr int TX = 32, TY = 8, threads = 320, cells = TX * TY;
    static constexpr int W = TX + 6, H = TY + 6, WH = W * H;
    static constexpr int R = TX * (TY + 2);            // reconstructed cells of a direction, at most
    static constexpr int FN = TX * (TY + 1);           // its faces, at most
    static constexpr int halo = 6 * TY + 6 * TX;       // halo positions of a plane (no corners)
    template <typename T>
    static constexpr size_t smem() { return sizeof(T) * 5 * (5 * cells + WH + 2 * R + FN); }
};

template <typename T>
__device__ __forceinline__ void tile3_prim(const Tile3Args& A, size_t s, const double sg[3], T w[5]) {
    const double rr = A.in[0][s], re = A.in[4][s];
    const double rho = (rr < 1e-14) ? 1e-14 : rr;
    const double ir = frcp(rho);
    const double u = A.in[1][s] * ir, v = A.in[2][s] * ir, ww = A.in[3][s] * ir;
    double ke = u * u;
    ke += v * v;
    ke += ww * ww;
    ke *= 0.5 * rho;
    const double e = re - ke;
    double p = A.P.eosStiffened ? (A.P.gamma - 1.0) * e - A.P.gamma * A.P.pInf : (A.P.gamma - 1.0) * e;
    if (!A.P.eosStiffened && p < 1e-14) p = 1e-14;
    w[0] = (T)rr;
    w[1] = (T)(sg[0] * u);
    w[2] = (T)(sg[1] * v);
    w[3] = (T)(sg[2] * ww);
    w[4] = (T)p;
}

template <typename T>
__device__ __forceinline__ Prim5<T> tile3_state(const T* a, int st, int c) {
    return Prim5<T>{a[c], a[st + c], a[2 * st + c], a[3 * st + c], a[4 * st + c]};
}

// Both face values of one cell, five variables st apart, stencil stride d.
template <typename T>
__device__ __forceinline__ void tile3_recon(const T* w, int st, int d, T eps, T* hi, T* lo, int c) {
#pragma unroll 1
    for (int v = 0; v < 5; ++v) {
        const T* f = w + v * st;
        weno5_pair(f[-2 * d], f[-d], f[0], f[d], f[2 * d], eps, hi[v * Tile3::R + c], lo[v * Tile3::R + c]);
    }
}

template <typename T>
__device__ __forceinline__ void tile3_store(T* f, int c, const Flux4<T>& F) {
    f[c] = F.mass;
    f[Tile3::FN + c] = F.m0;
    f[2 * Tile3::FN + c] = F.m1;
    f[3 * Tile3::FN + c] = F.m2;
    f[4 * Tile3::FN + c] = F.energy;
}

template <typename T, int RS>
__global__ void __launch_bounds__(Tile3::threads, 2) k_tile3d(const __grid_constant__ Tile3Args A) {
    constexpr int TX = Tile3::TX, TY = Tile3::TY, W = Tile3::W, WH = Tile3::WH, NC = Tile3::cells, R = Tile3::R;
    extern __shared__ __align__(16) unsigned char smemRaw[];
    T* const ring = reinterpret_cast<T*>(smemRaw);   // [5 planes][5 variables][cells]
    T* const tile = ring + 25 * NC;                  // [5][38 x 14], the centre plane
    T* const sHi = tile + 5 * WH;
    T* const sLo = sHi + 5 * R;
    T* const sF = sLo + 5 * R;
    grid_dep_launch();
    grid_dep_wait();
    if (A.ctl->skip) return;
    const Params& P = A.P;
    const int tid = threadIdx.x;
    const int i0 = (int)(blockIdx.x % A.tilesX) * TX, j0 = (int)(blockIdx.x / A.tilesX % A.tilesY) * TY;
    const int z0 = (int)(blockIdx.x / (A.tilesX * A.tilesY)) * A.segPlanes, z1 = min(z0 + A.segPlanes, P.nz);
    const int lx = min(TX, P.nx - i0), ly = min(TY, P.ny - j0);
    const T eps = (T)A.eps;
    const double a3dt = A.a3 * A.ctl->dt;
    const size_t sz = (size_t)P.nxT * P.nyT;

    // the thread's cell (columns past the mesh's edge serve as halo up to the third ghost)
    const int ci = tid % TX, cj = tid / TX;
    const bool column = tid < NC && i0 + ci < P.nx + 3 && j0 + cj < P.ny + 3;
    const bool mine = tid < NC && ci < lx && cj < ly;
    // the (x, y) part of the ghost map of a position: source offset and velocity signs
    auto map_xy = [&](int i, int j, size_t& off, double sg[3]) {
        double sn, sa;
        sg[0] = sg[1] = sg[2] = 1.0;
        const int si = prim_src(i, P.nx, P.bc[0], P.bc[1], sn, sa);
        if (si != i) { sg[0] *= sn * sa; sg[1] *= sa; sg[2] *= sa; }
        const int sj = prim_src(j, P.ny, P.bc[2], P.bc[3], sn, sa);
        if (sj != j) { sg[0] *= sa; sg[1] *= sn * sa; sg[2] *= sa; }
        off = (size_t)(si + P.ngx) + (size_t)P.nxT * (size_t)(sj + P.ngy);
    };
    size_t cOff = 0, hOff = 0;
    double cSg[3] = {1.0, 1.0, 1.0}, hSg[3] = {1.0, 1.0, 1.0};
    if (column) map_xy(i0 + ci, j0 + cj, cOff, cSg);
    // the thread's halo position of the tile: rows above and below, then columns left and right
    int hPos = -1;
    if (tid < Tile3::halo) {
        int a, b;
        if (tid < 6 * TX) {
            a = tid % TX + 3;
            b = tid / TX;
            b = (b < 3) ? b : b + TY;
        } else {
            const int q = tid - 6 * TX;
            a = q % 6;
            a = (a < 3) ? a : a + TX;
            b = q / 6 + 3;
        }
        const int i = i0 + a - 3, j = j0 + b - 3;
        if (i < P.nx + 3 && j < P.ny + 3) {
            hPos = a + W * b;
            map_xy(i, j, hOff, hSg);
        }
    }
    auto plane_prim = [&](int k, size_t off, const double* sgxy, T* w) {
        double sn, sa, sg[3] = {sgxy[0], sgxy[1], sgxy[2]};
        const int sk = prim_src(k, P.nz, P.bc[4], P.bc[5], sn, sa);
        if (sk != k) { sg[0] *= sa; sg[1] *= sa; sg[2] *= sn * sa; }
        tile3_prim<T>(A, off + sz * (size_t)(sk + P.ngz), sg, w);
    };
    auto to_ring = [&](int k) {   // the thread's cell of plane k
        if (!column || k >= P.nz + 3) return;
        T w[5];
        plane_prim(k, cOff, cSg, w);
        T* r = ring + ((k + 10) % 5) * 5 * NC + tid;
#pragma unroll
        for (int v = 0; v < 5; ++v) r[v * NC] = w[v];
    };

    Prim5<T> Lz = {(T)0, (T)0, (T)0, (T)0, (T)0};   // value at the high z face of plane k, from below
    Flux4<T> Fz = {(T)0, (T)0, (T)0, (T)0, (T)0};   // flux at its low z face
    double limit = __longlong_as_double(0x7ff0000000000000LL);
    for (int k = z0 - 3; k <= z0; ++k) to_ring(k);
    for (int k = z0 - 2; k < z1; ++k) {
        const bool run = k >= z0;   // the two planes below only start the z faces
        // ---- A ----
        to_ring(k + 3);
        if (run) {
            if (column) {
                const T* r = ring + ((k + 10) % 5) * 5 * NC + tid;
                T* t = tile + (ci + 3) + W * (cj + 3);
#pragma unroll
                for (int v = 0; v < 5; ++v) t[v * WH] = r[v * NC];
            }
            if (hPos >= 0) {
                T w[5];
                plane_prim(k, hOff, hSg, w);
#pragma unroll
                for (int v = 0; v < 5; ++v) tile[v * WH + hPos] = w[v];
            }
            __syncthreads();
        }
        // ---- B: z of plane k + 1, then x values ----
        double r[5];
        if (mine) {
            const T* p[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) p[q] = ring + ((k - 1 + q + 10) % 5) * 5 * NC + tid;
            T l[5], h[5];
#pragma unroll
            for (int v = 0; v < 5; ++v)
                weno5_pair(p[0][v * NC], p[1][v * NC], p[2][v * NC], p[3][v * NC], p[4][v * NC], eps, h[v], l[v]);
            const Prim5<T> Rz = {l[0], l[1], l[2], l[3], l[4]};
            Flux4<T> Fn;
            face_flux<2, 3, T>(RS, A.C, Lz, Rz, Fn);
            Lz = Prim5<T>{h[0], h[1], h[2], h[3], h[4]};
            if (run) {
                const double ci2 = A.inv[2][k + P.ngz];
                r[0] = ci2 * ((double)Fz.mass - (double)Fn.mass);
                r[1] = ci2 * ((double)Fz.m0 - (double)Fn.m0);
                r[2] = ci2 * ((double)Fz.m1 - (double)Fn.m1);
                r[3] = ci2 * ((double)Fz.m2 - (double)Fn.m2);
                r[4] = ci2 * ((double)Fz.energy - (double)Fn.energy);
            }
            Fz = Fn;
        }
        if (!run) continue;
        if (tid < (TX + 2) * TY) {
            const int a = tid % (TX + 2), b = tid / (TX + 2);   // cell (a - 1, b)
            if (a <= lx + 1 && b < ly) tile3_recon<T>(tile + (a + 2) + W * (b + 3), WH, 1, eps, sHi, sLo, tid);
        }
        __syncthreads();
        // ---- C: x fluxes ----
        if (tid < (TX + 1) * TY) {
            const int a = tid % (TX + 1), b = tid / (TX + 1);
            if (a <= lx && b < ly) {
                const int c = a + (TX + 2) * b;
                Flux4<T> F;
                face_flux<0, 3, T>(RS, A.C, tile3_state(sHi, R, c), tile3_state(sLo, R, c + 1), F);
                tile3_store(sF, tid, F);
            }
        }
        __syncthreads();
        // ---- D: x divergence, y values ----
        if (mine) {
            const double ci0 = A.inv[0][i0 + ci + P.ngx];
            const int f = ci + (TX + 1) * cj;
#pragma unroll
            for (int v = 0; v < 5; ++v)
                r[v] += ci0 * ((double)sF[v * Tile3::FN + f] - (double)sF[v * Tile3::FN + f + 1]);
        }
        {
            const int a = tid % TX, b = tid / TX;   // cell (a, b - 1)
            if (a < lx && b <= ly + 1) tile3_recon<T>(tile + (a + 3) + W * (b + 2), WH, W, eps, sHi, sLo, tid);
        }
        __syncthreads();
        // ---- E: y fluxes ----
        if (tid < TX * (TY + 1)) {
            const int a = tid % TX, b = tid / TX;
            if (a < lx && b <= ly) {
                Flux4<T> F;
                face_flux<1, 3, T>(RS, A.C, tile3_state(sHi, R, tid), tile3_state(sLo, R, tid + TX), F);
                tile3_store(sF, tid, F);
            }
        }
        __syncthreads();
        // ---- F: y divergence and the update ----
        if (mine) {
            const double ci1 = A.inv[1][j0 + cj + P.ngy];
            const size_t c = cOff + sz * (size_t)(k + P.ngz);
            double n[5];
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                r[v] += ci1 * ((double)sF[v * Tile3::FN + tid] - (double)sF[v * Tile3::FN + tid + TX]);
                double x = A.a1 * A.in[v][c] + a3dt * r[v];
                if (A.u0[0]) x += A.a2 * A.u0[v][c];
                n[v] = x;
            }
#pragma unroll
            for (int v = 0; v < 5; ++v) A.out[v][c] = n[v];
            if (A.last) {   // primitives of the new state (cons_to_prim_cell, single phase)
                const double rho = (n[0] < 1e-14) ? 1e-14 : n[0];
                const double ir = frcp(rho);
                const double u = n[1] * ir, v = n[2] * ir, w = n[3] * ir;
                double ke = u * u;
                ke += v * v;
                ke += w * w;
                ke *= 0.5 * rho;
                const double e = n[4] - ke;
                const double p = P.eosStiffened ? (P.gamma - 1.0) * e - P.gamma * P.pInf
                                                : ((P.gamma - 1.0) * e < 1e-14 ? 1e-14 : (P.gamma - 1.0) * e);
                A.velU[c] = u;
                A.velV[c] = v;
                A.velW[c] = w;
                A.pres[c] = p;
                if (A.dtNext) {   // k_dt_acoustic's cell term
                    const double cs = single_sound_speed(P, n[0], p);
                    double dtCell = A.dx[i0 + ci + P.ngx] / (fabs(u) + cs);
                    dtCell = smin(dtCell, A.dy[j0 + cj + P.ngy] / (fabs(v) + cs));
                    dtCell = smin(dtCell, A.dz[k + P.ngz] / (fabs(w) + cs));
                    limit = smin(limit, A.cfl * dtCell);   // a NaN candidate leaves it
                }
            }
        }
    }
    if (A.last && A.dtNext) block_min_to(limit, &A.ctl->dtBits);
}

// The stage output's interior cells copied over the state's (RK1, whose only
// stage cannot update in place).  The scratch has no ghost layers of its own:
// those of the state's momenta and energy stay as the caller left them, as in
// the schemes of more stages.
struct Copy5 {
    const double* src[5];
    double* dst[5];
};
__global__ void __launch_bounds__(256) k_copy_interior(Params P, const Ctl* ctl, Copy5 A) {
    if (ctl->skip) return;
    int i, j, k;
    if (!int_coords(P, (long long)blockIdx.x * blockDim.x + threadIdx.x, i, j, k)) return;
    const size_t c = cidx(P, i, j, k);
#pragma unroll
    for (int q = 0; q < 5; ++q) A.dst[q][c] = A.src[q][c];
}

}  // namespace sifv
