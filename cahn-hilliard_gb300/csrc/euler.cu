// euler.cu — fused explicit finite-difference steps (`euler`, `euler_mobility`).
//
// One kernel launch is one time step, one HBM pass: each CTA stages a tile of
// psi with a halo of 2 cells in shared memory, computes the chemical
// potential mu = f'(psi) - 2k lap(psi) on the tile plus a halo of 1 (and, for
// `euler_mobility`, the mobility M on the same cells), then writes
// psi + dt * div(M grad mu) for its tile.  Nothing but psi_in and psi_out
// touches HBM.  3D tiles march along z with rolling planes of psi (5) and
// mu (3) so the halo recomputation stays in x and y only.
//
// Reference: src/integrators/EulerCPU.cpp:18-36 (three passes, Laplacian
// :58-88) and src/integrators/EulerMobilityCPU.cpp:31-83 (face fluxes and the
// divergence of src/integrators/EulerCPU.cpp:114-128).  The 2D and 3D
// neighbour sums are formed in fixed point and rounded once (fxsum.cuh), not
// added in the reference's order (-x, +x, -y, +y, -z, +z); 1D keeps that order.
// Constants are folded (c2 = 2k/dx^2, c1 = dt M/dx^2).  Both move results by at
// most a few ulp per step.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "bfp.cuh"
#include "bounds.cuh"
#include "common.cuh"
#include "fxsum.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace chgb {

// Index checks of the bounds-check build: CHGB_BC (bounds.cuh).

// euler_mobility kernels' mobility kind for a CHGB_MOBILITY_* type.
int mobility_kind(int mobility_type) {
    switch(mobility_type) {
        case CHGB_MOBILITY_FREE_ENERGY: return 2;
        case CHGB_MOBILITY_REGULARISED:
        case CHGB_MOBILITY_GEL: return 3;
        default: return 1;
    }
}

// f' of one cell; with the free-energy mobility of simple_wertheim it also
// returns rho X^v, which the mobility of the same cell reuses.
template <int KIND, int MOB>
__device__ __forceinline__ double der_bulk_x(const ModelDev &m, const double *r, double *d) {
    if constexpr(KIND == CHGB_MODEL_SIMPLE_WERTHEIM && MOB == 2) {
        const SwCell c = sw_cell(m, r[0]);
        d[0] = c.der;
        return c.rhoXv;
    }
    else {
        der_bulk<KIND>(m, r, d);
        return 0.0;
    }
}

// The mobility of one cell for the template mobility kind: 1 constant, 2 the
// free-energy mobility of the cell's density (rho X^v from der_bulk_x), 3 the field
// computed before the step (regularised / gel; `gi` is the cell's index in one
// species' field).
template <int MOB>
__device__ __forceinline__ double cell_mobility(const ModelDev &m, const EulerConsts &c, int s, double r, double rhoXv,
                                                size_t bins, size_t gi) {
    if constexpr(MOB == 2) return c.M * rhoXv;
    else if constexpr(MOB == 3) return CHGB_BC(40, gi, bins) ? c.mobf[s * bins + gi] : 0.0;
    else return c.M;
}

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------

// Sum of the 2*DIMS neighbours of p and lap = sum - 2*DIMS*v (1D: the
// reference's FP64 sum; 2D and 3D: fx_sum).
template <int DIMS>
__device__ __forceinline__ double lap_sum(const double *p, int sx, int sy, int sz, double v) {
    if constexpr(DIMS == 1) return fma(-2.0, v, p[-sx] + p[sx]);
    else if constexpr(DIMS == 2) return lap4(p[-sx], p[sx], p[-sy], p[sy], v);
    else return lap6(p[-sx], p[sx], p[-sy], p[sy], p[-sz], p[sz], v);
}

// Sum of the 2*DIMS neighbours only (DIMS 1, 2).
template <int DIMS>
__device__ __forceinline__ double nb_sum(const double *p, int sx, int sy) {
    if constexpr(DIMS == 1) return p[-sx] + p[sx];
    else return nb_sum4(p[-sx], p[sx], p[-sy], p[sy]);
}

// Chemical potential of one cell and species from its value r, its model
// derivative d (unused for Landau) and the sum of its 2*DIMS neighbours:
//   mu = f'(r) - c2 (sum - 2 DIMS r).
// For Landau f' = r^3 - eps r is folded with the diagonal of the Laplacian,
//   mu = r (r^2 + (2 DIMS c2 - eps)) - c2 sum,
// one FP64 instruction fewer per cell; the FP64 pipe is this kernel's bound.
template <int KIND, int DIMS>
__device__ __forceinline__ double mu_cell(const ModelDev &m, const EulerConsts &c, int s, double r, double d,
                                          double sum) {
    if constexpr(KIND == CHGB_MODEL_LANDAU) {
        return fma(-c.c2[s], sum, r * fma(r, r, c.lshift[DIMS - 1]));
    }
    else {
        return fma(-c.c2[s], fma(-2.0 * DIMS, r, sum), d);
    }
}

// ---------------------------------------------------------------------------
// 1D: tiles of T cells
// ---------------------------------------------------------------------------
template <int KIND, int MOB, int T>
__global__ void __launch_bounds__(256) euler1d_kernel(const double *__restrict__ in, double *__restrict__ out, Geom g,
                                                      ModelDev m, EulerConsts c) {
    constexpr int S = NSpecies<KIND>::value;
    constexpr int P = T + 4, Q = T + 2;
    __shared__ double psi[S][P];
    __shared__ double mu[S][Q];
    __shared__ double mob[MOB ? S : 1][MOB ? Q : 1];
    const int x0 = blockIdx.x * T;
    const size_t bins = (size_t) g.bins;
    for(int i = threadIdx.x; i < P; i += blockDim.x) {
        int gx = (x0 - 2 + i) & g.mask;
#pragma unroll
        for(int s = 0; s < S; s++) psi[s][i] = CHGB_BC(41, gx, bins) ? in[s * bins + gx] : 0.0;
    }
    __syncthreads();
    for(int i = threadIdx.x; i < Q; i += blockDim.x) {
        double r[S], d[S];
#pragma unroll
        for(int s = 0; s < S; s++) r[s] = psi[s][i + 1];
        const double xsw = der_bulk_x<KIND, MOB>(m, r, d);
#pragma unroll
        for(int s = 0; s < S; s++) {
            mu[s][i] = mu_cell<KIND, 1>(m, c, s, r[s], d[s], nb_sum<1>(&psi[s][i + 1], 1, 0));
            if(MOB) mob[s][i] = cell_mobility<MOB>(m, c, s, r[s], xsw, bins, (size_t) ((x0 - 1 + i) & g.mask));
        }
    }
    __syncthreads();
    for(int i = threadIdx.x; i < T; i += blockDim.x) {
#pragma unroll
        for(int s = 0; s < S; s++) {
            const double *u = &mu[s][i + 1];
            double res;
            if(MOB) {
                const double *mm = &mob[s][i + 1];
                double jp = (mm[0] + mm[1]) * (u[1] - u[0]);
                double jm = (mm[-1] + mm[0]) * (u[0] - u[-1]);
                res = fma(c.dt * c.half_inv_dx2, jp - jm, psi[s][i + 2]);
            }
            else {
                res = fma(c.c1, lap_sum<1>(u, 1, 0, 0, u[0]), psi[s][i + 2]);
            }
            if(CHGB_BC(42, x0 + i, bins)) out[s * bins + x0 + i] = res;
        }
    }
}

// ---------------------------------------------------------------------------
// 2D: TX x TY tiles, 256 threads
// ---------------------------------------------------------------------------
// One TX x TY tile at (x0, y0); shared by the single-box and the batched kernels.
template <int KIND, int MOB, int TX, int TY>
__device__ __forceinline__ void euler2d_tile(const double *__restrict__ in, double *__restrict__ out, const Geom &g,
                                             const ModelDev &m, const EulerConsts &c, int x0, int y0, double *smem) {
    constexpr int S = NSpecies<KIND>::value;
    constexpr int PX = TX + 4, PY = TY + 4, PP = PX * PY;
    constexpr int MX = TX + 2, MY = TY + 2, MP = MX * MY;
    double *psi = smem;               // [S][PY][PX]
    double *mu = psi + S * PP;        // [S][MY][MX]
    double *mob = mu + S * MP;        // [S][MY][MX] (euler_mobility only)
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    const int nthr = blockDim.x * blockDim.y;
    const size_t bins = (size_t) g.bins;

    for(int i = tid; i < PP; i += nthr) {
        int ly = i / PX, lx = i - ly * PX;
        int gx = (x0 - 2 + lx) & g.mask, gy = (y0 - 2 + ly) & g.mask;
        int gi = gx + (gy << g.log2N);
#pragma unroll
        for(int s = 0; s < S; s++) psi[s * PP + i] = CHGB_BC(43, gi, bins) ? in[s * bins + gi] : 0.0;
    }
    __syncthreads();
    for(int i = tid; i < MP; i += nthr) {
        int ly = i / MX, lx = i - ly * MX;
        int p = (ly + 1) * PX + (lx + 1);
        if(!CHGB_BC(44, p - PX, PP) || !CHGB_BC(44, p + PX, PP)) continue;
        double r[S], d[S];
#pragma unroll
        for(int s = 0; s < S; s++) r[s] = psi[s * PP + p];
        const double xsw = der_bulk_x<KIND, MOB>(m, r, d);
#pragma unroll
        for(int s = 0; s < S; s++) {
            mu[s * MP + i] = mu_cell<KIND, 2>(m, c, s, r[s], d[s], nb_sum<2>(psi + s * PP + p, 1, PX));
            if(MOB) {
                const size_t gi = (size_t) ((x0 - 1 + lx) & g.mask) + ((size_t) ((y0 - 1 + ly) & g.mask) << g.log2N);
                mob[s * MP + i] = cell_mobility<MOB>(m, c, s, r[s], xsw, bins, gi);
            }
        }
    }
    __syncthreads();
    for(int i = tid; i < TX * TY; i += nthr) {
        int ly = i / TX, lx = i - ly * TX;
        int q = (ly + 1) * MX + (lx + 1);
        int gi = (x0 + lx) + ((y0 + ly) << g.log2N);
        if(!CHGB_BC(45, q - MX, MP) || !CHGB_BC(45, q + MX, MP) || !CHGB_BC(45, gi, bins)) continue;
#pragma unroll
        for(int s = 0; s < S; s++) {
            const double *u = mu + s * MP + q;
            double psi0 = psi[s * PP + (ly + 2) * PX + (lx + 2)];
            double res;
            if(MOB) {
                const double *mm = mob + s * MP + q;
                double jxp = (mm[0] + mm[1]) * (u[1] - u[0]);
                double jxm = (mm[-1] + mm[0]) * (u[0] - u[-1]);
                double jyp = (mm[0] + mm[MX]) * (u[MX] - u[0]);
                double jym = (mm[-MX] + mm[0]) * (u[0] - u[-MX]);
                double div = (jxp - jxm) + (jyp - jym);
                res = fma(c.dt * c.half_inv_dx2, div, psi0);
            }
            else {
                res = fma(c.c1, lap_sum<2>(u, 1, MX, 0, u[0]), psi0);
            }
            out[s * bins + gi] = res;
        }
    }
}

template <int KIND, int MOB, int TX, int TY>
__global__ void __launch_bounds__(256) euler2d_kernel(const double *__restrict__ in, double *__restrict__ out, Geom g,
                                                      ModelDev m, EulerConsts c) {
    extern __shared__ double smem[];
    euler2d_tile<KIND, MOB, TX, TY>(in, out, g, m, c, blockIdx.x * TX, blockIdx.y * TY, smem);
}

// Two time steps of plain `euler` per launch on a TX x TY tile, for small 2D
// boxes whose steps are too short to hide a launch: psi with a halo of 4 in
// shared memory, mu on the tile + 3, psi after one step on the tile + 2, mu
// again on the tile + 1, psi after two steps on the tile.  The halo costs
// extra FP64 work (16x16 tiles: 15.9 instructions per cell and step against
// 12.6), so it pays only where the launch, not the FP64 pipe, sets the pace.
// Every value comes from the same helpers as euler2d_tile's, so two steps here
// are the same bits as two launches of the one-step kernel.  With `mid` set,
// the state after the first step is stored too (the adjoint's recomputed
// segments keep every state).
template <int KIND, int TX, int TY>
__global__ void __launch_bounds__(256) euler2d_two_kernel(const double *__restrict__ in, double *__restrict__ out,
                                                          double *__restrict__ mid, Geom g, ModelDev m,
                                                          EulerConsts c) {
    constexpr int S = NSpecies<KIND>::value;
    constexpr int P0X = TX + 8, P0 = P0X * (TY + 8);
    constexpr int M0X = TX + 6, M0 = M0X * (TY + 6);
    constexpr int P1X = TX + 4, P1 = P1X * (TY + 4);
    constexpr int M1X = TX + 2, M1 = M1X * (TY + 2);
    extern __shared__ double smem[];
    double *p0 = smem;              // [S][TY + 8][TX + 8]  psi
    double *mu0 = p0 + S * P0;      // [S][TY + 6][TX + 6]  mu(psi)
    double *p1 = mu0 + S * M0;      // [S][TY + 4][TX + 4]  psi after one step
    double *mu1 = p1 + S * P1;      // [S][TY + 2][TX + 2]  mu of that
    const int tid = threadIdx.x + blockDim.x * threadIdx.y, nthr = blockDim.x * blockDim.y;
    const size_t bins = (size_t) g.bins;
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
    for(int i = tid; i < P0; i += nthr) {
        int ly = i / P0X, lx = i - ly * P0X;
        int gx = (x0 - 4 + lx) & g.mask, gy = (y0 - 4 + ly) & g.mask;
        size_t gi = (size_t) gx + ((size_t) gy << g.log2N);
#pragma unroll
        for(int s = 0; s < S; s++) p0[s * P0 + i] = CHGB_BC(46, gi, bins) ? in[s * bins + gi] : 0.0;
    }
    __syncthreads();
    for(int i = tid; i < M0; i += nthr) {
        int ly = i / M0X, lx = i - ly * M0X;
        int p = (ly + 1) * P0X + (lx + 1);
        if(!CHGB_BC(47, p - P0X, P0) || !CHGB_BC(47, p + P0X, P0)) continue;
        double r[S], d[S];
#pragma unroll
        for(int s = 0; s < S; s++) r[s] = p0[s * P0 + p];
        der_bulk<KIND>(m, r, d);
#pragma unroll
        for(int s = 0; s < S; s++)
            mu0[s * M0 + i] = mu_cell<KIND, 2>(m, c, s, r[s], d[s], nb_sum<2>(p0 + s * P0 + p, 1, P0X));
    }
    __syncthreads();
    for(int i = tid; i < P1; i += nthr) {
        int ly = i / P1X, lx = i - ly * P1X;
        int q = (ly + 1) * M0X + (lx + 1);
        const bool inner = mid && lx >= 2 && lx < TX + 2 && ly >= 2 && ly < TY + 2;
        const size_t gi = (size_t) (x0 + lx - 2) + ((size_t) (y0 + ly - 2) << g.log2N);
        if(!CHGB_BC(48, q - M0X, M0) || !CHGB_BC(48, q + M0X, M0) || (inner && !CHGB_BC(48, gi, bins))) continue;
#pragma unroll
        for(int s = 0; s < S; s++) {
            const double *u = mu0 + s * M0 + q;
            const double v = fma(c.c1, lap_sum<2>(u, 1, M0X, 0, u[0]), p0[s * P0 + (ly + 2) * P0X + (lx + 2)]);
            p1[s * P1 + i] = v;
            if(inner) mid[s * bins + gi] = v;
        }
    }
    __syncthreads();
    for(int i = tid; i < M1; i += nthr) {
        int ly = i / M1X, lx = i - ly * M1X;
        int p = (ly + 1) * P1X + (lx + 1);
        if(!CHGB_BC(49, p - P1X, P1) || !CHGB_BC(49, p + P1X, P1)) continue;
        double r[S], d[S];
#pragma unroll
        for(int s = 0; s < S; s++) r[s] = p1[s * P1 + p];
        der_bulk<KIND>(m, r, d);
#pragma unroll
        for(int s = 0; s < S; s++)
            mu1[s * M1 + i] = mu_cell<KIND, 2>(m, c, s, r[s], d[s], nb_sum<2>(p1 + s * P1 + p, 1, P1X));
    }
    __syncthreads();
    for(int i = tid; i < TX * TY; i += nthr) {
        int ly = i / TX, lx = i - ly * TX;
        int q = (ly + 1) * M1X + (lx + 1);
        size_t gi = (size_t) (x0 + lx) + ((size_t) (y0 + ly) << g.log2N);
        if(!CHGB_BC(50, q - M1X, M1) || !CHGB_BC(50, q + M1X, M1) || !CHGB_BC(50, gi, bins)) continue;
#pragma unroll
        for(int s = 0; s < S; s++) {
            const double *u = mu1 + s * M1 + q;
            out[s * bins + gi] = fma(c.c1, lap_sum<2>(u, 1, M1X, 0, u[0]), p1[s * P1 + (ly + 2) * P1X + (lx + 2)]);
        }
    }
}

// 2D `euler` on a box small enough to live in the shared memory of one
// thread-block cluster (N = 4 T: 16 CTAs, one T x T tile each).  Each CTA keeps
// its tile in shared memory for the whole launch, double-buffered, and one
// launch runs many steps: global memory is read at the start and written at
// the end.  A step:
//   1. gathers the 2-cell halo ring of psi from the neighbouring CTAs' shared
//      memory (distributed shared memory; each thread's remote addresses are
//      resolved once per launch);
//   2. computes mu on the ring of the tile + 1 that needs the halo;
//   3. updates the tile into the other buffer;
//   4. arrives on the cluster barrier (publishing the new tile), computes mu on
//      the tile's interior for the next step -- local data only, which hides the
//      barrier's latency -- and waits on the barrier.
// The barrier also orders every remote read of a buffer before its next
// overwrite.  The values come from the same helpers as euler2d_tile's: the
// same bits as one launch per step.
constexpr int CLUSTER_TILES = 4;   // tiles per side of the box: 16 CTAs per cluster

// Position (ly, lx) in the (T + 4)^2 psi frame of halo-ring cell r (the frame
// minus its central T x T tile): two full rows on top and below, then two
// columns on each side.
__device__ __forceinline__ void cluster_ring_psi(int r, int T, int &ly, int &lx) {
    const int PX = T + 4;
    if(r < 2 * PX) {
        ly = r / PX;
        lx = r - ly * PX;
    }
    else if(r < 4 * PX) {
        r -= 2 * PX;
        ly = T + 2 + r / PX;
        lx = r % PX;
    }
    else if(r < 4 * PX + 2 * T) {
        r -= 4 * PX;
        ly = 2 + r / 2;
        lx = r % 2;
    }
    else {
        r -= 4 * PX + 2 * T;
        ly = 2 + r / 2;
        lx = T + 2 + r % 2;
    }
}

// Position (my, mx) in the (T + 2)^2 mu frame of ring cell r (8 T cells: the
// frame minus the (T - 2)^2 cells whose stencil stays on the tile).
__device__ __forceinline__ void cluster_ring_mu(int r, int T, int &my, int &mx) {
    const int MX = T + 2;
    if(r < 2 * MX) {
        my = r / MX;
        mx = r - my * MX;
    }
    else if(r < 4 * MX) {
        r -= 2 * MX;
        my = T + r / MX;
        mx = r % MX;
    }
    else if(r < 4 * MX + 2 * (T - 2)) {
        r -= 4 * MX;
        my = 2 + r / 2;
        mx = r % 2;
    }
    else {
        r -= 4 * MX + 2 * (T - 2);
        my = 2 + r / 2;
        mx = T + r % 2;
    }
}

template <int KIND, int T>
__device__ __forceinline__ void cluster_mu_cell(const ModelDev &m, const EulerConsts &c, const double (*P)[(T + 4) * (T + 4)],
                                                double (*MU)[(T + 2) * (T + 2)], int my, int mx) {
    constexpr int S = NSpecies<KIND>::value, PX = T + 4, MX = T + 2;
    const int p = (my + 1) * PX + (mx + 1);
    if(!CHGB_BC(51, p - PX, (T + 4) * (T + 4)) || !CHGB_BC(51, p + PX, (T + 4) * (T + 4)) ||
       !CHGB_BC(51, my * MX + mx, (T + 2) * (T + 2)))
        return;
    double r[S], d[S];
#pragma unroll
    for(int s = 0; s < S; s++) r[s] = P[s][p];
    der_bulk<KIND>(m, r, d);
#pragma unroll
    for(int s = 0; s < S; s++) MU[s][my * MX + mx] = mu_cell<KIND, 2>(m, c, s, r[s], d[s], nb_sum<2>(&P[s][p], 1, PX));
}

template <int KIND, int T, int NTHR>
__global__ void __launch_bounds__(NTHR) euler2d_cluster_kernel(const double *__restrict__ in,
                                                               double *__restrict__ out, Geom g, ModelDev m,
                                                               EulerConsts c, int nsteps) {
    static_assert(NTHR >= T * T, "one tile cell per thread");
    constexpr int S = NSpecies<KIND>::value;
    constexpr int TT = T * T, NT = CLUSTER_TILES * CLUSTER_TILES;
    constexpr int PX = T + 4, PP = PX * PX, MX = T + 2, MP = MX * MX;
    constexpr int NRING = PP - TT, NRING_MU = 8 * T, NINNER = (T - 2) * (T - 2);
    constexpr int KR = (NRING + NTHR - 1) / NTHR;   // halo-ring cells per thread
    __shared__ double own[2][S][TT];
    __shared__ double P[S][PP];        // psi on the tile + 2 (centre: this step's tile)
    __shared__ double MU[S][MP];       // mu on the tile + 1
    __shared__ unsigned rank_of[NT];   // cluster rank of the CTA that owns tile (tx, ty), at tx + 4 ty
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x;
    const bool cell = tid < TT;
    const int ly0 = (cell ? tid : 0) / T, lx0 = (cell ? tid : 0) % T;
    const int x0 = blockIdx.x * T, y0 = blockIdx.y * T;
    const size_t bins = (size_t) g.bins;
    const size_t gi0 = (size_t) (x0 + lx0) + ((size_t) (y0 + ly0) << g.log2N);
    const int pc = (ly0 + 2) * PX + (lx0 + 2);
    if(cell && CHGB_BC(52, gi0, bins)) {
#pragma unroll
        for(int s = 0; s < S; s++) {
            const double v = in[s * bins + gi0];
            own[0][s][tid] = v;
            P[s][pc] = v;
        }
    }
    // every CTA of the cluster is running past this barrier: publish this
    // CTA's rank into every CTA's table, then wait until all tables are full
    cluster.sync();
    if(tid < NT) {
        unsigned *dst = cluster.map_shared_rank(rank_of, (unsigned) tid);
        dst[blockIdx.x + CLUSTER_TILES * blockIdx.y] = cluster.block_rank();
    }
    cluster.sync();
    int rp[KR];
    const double *src[2][KR];
#pragma unroll
    for(int k = 0; k < KR; k++) {
        const int r = (tid + k * NTHR < NRING) ? tid + k * NTHR : 0;
        int ly, lx;
        cluster_ring_psi(r, T, ly, lx);
        rp[k] = ly * PX + lx;
        const int gx = (x0 - 2 + lx) & g.mask, gy = (y0 - 2 + ly) & g.mask;
        const int tx = gx / T, ty = gy / T;
        int off = (gx - tx * T) + (gy - ty * T) * T;
        int tile = tx + CLUSTER_TILES * ty;
        if(!CHGB_BC(53, off, TT) || !CHGB_BC(53, tile, NT) || !CHGB_BC(53, rp[k], PP)) {
            off = 0;
            tile = 0;
            rp[k] = 0;
        }
        src[0][k] = cluster.map_shared_rank(&own[0][0][0], rank_of[tile]) + off;
        src[1][k] = cluster.map_shared_rank(&own[1][0][0], rank_of[tile]) + off;
    }
    for(int j = tid; j < NINNER; j += NTHR) cluster_mu_cell<KIND, T>(m, c, P, MU, 2 + j / (T - 2), 2 + j % (T - 2));
    for(int step = 0; step < nsteps; step++) {
        const int cur = step & 1;
        double v[KR][S];
#pragma unroll
        for(int k = 0; k < KR; k++) {
            const double *q = cur ? src[1][k] : src[0][k];
#pragma unroll
            for(int s = 0; s < S; s++) v[k][s] = (tid + k * NTHR < NRING) ? q[s * TT] : 0.0;
        }
#pragma unroll
        for(int k = 0; k < KR; k++)
            if(tid + k * NTHR < NRING) {
#pragma unroll
                for(int s = 0; s < S; s++) P[s][rp[k]] = v[k][s];
            }
        __syncthreads();
        for(int r = tid; r < NRING_MU; r += NTHR) {
            int my, mx;
            cluster_ring_mu(r, T, my, mx);
            cluster_mu_cell<KIND, T>(m, c, P, MU, my, mx);
        }
        __syncthreads();
        if(cell) {
            const int q = (ly0 + 1) * MX + (lx0 + 1);
#pragma unroll
            for(int s = 0; s < S; s++) {
                const double nv = fma(c.c1, lap_sum<2>(&MU[s][q], 1, MX, 0, MU[s][q]), P[s][pc]);
                own[cur ^ 1][s][tid] = nv;
                P[s][pc] = nv;
            }
        }
        __syncthreads();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        for(int j = tid; j < NINNER; j += NTHR) cluster_mu_cell<KIND, T>(m, c, P, MU, 2 + j / (T - 2), 2 + j % (T - 2));
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    if(cell && CHGB_BC(54, gi0, bins)) {
#pragma unroll
        for(int s = 0; s < S; s++) out[s * bins + gi0] = own[nsteps & 1][s][tid];
    }
}

// Batched 2D `euler`: CTA b takes tile items[b].y of replica items[b].x; every
// replica steps a -> b (parity 0) or b -> a (parity 1).  All tiles have the
// same size, so the CTAs carry equal work whatever the replicas' N.
template <int KIND, int TX, int TY>
__global__ void __launch_bounds__(256) euler2d_batch_kernel(const EulerBatchRep *__restrict__ reps,
                                                            const int2 *__restrict__ items, int parity) {
    extern __shared__ double smem[];
    const int2 it = items[blockIdx.x];
    const EulerBatchRep &r = reps[it.x];
    const int tiles_x = r.g.N / TX;
    const int ty = it.y / tiles_x, tx = it.y - ty * tiles_x;
    const double *in = parity ? r.b : r.a;
    double *out = parity ? r.a : r.b;
    euler2d_tile<KIND, 0, TX, TY>(in, out, r.g, r.m, r.c, tx * TX, ty * TY, smem);
}

// ---------------------------------------------------------------------------
// 3D: TX x TY tiles marching over ZC planes, rolling windows in shared memory
// ---------------------------------------------------------------------------
template <int KIND, int MOB, int TX, int TY>
__global__ void __launch_bounds__(256) euler3d_kernel(const double *__restrict__ in, double *__restrict__ out, Geom g,
                                                      ModelDev m, EulerConsts c, int zc) {
    constexpr int S = NSpecies<KIND>::value;
    constexpr int PX = TX + 4, PY = TY + 4, PP = PX * PY;
    constexpr int MX = TX + 2, MY = TY + 2, MP = MX * MY;
    extern __shared__ double smem[];
    double *psi = smem;                    // [5][S][PP]
    double *mu = psi + 5 * S * PP;         // [3][S][MP]
    double *mob = mu + 3 * S * MP;         // [3][S][MP]
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    const int nthr = blockDim.x * blockDim.y;
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY, z0 = blockIdx.z * zc;
    const size_t bins = (size_t) g.bins;
    const int sh2 = 2 * g.log2N;

    auto load_plane = [&](int z) {
        double *dst = psi + ((z + 5) % 5) * S * PP;
        size_t zoff = (size_t) (z & g.mask) << sh2;
        for(int i = tid; i < PP; i += nthr) {
            int ly = i / PX, lx = i - ly * PX;
            int gx = (x0 - 2 + lx) & g.mask, gy = (y0 - 2 + ly) & g.mask;
            size_t gi = zoff + gx + (gy << g.log2N);
#pragma unroll
            for(int s = 0; s < S; s++) dst[s * PP + i] = CHGB_BC(55, gi, bins) ? in[s * bins + gi] : 0.0;
        }
    };
    auto mu_plane = [&](int z) {
        const double *pc = psi + ((z + 5) % 5) * S * PP;
        const double *pm = psi + ((z + 4) % 5) * S * PP;
        const double *pp = psi + ((z + 6) % 5) * S * PP;
        double *mdst = mu + ((z + 3) % 3) * S * MP;
        double *bdst = mob + ((z + 3) % 3) * S * MP;
        for(int i = tid; i < MP; i += nthr) {
            int ly = i / MX, lx = i - ly * MX;
            int p = (ly + 1) * PX + (lx + 1);
            if(!CHGB_BC(56, p - PX, PP) || !CHGB_BC(56, p + PX, PP)) continue;
            double r[S], d[S];
#pragma unroll
            for(int s = 0; s < S; s++) r[s] = pc[s * PP + p];
            const double xsw = der_bulk_x<KIND, MOB>(m, r, d);
#pragma unroll
            for(int s = 0; s < S; s++) {
                const double *q = pc + s * PP + p;
                const double sum = nb_sum6(q[-1], q[1], q[-PX], q[PX], pm[s * PP + p], pp[s * PP + p]);
                mdst[s * MP + i] = mu_cell<KIND, 3>(m, c, s, r[s], d[s], sum);
                if(MOB) {
                    const size_t gi = (size_t) ((x0 - 1 + lx) & g.mask) +
                                      ((size_t) ((y0 - 1 + ly) & g.mask) << g.log2N) +
                                      ((size_t) (z & g.mask) << sh2);
                    bdst[s * MP + i] = cell_mobility<MOB>(m, c, s, r[s], xsw, bins, gi);
                }
            }
        }
    };
    auto out_plane = [&](int z) {
        const double *uc = mu + ((z + 3) % 3) * S * MP;
        const double *um = mu + ((z + 2) % 3) * S * MP;
        const double *up = mu + ((z + 4) % 3) * S * MP;
        const double *bc = mob + ((z + 3) % 3) * S * MP;
        const double *bm = mob + ((z + 2) % 3) * S * MP;
        const double *bp = mob + ((z + 4) % 3) * S * MP;
        const double *pc = psi + ((z + 5) % 5) * S * PP;
        size_t zoff = (size_t) z << sh2;
        for(int i = tid; i < TX * TY; i += nthr) {
            int ly = i / TX, lx = i - ly * TX;
            int q = (ly + 1) * MX + (lx + 1);
            size_t gi = zoff + (x0 + lx) + ((y0 + ly) << g.log2N);
            if(!CHGB_BC(57, q - MX, MP) || !CHGB_BC(57, q + MX, MP) || !CHGB_BC(57, gi, bins)) continue;
#pragma unroll
            for(int s = 0; s < S; s++) {
                const double *u = uc + s * MP + q;
                double psi0 = pc[s * PP + (ly + 2) * PX + (lx + 2)];
                double res;
                if(MOB) {
                    const double *mm = bc + s * MP + q;
                    double mzm = bm[s * MP + q], mzp = bp[s * MP + q];
                    double uzm = um[s * MP + q], uzp = up[s * MP + q];
                    double jxp = (mm[0] + mm[1]) * (u[1] - u[0]);
                    double jxm = (mm[-1] + mm[0]) * (u[0] - u[-1]);
                    double jyp = (mm[0] + mm[MX]) * (u[MX] - u[0]);
                    double jym = (mm[-MX] + mm[0]) * (u[0] - u[-MX]);
                    double jzp = (mm[0] + mzp) * (uzp - u[0]);
                    double jzm = (mzm + mm[0]) * (u[0] - uzm);
                    double div = ((jxp - jxm) + (jyp - jym)) + (jzp - jzm);
                    res = fma(c.dt * c.half_inv_dx2, div, psi0);
                }
                else {
                    res = fma(c.c1, lap6(u[-1], u[1], u[-MX], u[MX], um[s * MP + q], up[s * MP + q], u[0]), psi0);
                }
                out[s * bins + gi] = res;
            }
        }
    };

    load_plane(z0 - 2);
    load_plane(z0 - 1);
    load_plane(z0);
    load_plane(z0 + 1);
    __syncthreads();
    mu_plane(z0 - 1);
    mu_plane(z0);
    for(int z = z0; z < z0 + zc; z++) {
        load_plane(z + 2);
        __syncthreads();
        mu_plane(z + 1);
        __syncthreads();
        out_plane(z);
    }
}

// ---------------------------------------------------------------------------
// Split step: kernel 1 writes mu (and the free-energy M) of every cell once,
// kernel 2 reads them back for the update.  No FP64 work is repeated on halo
// cells; the cost is 8 B (16 B with M) per cell and step of extra traffic,
// which is cheap next to the FP64 pipe on this part.  The arithmetic is the
// fused kernels' (the fixed-point sums do not depend on where the terms'
// fixed-point forms are made), so both variants give bit-identical results.
// Tiles are 32 x 8 cells per 256-thread block, one cell per thread; 3D
// marches over `zc` planes with a ring of three planes in shared memory.
// ---------------------------------------------------------------------------
// The plain (Landau, constant-mobility) split kernels are compiled for eight
// CTAs per SM (32 registers a thread): with the plane prefetch in registers
// they would otherwise take 40-46 and fit five or six (3D N=256 on GB300:
// 5.9e10 cell-steps/s at five, 6.5e10 at eight).  The other models' kernels
// need more registers than that and keep the default.
constexpr int STX = 32, STY = 8, SPX = STX + 2, SPY = STY + 2, SPP = SPX * SPY;

// Programmatic dependent launch of the split pair: each kernel waits for the
// previous kernel of the stream to finish (and its writes to land) before its
// first global access, then lets the next kernel's CTAs be placed on the SMs
// this grid no longer needs, which hides the launch gap between the two
// kernels of a step and between steps.  Without the launch attribute the wait
// returns at once.  (Measured on GB300: 2D N=1024 split step 25.9 -> 25.1 us,
// N=256 4.5 -> 4.2 us; the 3D N=256 step is unchanged.  The fused kernels,
// whose single wave would then hold idle waiting CTAs, do not use it.)

template <int DIMS, int S>
__device__ __forceinline__ void split_load_plane(double (*dst)[SPP], const double *__restrict__ src, const Geom &g,
                                                 int x0, int y0, int z, size_t bins, int tid) {
    const size_t zoff = (DIMS == 3) ? ((size_t) (z & g.mask) << (2 * g.log2N)) : 0;
    for(int i = tid; i < SPP; i += STX * STY) {
        int ly = i / SPX, lx = i - ly * SPX;
        int gx = (x0 - 1 + lx) & g.mask, gy = (y0 - 1 + ly) & g.mask;
        size_t gi = zoff + gx + ((size_t) gy << g.log2N);
#pragma unroll
        for(int s = 0; s < S; s++)
            if(CHGB_BC(1, gi, bins)) dst[s][i] = src[s * bins + gi];
    }
}

// The same plane load for a single-species field, also storing each value's
// fixed-point form (fx_term) for the neighbour sums.
template <int DIMS>
__device__ __forceinline__ void split_load_plane_fx(double *dst, long long *dT, int *dE, const double *__restrict__ src,
                                                    const Geom &g, int x0, int y0, int z, int tid) {
    const size_t zoff = (DIMS == 3) ? ((size_t) (z & g.mask) << (2 * g.log2N)) : 0;
    for(int i = tid; i < SPP; i += STX * STY) {
        int ly = i / SPX, lx = i - ly * SPX;
        int gx = (x0 - 1 + lx) & g.mask, gy = (y0 - 1 + ly) & g.mask;
        const size_t gi = zoff + gx + ((size_t) gy << g.log2N);
        const double v = CHGB_BC(2, gi, g.bins) ? src[gi] : 0.0;
        dst[i] = v;
        fx_term(v, dT[i], dE[i]);
    }
}

// The same, in two halves: fetch a plane's values into registers (two per
// thread: 340 values, 256 threads), then store them with their fixed-point
// forms.  The 3D kernels fetch plane z + 2 while they compute plane z, so the
// global-memory latency of staging is not waited for at the barrier.
constexpr int SPF = (SPP + STX * STY - 1) / (STX * STY);

template <int DIMS>
__device__ __forceinline__ void split_fetch_plane(double (&v)[SPF], const double *__restrict__ src, const Geom &g,
                                                  int x0, int y0, int z, int tid) {
    const size_t zoff = (DIMS == 3) ? ((size_t) (z & g.mask) << (2 * g.log2N)) : 0;
#pragma unroll
    for(int k = 0; k < SPF; k++) {
        const int i = tid + k * STX * STY;
        if(i < SPP) {
            int ly = i / SPX, lx = i - ly * SPX;
            int gx = (x0 - 1 + lx) & g.mask, gy = (y0 - 1 + ly) & g.mask;
            const size_t gi = zoff + gx + ((size_t) gy << g.log2N);
            v[k] = CHGB_BC(3, gi, g.bins) ? src[gi] : 0.0;
        }
    }
}

__device__ __forceinline__ void split_commit_plane_fx(double *dst, long long *dT, int *dE, const double (&v)[SPF],
                                                      int tid) {
#pragma unroll
    for(int k = 0; k < SPF; k++) {
        const int i = tid + k * STX * STY;
        if(i < SPP) {
            dst[i] = v[k];
            fx_term(v[k], dT[i], dE[i]);
        }
    }
}

// Neighbour sum of the cell at p of a staged plane ring (fixed-point forms
// computed at staging): planes c (the cell's), zm and zp (3D).
template <int DIMS, bool INT_ROUND>
__device__ __forceinline__ double split_nb_sum_fx(const double (*ring)[SPP], const long long (*rT)[SPP],
                                                  const int (*rE)[SPP], int c, int zm, int zp, int p) {
    constexpr int K = 2 * DIMS;
    long long T[K];
    int ek[K];
    const int off[4] = {-1, 1, -SPX, SPX};
    if(!CHGB_BC(7, p - SPX, SPP) || !CHGB_BC(7, p + SPX, SPP)) return 0.0;
#pragma unroll
    for(int i = 0; i < 4; i++) {
        T[i] = rT[c][p + off[i]];
        ek[i] = rE[c][p + off[i]];
    }
    if constexpr(DIMS == 3) {
        T[4] = rT[zm][p];
        ek[4] = rE[zm][p];
        T[5] = rT[zp][p];
        ek[5] = rE[zp][p];
    }
    const int emax = fx_emax<K>(ek);
    if(!fx_in_range(emax)) {
        const double *q = &ring[c][p];
        return seq_sum(q[-1], q[1], q[-SPX], q[SPX], DIMS == 3 ? ring[zm][p] : 0.0, DIMS == 3 ? ring[zp][p] : 0.0, K);
    }
    return fx_total<K, INT_ROUND>(T, ek, emax);
}

// The Laplacian's numerator at p of a staged plane ring: the neighbour sum
// minus 2 dims times the centre, rounded once (fx_lap).
template <int DIMS>
__device__ __forceinline__ double split_lap_fx(const double (*ring)[SPP], const long long (*rT)[SPP],
                                               const int (*rE)[SPP], int c, int zm, int zp, int p) {
    constexpr int K = 2 * DIMS;
    long long T[K];
    int ek[K];
    const int off[4] = {-1, 1, -SPX, SPX};
    if(!CHGB_BC(7, p - SPX, SPP) || !CHGB_BC(7, p + SPX, SPP)) return 0.0;
#pragma unroll
    for(int i = 0; i < 4; i++) {
        T[i] = rT[c][p + off[i]];
        ek[i] = rE[c][p + off[i]];
    }
    if constexpr(DIMS == 3) {
        T[4] = rT[zm][p];
        ek[4] = rE[zm][p];
        T[5] = rT[zp][p];
        ek[5] = rE[zp][p];
    }
    const long long Tv = rT[c][p];
    const int ekv = rE[c][p];
    int emax = fx_emax<K>(ek);
    emax = ekv > emax ? ekv : emax;
    if(!fx_in_range(emax)) {
        const double *q = &ring[c][p];
        return fma(-2.0 * DIMS, q[0],
                   seq_sum(q[-1], q[1], q[-SPX], q[SPX], DIMS == 3 ? ring[zm][p] : 0.0, DIMS == 3 ? ring[zp][p] : 0.0, K));
    }
    return fx_total<K>(T, ek, emax, -(long long) K * Tv, ekv);
}

// CTAs an SM: eight for plain Landau; the integer Wertheim models, whose chains
// are long, five in 3D and six in 2D (48 and 40 registers; simple_wertheim with
// the free-energy mobility, us a step with the compiler's choice, 4, 5, 6: 3D
// N=64 19.4 17.4 18.9 21.0, N=128 77.7 73.5 72.8 75.4, N=256 536 506 490 492;
// 2D N=2048 118.1 118.0 117.7 113.7).
template <int KIND, int MOB, int DIMS>
constexpr int MU_CTAS = KIND == CHGB_MODEL_LANDAU && MOB == 0 ? 8
                        : KIND == CHGB_MODEL_SIMPLE_WERTHEIM  ? (DIMS == 3 ? 5 : 6)
                                                              : 1;

template <int KIND, int MOB, int DIMS>
__global__ void __launch_bounds__(256, MU_CTAS<KIND, MOB, DIMS>) mu_kernel(const double *__restrict__ in, double *__restrict__ mu,
                                                 double *__restrict__ mob, Geom g, ModelDev m, EulerConsts c, int zc,
                                                 unsigned *__restrict__ key) {
    constexpr int S = NSpecies<KIND>::value;
    constexpr int R = (DIMS == 3) ? 3 : 1;
    // single species: each staged value's fixed-point form is computed once,
    // at staging, instead of at each of its seven uses
    constexpr bool PRE = S == 1;
    constexpr bool KEYED = S == 1 && (MOB == 1 || MOB == 2);   // the forms update_mob_fx_kernel follows
    __shared__ double ring[R][S][SPP];
    __shared__ long long ringT[PRE ? R : 1][PRE ? SPP : 1];
    __shared__ int ringE[PRE ? R : 1][PRE ? SPP : 1];
    const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + STX * ty;
    const int x0 = blockIdx.x * STX, y0 = blockIdx.y * STY;
    const int z0 = (DIMS == 3) ? blockIdx.z * zc : 0;
    const int nz = (DIMS == 3) ? zc : 1;
    const size_t bins = (size_t) g.bins;
    const int p = (ty + 1) * SPX + (tx + 1);
    auto stage = [&](int slot, int z) {
        if constexpr(PRE) split_load_plane_fx<DIMS>(ring[slot][0], ringT[slot], ringE[slot], in, g, x0, y0, z, tid);
        else split_load_plane<DIMS, S>(ring[slot], in, g, x0, y0, z, bins, tid);
    };
    pdl_begin();
    unsigned top_mu = 0, top_mob = 0;   // with a key: the largest high words of |mu| and |M|
    double pf[SPF];   // plane z + 1, fetched during the previous plane (3D single species)
    if constexpr(DIMS == 3) {
        stage((z0 + 2) % 3, z0 - 1);
        stage(z0 % 3, z0);
        if constexpr(PRE) split_fetch_plane<DIMS>(pf, in, g, x0, y0, z0 + 1, tid);
    }
    for(int z = z0; z < z0 + nz; z++) {
        const int cz = (DIMS == 3) ? z % 3 : 0;
        if constexpr(DIMS == 3 && PRE) {
            split_commit_plane_fx(ring[(z + 1) % 3][0], ringT[(z + 1) % 3], ringE[(z + 1) % 3], pf, tid);
            if(z + 1 < z0 + nz) split_fetch_plane<DIMS>(pf, in, g, x0, y0, z + 2, tid);
        }
        else if constexpr(DIMS == 3) stage((z + 1) % 3, z + 1);
        else stage(0, 0);
        __syncthreads();
        double r[S], d[S];
#pragma unroll
        for(int s = 0; s < S; s++) r[s] = ring[cz][s][p];
        const double xsw = der_bulk_x<KIND, MOB>(m, r, d);
        const size_t gi = (size_t) (x0 + tx) + ((size_t) (y0 + ty) << g.log2N) +
                          ((DIMS == 3) ? ((size_t) z << (2 * g.log2N)) : 0);
#pragma unroll
        for(int s = 0; s < S; s++) {
            const double *q = &ring[cz][s][p];
            double sum;
            if constexpr(PRE)
                // 2D Landau: four neighbours leave the integer pipes room, while the
                // mu spends three FP64 instructions of its own -- round in integers
                // (measured on GB300: 2D N=1024 5.92e10 -> 6.23e10 cell-steps/s; in 3D
                // the six-neighbour sum already fills the integer pipe, 5.52e10 -> 5.11e10)
                sum = split_nb_sum_fx<DIMS, KIND == CHGB_MODEL_LANDAU && DIMS == 2>(
                    reinterpret_cast<const double (*)[SPP]>(&ring[0][0][0]), ringT, ringE, cz, (z + 2) % 3, (z + 1) % 3, p);
            else
                sum = (DIMS == 3) ? nb_sum6(q[-1], q[1], q[-SPX], q[SPX], ring[(z + 2) % 3][s][p], ring[(z + 1) % 3][s][p])
                                  : nb_sum4(q[-1], q[1], q[-SPX], q[SPX]);
            const double mv = mu_cell<KIND, DIMS>(m, c, s, r[s], d[s], sum);
            if(CHGB_BC(4, gi, bins)) mu[s * bins + gi] = mv;
            if(KEYED) top_mu = max(top_mu, (unsigned) fx_mag(mv));
            if(MOB == 2) {
                const double Mv = c.M * xsw;
                mob[s * bins + gi] = Mv;
                top_mob = max(top_mob, (unsigned) fx_mag(Mv));
            }
        }
        __syncthreads();
    }
    if constexpr(KEYED) {
        if(key) {
            __shared__ unsigned top[2][STY];
            top_mu = __reduce_max_sync(0xFFFFFFFFu, top_mu);
            top_mob = __reduce_max_sync(0xFFFFFFFFu, top_mob);
            if(tx == 0) {
                top[0][ty] = top_mu;
                top[1][ty] = top_mob;
            }
            __syncthreads();
            if(tid < 2) {
                unsigned v = top[tid][0];
                for(int w = 1; w < STY; w++) v = max(v, top[tid][w]);
                atomicMax(&key[tid], v);
            }
        }
    }
}

template <int S, int MOB, int DIMS>
__global__ void __launch_bounds__(256, (S == 1 && MOB == 0) ? 8 : 1) update_kernel(const double *__restrict__ psi_in, const double *__restrict__ mu,
                                                     const double *__restrict__ mob, double *__restrict__ out, Geom g,
                                                     EulerConsts c, int zc) {
    constexpr int R = (DIMS == 3) ? 3 : 1;
    constexpr bool MFIELD = MOB >= 2;   // per-cell mobility read from `mob` (written by mu_kernel or given)
    constexpr int MR = MFIELD ? R : 1;
    constexpr bool PRE = S == 1 && MOB == 0;   // fixed-point forms staged with mu (see mu_kernel)
    // single-species euler_mobility: each face flux (M_i + M_j)(mu_j - mu_i) is
    // formed once -- x and y faces of a plane in shared memory, the z face
    // carried from one plane to the next in a register -- instead of once by
    // each of its two cells.  Same expression, so the same bits.
    constexpr bool FACES = S == 1 && MOB != 0;
    constexpr int FXW = STX + 1, FXN = FXW * STY, FYN = STX * (STY + 1);
    __shared__ double ring[R][S][SPP];
    __shared__ double mring[MR][MFIELD ? S : 1][MFIELD ? SPP : 1];
    __shared__ double fx[FACES ? FXN : 1], fy[FACES ? FYN : 1];
    __shared__ long long ringT[PRE ? R : 1][PRE ? SPP : 1];
    __shared__ int ringE[PRE ? R : 1][PRE ? SPP : 1];
    const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + STX * ty;
    const int x0 = blockIdx.x * STX, y0 = blockIdx.y * STY;
    const int z0 = (DIMS == 3) ? blockIdx.z * zc : 0;
    const int nz = (DIMS == 3) ? zc : 1;
    const size_t bins = (size_t) g.bins;
    const int p = (ty + 1) * SPX + (tx + 1);
    auto stage = [&](int slot, int z) {
        if constexpr(PRE) split_load_plane_fx<DIMS>(ring[slot][0], ringT[slot], ringE[slot], mu, g, x0, y0, z, tid);
        else split_load_plane<DIMS, S>(ring[slot], mu, g, x0, y0, z, bins, tid);
    };
    pdl_begin();
    double pf[SPF];   // plane z + 1 of mu, fetched during the previous plane (3D single species)
    double jz_prev = 0.0;   // FACES, 3D: the z face below the next plane (this plane's upper face)
    if constexpr(DIMS == 3) {
        stage((z0 + 2) % 3, z0 - 1);
        stage(z0 % 3, z0);
        if constexpr(PRE) split_fetch_plane<DIMS>(pf, mu, g, x0, y0, z0 + 1, tid);
        if constexpr(MFIELD) {
            split_load_plane<DIMS, S>(mring[(z0 + 2) % 3], mob, g, x0, y0, z0 - 1, bins, tid);
            split_load_plane<DIMS, S>(mring[z0 % 3], mob, g, x0, y0, z0, bins, tid);
        }
    }
    for(int z = z0; z < z0 + nz; z++) {
        const int cz = (DIMS == 3) ? z % 3 : 0, zm = (z + 2) % 3, zp = (z + 1) % 3;
        const size_t gi = (size_t) (x0 + tx) + ((size_t) (y0 + ty) << g.log2N) +
                          ((DIMS == 3) ? ((size_t) z << (2 * g.log2N)) : 0);
        // the cell's psi is read before the plane is staged, so that its
        // latency overlaps the staging and the barrier
        double psi_cell[S];
#pragma unroll
        for(int s = 0; s < S; s++) psi_cell[s] = CHGB_BC(5, gi, bins) ? psi_in[s * bins + gi] : 0.0;
        if constexpr(DIMS == 3) {
            if constexpr(PRE) {
                split_commit_plane_fx(ring[zp][0], ringT[zp], ringE[zp], pf, tid);
                if(z + 1 < z0 + nz) split_fetch_plane<DIMS>(pf, mu, g, x0, y0, z + 2, tid);
            }
            else stage(zp, z + 1);
            if constexpr(MFIELD) split_load_plane<DIMS, S>(mring[zp], mob, g, x0, y0, z + 1, bins, tid);
        }
        else {
            stage(0, 0);
            if constexpr(MFIELD) split_load_plane<DIMS, S>(mring[0], mob, g, x0, y0, 0, bins, tid);
        }
        __syncthreads();
        if constexpr(FACES) {
            // x face f between tile columns lx - 1 and lx (lx in 0..STX), y face
            // between tile rows ly - 1 and ly (ly in 0..STY)
            for(int f = tid; f < FXN + FYN; f += STX * STY) {
                int a, b;
                if(f < FXN) {
                    const int ly = f / FXW, lx = f - ly * FXW;
                    a = (ly + 1) * SPX + lx;
                    b = a + 1;
                }
                else {
                    const int g2 = f - FXN, ly = g2 / STX, lx = g2 - ly * STX;
                    a = ly * SPX + lx + 1;
                    b = a + SPX;
                }
                const double ma = MFIELD ? mring[cz][0][a] : c.M, mb = MFIELD ? mring[cz][0][b] : c.M;
                const double j = (ma + mb) * (ring[cz][0][b] - ring[cz][0][a]);
                if(f < FXN) fx[f] = j;
                else fy[f - FXN] = j;
            }
            __syncthreads();
        }
#pragma unroll
        for(int s = 0; s < S; s++) {
            const double *u = &ring[cz][s][p];
            const double psi0 = psi_cell[s];
            double res;
            if(FACES) {
                const double jxm = fx[ty * FXW + tx], jxp = fx[ty * FXW + tx + 1];
                const double jym = fy[ty * STX + tx], jyp = fy[(ty + 1) * STX + tx];
                double div = (jxp - jxm) + (jyp - jym);
                if(DIMS == 3) {
                    const double m0 = MFIELD ? mring[cz][s][p] : c.M;
                    const double mzp = MFIELD ? mring[zp][s][p] : c.M;
                    const double jzp = (m0 + mzp) * (ring[zp][s][p] - u[0]);
                    double jzm;
                    if(z == z0) {
                        const double mzm = MFIELD ? mring[zm][s][p] : c.M;
                        jzm = (mzm + m0) * (u[0] - ring[zm][s][p]);
                    }
                    else {
                        jzm = jz_prev;
                    }
                    jz_prev = jzp;
                    div = div + (jzp - jzm);
                }
                res = fma(c.dt * c.half_inv_dx2, div, psi0);
            }
            else if(MOB) {
                double m0, mxm, mxp, mym, myp, mzm = 0, mzp = 0;
                if(MFIELD) {
                    const double *mm = &mring[cz][s][p];
                    m0 = mm[0];
                    mxm = mm[-1];
                    mxp = mm[1];
                    mym = mm[-SPX];
                    myp = mm[SPX];
                    if(DIMS == 3) {
                        mzm = mring[zm][s][p];
                        mzp = mring[zp][s][p];
                    }
                }
                else {
                    m0 = mxm = mxp = mym = myp = mzm = mzp = c.M;
                }
                double jxp = (m0 + mxp) * (u[1] - u[0]);
                double jxm = (mxm + m0) * (u[0] - u[-1]);
                double jyp = (m0 + myp) * (u[SPX] - u[0]);
                double jym = (mym + m0) * (u[0] - u[-SPX]);
                double div = (jxp - jxm) + (jyp - jym);
                if(DIMS == 3) {
                    double jzp = (m0 + mzp) * (ring[zp][s][p] - u[0]);
                    double jzm = (mzm + m0) * (u[0] - ring[zm][s][p]);
                    div = div + (jzp - jzm);
                }
                res = fma(c.dt * c.half_inv_dx2, div, psi0);
            }
            else {
                double lap;
                if constexpr(PRE)
                    lap = split_lap_fx<DIMS>(reinterpret_cast<const double (*)[SPP]>(&ring[0][0][0]), ringT, ringE, cz,
                                             zm, zp, p);
                else
                    lap = (DIMS == 3) ? lap6(u[-1], u[1], u[-SPX], u[SPX], ring[zm][s][p], ring[zp][s][p], u[0])
                                      : lap4(u[-1], u[1], u[-SPX], u[SPX], u[0]);
                res = fma(c.c1, lap, psi0);
            }
            if(CHGB_BC(6, gi, bins)) out[s * bins + gi] = res;
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// The update of euler_mobility in block fixed point (kernel_variant 5,
// one species, constant or free-energy mobility): mu_kernel writes mu and M and
// folds their largest magnitudes into a key; here one exponent for each serves
// the field, U = mu 2^(60-su) and W = M 2^(60-sm) are integers below 2^60, a
// face's flux (W_a + W_b)(U_b - U_a) is the upper part, in units of 2^62, of one
// product on IMAD.WIDE (a constant M: the difference itself, |U| < 2^59), and
// the divergence an int64 sum -- the same integer for both cells of a face, so
// the fluxes cancel exactly.  Per face the integers are off by one unit with a
// constant M (half a one for each U) and by three else (half a one each for W and
// the difference, two for the product's upper part).  They are taken where all
// that stays below 2^-56 of psi, an eighth of its last place; a warp (32 x 4 cells
// of each plane) with a density for which it does not, many decades below the
// field's largest, does the step in FP64.  (A Landau field passes through zero,
// where its value does not tell the scale of what is summed there: the warp's
// largest value stands for it.)  A cell takes two FP64 instructions (a conversion
// and the final FMA) where update_kernel takes 16, which bound it (75 % of that
// pipe).  simple_wertheim with the free-energy mobility on GB300, us a step (mu
// and update), the FP64 update and this one: 3D N=32 8.6 and 7.2, N=64 28.6 and
// 17.1, N=128 128.8 and 71.6, N=256 901 and 483; 2D N=512 16.4 and 11.9, N=1024
// 47.8 and 31.7.  A field of twelve decades, N=128: 287 and 122.
//
// A CTA of 128 threads has a tile of 32 x 16 cells, a warp each of four rows
// of it: a thread's four cells lie above one another, so that their y faces are
// formed once but for the warps' borders and the z faces carried from plane to
// plane; x faces come from the lane to the left, the tile's left ones from one
// extra product of lanes 0-3.  One barrier a plane, the next plane's values in
// flight during it.
// ---------------------------------------------------------------------------
constexpr int MTX = 32, MTY = 16, MTHR = 128, MPX = MTX + 2, MPP = MPX * (MTY + 2);
constexpr int MPF = (MPP + MTHR - 1) / MTHR;

// a b 2^-62, |a| and |b| below 2^61 (within 2 units, the same way for every pair).
__device__ __forceinline__ long long face_flux(long long a, long long b) {
    const int ah = (int) (a >> 31), al = (int) a & 0x7FFFFFFF, bh = (int) (b >> 31), bl = (int) b & 0x7FFFFFFF;
    return wide(ah, bh) + (wide(ah, bl, wide(al, bh)) >> 31);
}

// The step of a warp's cells (32 x 4 of each of `d` planes; a thread has a column of
// four) in FP64, for fields outside the integer path's range (zeros, NaN,
// infinities, exponents near the ends) and warps outside its precision.  A thread
// forms the y faces between its cells and the z faces between planes once (N=128, a
// field of twelve decades, 142 -> 122 us a step; one with a Landau spot 110 -> 98).
template <int DIMS, bool CONST>
__device__ __noinline__ void mob_slow_cells(const double *__restrict__ psi, const double *__restrict__ mu,
                                            const double *__restrict__ mob, double *__restrict__ out, int mask,
                                            int log2N, double M, double k, int x, int y0, int z0, int d) {
    const unsigned xm = (x - 1) & mask, xp = (x + 1) & mask;
    auto row = [&](int Y, int Z) {   // below 2^30
        return ((unsigned) (Y & mask) << log2N) + (DIMS == 3 ? (unsigned) (Z & mask) << (2 * log2N) : 0u);
    };
    auto W = [&](unsigned c) { return CONST ? M : mob[c]; };
    double jz[4] = {0.0, 0.0, 0.0, 0.0};
    if constexpr(DIMS == 3)
#pragma unroll
        for(int r = 0; r < 4; r++) {
            const unsigned c = row(y0 + r, z0) + x, b = row(y0 + r, z0 - 1) + x;
            jz[r] = (W(b) + W(c)) * (mu[c] - mu[b]);
        }
    for(int z = z0; z < z0 + d; z++) {
        const unsigned below = row(y0 - 1, z) + x;
        double u = mu[row(y0, z) + x], w = W(row(y0, z) + x);
        double jym = (W(below) + w) * (u - mu[below]);
#pragma unroll
        for(int r = 0; r < 4; r++) {
            const unsigned line = row(y0 + r, z), c = line + x, n = row(y0 + r + 1, z) + x;
            const double un = mu[n], wn = W(n), jyp = (w + wn) * (un - u);
            const double jxp = (w + W(line + xp)) * (mu[line + xp] - u), jxm = (W(line + xm) + w) * (u - mu[line + xm]);
            double div = (jxp - jxm) + (jyp - jym);
            if constexpr(DIMS == 3) {
                const unsigned a = row(y0 + r, z + 1) + x;
                const double jzp = (w + W(a)) * (mu[a] - u);
                div = div + (jzp - jz[r]);
                jz[r] = jzp;
            }
            if(CHGB_BC(20, c, (long long) 1 << (DIMS * log2N))) out[c] = fma(k, div, psi[c]);
            jym = jyp;
            u = un;
            w = wn;
        }
    }
}

// CTAs an SM the registers are limited for.  2D: eight, 64 registers (2D N=512 14.1
// -> 11.9 us a step).  3D: five (96 registers instead of 112) where the launch has
// as many CTAs, none for the small boxes (free-energy mobility, us a step without and
// with the limit: N=256 491 and 483, N=128 72.4 and 72.2, with three boxes at once
// 61.2 and 59.9; N=64 17.4 and 18.1, N=32 7.6 and 8.6).
template <int DIMS, bool CONST, bool DENSITY, int CTAS>
__global__ void __launch_bounds__(MTHR, CTAS) update_mob_fx_kernel(const double *__restrict__ psi_in,
                                                             const double *__restrict__ mu,
                                                             const double *__restrict__ mob, double *__restrict__ out,
                                                             Geom g, EulerConsts c, int zc, unsigned *__restrict__ key,
                                                             int parity) {
    constexpr int R = DIMS == 3 ? 3 : 1;
    constexpr int WR = CONST ? 1 : R, WP = CONST ? 1 : MPP;
    __shared__ long long rU[R][MPP], rW[WR][WP];
    const int tid = threadIdx.x, tx = tid & 31, row0 = (tid >> 5) * 4;
    const int x0 = blockIdx.x * MTX, y0 = blockIdx.y * MTY, z0 = DIMS == 3 ? blockIdx.z * zc : 0;
    const int nz = DIMS == 3 ? zc : 1;
    pdl_begin();
    const int eu = (int) (__ldcg(&key[2 * parity]) >> 20), ew = CONST ? 1022 : (int) (__ldcg(&key[2 * parity + 1]) >> 20);
    if(tid < 2 && blockIdx.x + blockIdx.y + blockIdx.z == 0) key[2 * (parity ^ 1) + tid] = 0;   // the next step's
    // the flux's unit is 2^(62 + (su - 60) + (sm - 60)), s = e - 1022, or with a
    // constant M, whose sum of two goes into k, 2^(su - 59)
    const int ek = CONST ? eu - 1022 - 59 : eu + ew - 2 * 1022 - 58;
    const double kd = c.dt * c.half_inv_dx2;
    bool safe = eu >= 300 && eu <= 1700 && ew >= 300 && ew <= 1700 && ek >= -800 && ek <= 800;
    if(safe) {
        const double k = (CONST ? kd * (c.M + c.M) : kd) * __hiloint2double((1023 + ek) << 20, 0);
        // psi above this (by its high word) is safe from the integers' error
        const int least = fx_mag(k * ((CONST ? 2.0 : 6.0) * DIMS * 0x1p56));
        int seen = DENSITY ? 0x7FFFFFFF : 0;   // the least, or the largest, of the thread's |psi|
        FxScale su, sw;
        su.sh = (CONST ? 59 : 60) - (eu - 1022);
        sw.sh = 60 - (ew - 1022);
        // this thread's cells of a staged plane
        int off[MPF];
#pragma unroll
        for(int i = 0; i < MPF; i++) {
            const int q = tid + i * MTHR, ly = q / MPX, lx = q - ly * MPX;
            off[i] = ((x0 - 1 + lx) & g.mask) + (((y0 - 1 + ly) & g.mask) << g.log2N);
        }
        auto plane = [&](int z) { return DIMS == 3 ? (size_t) (z & g.mask) << (2 * g.log2N) : 0; };
        double fu[MPF], fw[MPF];
        auto fetch = [&](int z) {
            const size_t b = plane(z);
#pragma unroll
            for(int i = 0; i < MPF; i++) {
                const bool in = tid + i * MTHR < MPP && CHGB_BC(18, b + off[i], g.bins);
                fu[i] = in ? mu[b + off[i]] : 0.0;
                if(!CONST) fw[i] = in ? mob[b + off[i]] : 0.0;
            }
        };
        auto commit = [&](int slot) {
#pragma unroll
            for(int i = 0; i < MPF; i++) {
                const int q = tid + i * MTHR;
                if(q < MPP) {
                    rU[slot][q] = fx_in(fu[i], su);
                    if(!CONST) rW[slot][q] = fx_in(fw[i], sw);
                }
            }
        };
        auto flux = [&](long long wa, long long wb, long long d) { return CONST ? d : face_flux(wa + wb, d); };
        auto W = [&](int slot, int p) { return CONST ? 0 : rW[CONST ? 0 : slot][CONST ? 0 : p]; };
        const int p0 = (row0 + 1) * MPX + tx + 1;   // the thread's first cell in a staged plane
        const size_t c0 = (size_t) (x0 + tx) + ((size_t) (y0 + row0) << g.log2N);
        long long jz[4] = {0, 0, 0, 0};
        fetch(z0);
        commit(DIMS == 3 ? z0 % 3 : 0);
        if constexpr(DIMS == 3) {
            fetch(z0 + 1);
            // the lowest z faces: the plane below is needed at the thread's own cells only
            __syncthreads();
            const size_t b = plane(z0 - 1) + c0;
#pragma unroll
            for(int r = 0; r < 4; r++) {
                const size_t gi = b + ((size_t) r << g.log2N);
                const bool in = CHGB_BC(19, gi, g.bins);
                const long long u = fx_in(in ? mu[gi] : 0.0, su), w = CONST ? 0 : fx_in(in ? mob[gi] : 0.0, sw);
                const int p = p0 + r * MPX;
                jz[r] = flux(w, W(z0 % 3, p), rU[z0 % 3][p] - u);
            }
        }
        for(int z = z0; z < z0 + nz; z++) {
            const int cz = DIMS == 3 ? z % 3 : 0, zp = DIMS == 3 ? (z + 1) % 3 : 0;
            const size_t b = plane(z) + c0;
            double psi[4];
#pragma unroll
            for(int r = 0; r < 4; r++) {
                const size_t gi = b + ((size_t) r << g.log2N);
                psi[r] = CHGB_BC(19, gi, g.bins) ? psi_in[gi] : 0.0;
            }
            if constexpr(DIMS == 3) {
                commit(zp);
                if(z + 1 < z0 + nz) fetch(z + 2);
            }
            __syncthreads();
            const long long *U = rU[cz];
            const int pe = (row0 + 1 + (tx & 3)) * MPX + 1;   // lanes 0-3: the tile's left faces of the four rows
            const long long edge = flux(W(cz, pe - 1), W(cz, pe), U[pe] - U[pe - 1]);
            long long u = U[p0], w = W(cz, p0);
            long long jym = flux(W(cz, p0 - MPX), w, u - U[p0 - MPX]);
#pragma unroll
            for(int r = 0; r < 4; r++) {
                const int p = p0 + r * MPX;
                const long long un = U[p + MPX], wn = W(cz, p + MPX);
                const long long jxp = flux(w, W(cz, p + 1), U[p + 1] - u), jyp = flux(w, wn, un - u);
                const long long left = __shfl_up_sync(0xFFFFFFFFu, jxp, 1), first = __shfl_sync(0xFFFFFFFFu, edge, r);
                long long D = (jxp - (tx == 0 ? first : left)) + (jyp - jym);
                if constexpr(DIMS == 3) {
                    const long long jzp = flux(w, W(zp, p), rU[zp][p] - u);
                    D += jzp - jz[r];
                    jz[r] = jzp;
                }
                jym = jyp;
                u = un;
                w = wn;
                const size_t gi = b + ((size_t) r << g.log2N);
                if(CHGB_BC(19, gi, g.bins)) out[gi] = fma(k, (double) D, psi[r]);
                seen = DENSITY ? min(seen, fx_mag(psi[r])) : max(seen, fx_mag(psi[r]));
            }
        }
        safe = seen > least;
    }
    if(!(DENSITY ? __all_sync(0xFFFFFFFFu, safe) : __any_sync(0xFFFFFFFFu, safe)))
        mob_slow_cells<DIMS, CONST>(psi_in, mu, mob, out, g.mask, g.log2N, c.M, kd, x0 + tx, y0 + row0, z0, nz);
}

// ---------------------------------------------------------------------------
// Block fixed point (kernel_variant 5: Landau `euler`): one kernel per step
// (euler2d_bfp_kernel, euler3d_bfp_kernel), and in 3D also a pair of kernels
// (mu_bfp_kernel, update_bfp_kernel), the same arithmetic and bits
// ---------------------------------------------------------------------------
// The split pair above aligns the terms of each neighbour sum to the largest
// exponent of that stencil: per cell a maximum over seven exponents and seven
// variable shifts, about half of a step's integer work.  Here one exponent
// serves the whole field for a step (block floating point, the field being the
// block), and mu is formed in integers throughout:
//   - psi: emax, the largest biased exponent of |psi| over the field, is read
//     from BfpState::key (below); |psi| < 2^s, s = emax - 1022.  Each value
//     becomes X = psi 2^(60-s) cut to an integer, |X| < 2^60, once, and a
//     neighbour sum S is a plain int64 sum, |S| < 2^62.6.
//   - mu = psi (psi^2 + lshift) - c2 sum.  With a = max(2 s, elin) (|lshift| +
//     2 D |c2| < 2^elin), |mu| < 2^(a+s+2) (one bit spare), and mu is stored as
//     M = mu 2^(56-a-s), |M| <= 2^57 + 1.  G = (psi^2 + lshift) 2^(61-a) =
//     (X^2 >> 59 + a - 2 s) + lsi, |G| < 2^62, and M = (X G 2^-64 +
//     S C 2^-64) >> 1, C = -c2 in the matching unit: the shifts do not depend
//     on the cell, the scales drop out.  All factors are taken as signed 32-bit
//     limbs (bfp.cuh), so the two products of M are eight IMAD.WIDE that
//     accumulate; the products of two low limbs are left out.  No FP64
//     instruction: FP64 issues at 1/64 of FP32's rate here, and the two that
//     psi (psi^2 + lshift) took were the pipe's larger share of a step.  27
//     instructions a cell; written as C++ products of sign-extended words they
//     were 42 (bfp.cuh, `wide`).
//   - the update: L = sum(M_nb) - 2 D M, exact (|L| < 2^61), and
//     psi' = psi + (c1 2^(a+s-56)) L: one int64 -> double rounding (on the FP64
//     pipe, or in the 2D kernel and the pair for every other cell in integers:
//     the same bits) and one FMA.
//     Each CTA folds the largest exponent of its psi' into the key.
// Errors, in units of M (mu's bound is 2^58 of them): X is cut 2^-60 below the
// field's bound, which enters c2 sum and psi^3 at less than 2^-58 of theirs; G
// drops at most 8 + 2 units of 2^-61 of its bound (X's low limb squared, the
// shifts), half a unit of M; the products' low limbs and shifts 1 unit; C's
// rounding 2^-4 unit.  So M is within 3 units of mu at the cut field, where the
// reference's FP64 products and sums round each at 2^-53 of their own value:
// at worst 2^-56 of mu's bound.  The results are not the other variants' bits.
// The key is (generation << 16) | emax, the largest of BFP_SLOTS 64-bit slots.
// A step reads generation g and folds each CTA's exponent into one slot of the
// other bank as ((g + 1) << 16) | e by atomicMax, so the newer generation
// supersedes the older with no reset between steps, and slots no CTA wrote in
// this step fall behind.  (The pair's mu kernel publishes g + 1, mu's exponent
// and the mode to its update kernel, BfpState::gen.)  Each chgb_step call first sets the key
// from the field (bfp_refresh_kernel, with a generation above all before it).  A field whose emax is
// below 128 or 2047 (zeros, values near the end of the double range, inf, NaN),
// or so large or small that mu's unit leaves [2^-900, 2^900], takes plain FP64
// sums in the reference's neighbour order for that step (mode 0).

// psi 2^(60-s) cut to an integer (`u` = emax, the biased exponent of 2^s's
// binade): the mantissa at the top of a word, down by 4 or more; its one's
// complement for negative values, the floor of all but whole ones.  Zeros and
// subnormals (the implicit bit set here does not belong) shift out: u >= 128.
__device__ __forceinline__ long long bfp_fixed(double x, int u) {
    const int hi = __double2hiint(x);
    const unsigned lo = (unsigned) __double2loint(x);
    const unsigned mh = __funnelshift_l(lo, (unsigned) hi, 11) | 0x80000000u;
    const unsigned long long m = fx_shr(((unsigned long long) mh << 32) | (lo << 11), u + 4 - ((hi >> 20) & 0x7FF));
    return (long long) (m ^ (unsigned long long) (long long) (hi >> 31));
}

// A step's scales, the same for every cell.
struct BfpScale {
    int emax, lmu, d;   // the field's exponent; M's unit is 2^lmu = 2^(a+s-56); a - 2 s
    int ch, cl;         // the limbs of C
    long long lsi;      // lshift in G's unit
    bool fast;
};

template <int DIMS>
__device__ __forceinline__ BfpScale bfp_scale(int emax, const EulerConsts &c, const BfpConsts &b) {
    BfpScale t;
    t.emax = emax;
    const int s = emax - 1022, a = max(2 * s, b.elin);
    t.lmu = a + s - 56;
    t.fast = emax >= 128 && emax <= 2046 && t.lmu >= -900 && t.lmu <= 900;
    t.d = min(a - 2 * s, 63);   // X^2 2^-59 is below 2^61: nothing is left of it from 62 on
    const double ls = c.lshift[DIMS - 1];
    // 2^(61-a): elin is at least -800 where lshift is not zero
    t.lsi = ls == 0.0 || !t.fast ? 0 : __double2ll_rn(ls * __hiloint2double((1023 + 61 - a) << 20, 0));
    // -c2 S 2^(s-60) in half units of M: mc is c2's mantissa times 2^10 and
    // 2^(1085-ec), so C = -mc 2^-(a+1024-ec), four or more places down, rounded:
    // the half is added in its own place, mc being up to 2^63 - 1024
    const int r = a + 1024 - b.ec;
    const long long C = r > 62 ? 0 : -(((b.mc >> (r - 1)) + 1) >> 1);
    t.ch = fx_hi(C);
    t.cl = fx_lo(C);
    return t;
}

// M of a cell from its X and neighbour sum.
__device__ __forceinline__ long long bfp_mu(long long X, long long S, const BfpScale &t) {
    const int xh = fx_hi(X), xl = fx_lo(X), sh = fx_hi(S), sl = fx_lo(S);
    const long long G = (((wide(xh, xh) << 5) + (wide(xh, xl) >> 26)) >> t.d) + t.lsi;
    const int gh = fx_hi(G), gl = fx_lo(G);
    const long long hi = wide(xh, gh, wide(sh, t.ch));
    const long long mid = wide(xh, gl, wide(xl, gh, wide(sh, t.cl, wide(sl, t.ch))));
    return (hi + (mid >> 32)) >> 1;
}

// L 2^0 as the nearest double: FP64 pipe, or the same bits in integers.
__device__ __forceinline__ double bfp_double_fp(long long L) { return __ll2double_rn(L); }
__device__ __forceinline__ double bfp_double_int(long long L) { return fx_nearest(L, 0); }

// Tiles of the 3D pair (taken where kernel_variant asks for 5 by number): 32 x
// 16 cells per 256-thread CTA, two cells adjacent in x per thread, marching
// over `zc` planes.  A thread keeps its own column of
// three planes in registers; the planes in shared memory (two, one barrier a
// plane) serve the x and y neighbours.  The tile's 96 halo cells are staged by
// three of the eight warps, the plane after next being fetched meanwhile.  Per
// cell this takes 2 + 2 shared loads of a pair's neighbours and half of each
// global access, where a 32 x 8 tile with one cell a thread (and the whole
// stencil in shared memory, 1.33 values staged a cell) took 7 and 1.33.
constexpr int BTX = 32, BTY = 16, BPITCH = BTX + 4, BPLANE = BPITCH * (BTY + 2);
constexpr int BHALO = 2 * BTX + 2 * BTY;

struct BfpTile {
    int own, halo;         // shared index of the own pair's left cell, of the halo cell (threads below BHALO)
    unsigned gown, ghalo;  // their offsets in a plane
    bool has_halo;
};

__device__ __forceinline__ BfpTile bfp_tile(const Geom &g, int tid) {
    BfpTile t;
    const int tx = tid & 15, ty = tid >> 4;
    const int x0 = blockIdx.x * BTX, y0 = blockIdx.y * BTY;
    t.own = (ty + 1) * BPITCH + 2 + 2 * tx;
    t.gown = (unsigned) (x0 + 2 * tx) + ((unsigned) (y0 + ty) << g.log2N);
    t.has_halo = tid < BHALO;
    int lx, ly;            // tile coordinates of the halo cell
    if(tid < 2 * BTX) {
        lx = tid & (BTX - 1);
        ly = tid < BTX ? -1 : BTY;
    }
    else {
        lx = tid < 2 * BTX + BTY ? -1 : BTX;
        ly = (tid - 2 * BTX) & (BTY - 1);
    }
    t.halo = (ly + 1) * BPITCH + 2 + lx;
    t.ghalo = (unsigned) ((x0 + lx) & g.mask) + ((unsigned) ((y0 + ly) & g.mask) << g.log2N);
    return t;
}

// x and y neighbours of the thread's pair in a staged plane: the pair's partial sums.
template <int PITCH>
__device__ __forceinline__ void bfp_xy_sums(const long long *plane, int own, long long a, long long b, long long &sa,
                                            long long &sb) {
    const longlong2 up = *reinterpret_cast<const longlong2 *>(plane + own - PITCH);
    const longlong2 dn = *reinterpret_cast<const longlong2 *>(plane + own + PITCH);
    sa = (plane[own - 1] + b) + (up.x + dn.x);
    sb = (a + plane[own + 2]) + (up.y + dn.y);
}

// Mode 0 (see above): the step of a w x h x d block of cells at (x0, y0, z0)
// by a whole CTA, from global memory, in FP64 and the reference's order of
// neighbours.  Returns the largest high word of the thread's |psi'|.  Not
// inlined: its registers would be the integer path's.
template <int DIMS>
__device__ __noinline__ int bfp_slow_block(const double *__restrict__ in, double *__restrict__ out, int mask, int log2N,
                                           double c1, double c2, double ls, int x0, int y0, int z0, int w, int h,
                                           int d) {
    auto index = [&](int X, int Y, int Z) {
        return (size_t) (X & mask) + ((size_t) (Y & mask) << log2N) +
               (DIMS == 3 ? ((size_t) (Z & mask) << (2 * log2N)) : 0);
    };
    auto psi = [&](int X, int Y, int Z) { return in[index(X, Y, Z)]; };
    auto mu = [&](int X, int Y, int Z) {
        const double r = psi(X, Y, Z);
        const double sum = seq_sum(psi(X - 1, Y, Z), psi(X + 1, Y, Z), psi(X, Y - 1, Z), psi(X, Y + 1, Z),
                                   DIMS == 3 ? psi(X, Y, Z - 1) : 0.0, DIMS == 3 ? psi(X, Y, Z + 1) : 0.0, 2 * DIMS);
        return fma(-c2, sum, r * fma(r, r, ls));
    };
    int mag = 0;
    for(int i = threadIdx.x; i < w * h * d; i += blockDim.x) {
        const int x = x0 + i % w, y = y0 + i / w % h, z = z0 + i / (w * h);
        const size_t gi = index(x, y, z);
        if(!CHGB_BC(17, gi, (long long) 1 << (DIMS * log2N))) continue;
        const double sum = seq_sum(mu(x - 1, y, z), mu(x + 1, y, z), mu(x, y - 1, z), mu(x, y + 1, z),
                                   DIMS == 3 ? mu(x, y, z - 1) : 0.0, DIMS == 3 ? mu(x, y, z + 1) : 0.0, 2 * DIMS);
        const double res = fma(c1, fma(-2.0 * DIMS, mu(x, y, z), sum), in[gi]);
        out[gi] = res;
        mag = max(mag, __double2hiint(res) & 0x7FFFFFFF);
    }
    return mag;
}

// The largest biased exponent of a block's per-thread values, given as the high
// words of |values|, folded into key slot `slot` as ((gen << 16) | e) by one
// atomicMax.  The CTAs of a launch spread over BFP_SLOTS
// slots, one 128-byte line each, so that their atomics do not queue on one
// address.
template <int WARPS>
__device__ __forceinline__ void bfp_fold_key(int mag, unsigned long long gen, unsigned long long *bank, int slot,
                                             int tid) {
    __shared__ int wmax[WARPS];
    const int e = __reduce_max_sync(0xffffffffu, mag);
    if((tid & 31) == 0) wmax[tid >> 5] = e;
    __syncthreads();
    if(tid == 0) {
        int m = wmax[0];
#pragma unroll
        for(int w = 1; w < WARPS; w++) m = wmax[w] > m ? wmax[w] : m;
        atomicMax(&bank[(slot % BFP_SLOTS) * BFP_SLOT_STRIDE], (gen << 16) | (unsigned long long) (m >> 20));
    }
}

// The field's key: the largest of the slots (the newest generation, then the
// largest exponent), read by warp 0 and shared through shared memory, so that
// one load per CTA reaches each slot's line.
__device__ __forceinline__ unsigned long long bfp_read_key(const unsigned long long *bank, int tid) {
    __shared__ unsigned long long s_key;
    if(tid < 32) {
        unsigned long long k = *(const volatile unsigned long long *) &bank[tid * BFP_SLOT_STRIDE];
#pragma unroll
        for(int o = 16; o > 0; o >>= 1) {
            const unsigned long long t = __shfl_xor_sync(0xffffffffu, k, o);
            k = t > k ? t : k;
        }
        if(tid == 0) s_key = k;
    }
    __syncthreads();
    return s_key;
}

__global__ void __launch_bounds__(256, 5) mu_bfp_kernel(const double *__restrict__ in, long long *__restrict__ mu,
                                                        Geom g, EulerConsts c, BfpConsts b, BfpState *st, int parity,
                                                        int zc) {
    __shared__ __align__(16) long long ring[2][BPLANE];
    const int tid = threadIdx.x;
    pdl_begin();
    const unsigned long long key = bfp_read_key(st->key[parity], tid);
    const BfpScale sc = bfp_scale<3>((int) (key & 0xFFFFu), c, b);
    if(blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && tid == 0) {
        st->gen = (key >> 16) + 1;
        st->lmu = sc.lmu;
        st->mode = sc.fast ? 1 : 0;
    }
    const BfpTile t = bfp_tile(g, tid);
    const int z0 = blockIdx.z * zc;
    if(!sc.fast) return;   // the update kernel does the whole step
    auto plane = [&](int z) { return (unsigned) (z & g.mask) << (2 * g.log2N); };   // element offsets: below 2^30
    auto pair = [&](int z) {
        const unsigned gi = plane(z) + t.gown;
        return CHGB_BC(11, gi + 1, g.bins) ? *reinterpret_cast<const double2 *>(in + gi) : make_double2(0.0, 0.0);
    };
    auto fixed = [&](double2 v) { return make_longlong2(bfp_fixed(v.x, sc.emax), bfp_fixed(v.y, sc.emax)); };
    auto halo = [&](int z) {
        return t.has_halo && CHGB_BC(12, plane(z) + t.ghalo, g.bins) ? in[plane(z) + t.ghalo] : 0.0;
    };
    auto stage = [&](int z, longlong2 X, double h) {
        long long *p = ring[z & 1];
        if(CHGB_BC(13, t.own + 1, BPLANE)) *reinterpret_cast<longlong2 *>(p + t.own) = X;
        if(t.has_halo && CHGB_BC(13, t.halo, BPLANE)) p[t.halo] = bfp_fixed(h, sc.emax);
    };
    const longlong2 Xfirst = fixed(pair(z0 - 1));
    longlong2 Xm = Xfirst, Xc = fixed(pair(z0));
    stage(z0, Xc, halo(z0));
    double2 next = pair(z0 + 1);
    double hnext = zc > 1 ? halo(z0 + 1) : 0.0;
    for(int z = z0; z < z0 + zc; z++) {
        __syncthreads();   // plane z staged; plane z - 1 read by every warp
        const longlong2 Xp = fixed(next);
        if(z + 1 < z0 + zc) {
            stage(z + 1, Xp, hnext);
            next = pair(z + 2);
            if(z + 2 < z0 + zc) hnext = halo(z + 2);
        }
        long long sa, sb;
        bfp_xy_sums<BPITCH>(ring[z & 1], t.own, Xc.x, Xc.y, sa, sb);
        const longlong2 M = make_longlong2(bfp_mu(Xc.x, sa + (Xm.x + Xp.x), sc), bfp_mu(Xc.y, sb + (Xm.y + Xp.y), sc));
        const unsigned gi = t.gown + plane(z);
        if(CHGB_BC(15, gi + 1, g.bins)) *reinterpret_cast<longlong2 *>(mu + gi) = M;
        Xm = Xc;
        Xc = Xp;
    }
}

__global__ void __launch_bounds__(256, 5) update_bfp_kernel(const double *__restrict__ psi_in,
                                                            const long long *__restrict__ mu, double *__restrict__ out,
                                                            Geom g, EulerConsts c, BfpState *st, int parity, int zc) {
    __shared__ __align__(16) long long ring[2][BPLANE];
    __shared__ unsigned long long s_gen;
    __shared__ int s_lmu, s_mode;
    const int tid = threadIdx.x;
    pdl_begin();
    if(tid == 0) {   // one load per CTA of the step's state, shared
        s_gen = *(const volatile unsigned long long *) &st->gen;
        s_lmu = *(const volatile int *) &st->lmu;
        s_mode = *(const volatile int *) &st->mode;
    }
    __syncthreads();
    const BfpTile t = bfp_tile(g, tid);
    const int z0 = blockIdx.z * zc;
    int mag = 0;
    if(s_mode) {
        const double c1 = c.c1 * __hiloint2double((1023 + s_lmu) << 20, 0);   // exact: |c1| is in [2^-100, 2^100] or 0
        auto plane = [&](int z) { return (unsigned) (z & g.mask) << (2 * g.log2N); };
        auto pair = [&](int z) {
            const unsigned gi = plane(z) + t.gown;
            return CHGB_BC(11, gi + 1, g.bins) ? *reinterpret_cast<const longlong2 *>(mu + gi) : make_longlong2(0, 0);
        };
        auto halo = [&](int z) {
            return t.has_halo && CHGB_BC(12, plane(z) + t.ghalo, g.bins) ? mu[plane(z) + t.ghalo] : 0ll;
        };
        auto stage = [&](int z, longlong2 X, long long h) {
            long long *p = ring[z & 1];
            if(CHGB_BC(16, t.own + 1, BPLANE)) *reinterpret_cast<longlong2 *>(p + t.own) = X;
            if(t.has_halo && CHGB_BC(16, t.halo, BPLANE)) p[t.halo] = h;
        };
        longlong2 Mm = pair(z0 - 1), Mc = pair(z0);
        stage(z0, Mc, halo(z0));
        longlong2 next = pair(z0 + 1);
        long long hnext = zc > 1 ? halo(z0 + 1) : 0;
        for(int z = z0; z < z0 + zc; z++) {
            const unsigned gi = t.gown + plane(z);
            const bool ok = CHGB_BC(17, gi + 1, g.bins);
            const double2 psi = ok ? *reinterpret_cast<const double2 *>(psi_in + gi) : make_double2(0.0, 0.0);
            __syncthreads();
            const longlong2 Mp = next;
            if(z + 1 < z0 + zc) {
                stage(z + 1, Mp, hnext);
                next = pair(z + 2);
                if(z + 2 < z0 + zc) hnext = halo(z + 2);
            }
            long long sa, sb;
            bfp_xy_sums<BPITCH>(ring[z & 1], t.own, Mc.x, Mc.y, sa, sb);
            sa += (Mm.x + Mp.x) - 6 * Mc.x;
            sb += (Mm.y + Mp.y) - 6 * Mc.y;
            const double2 res = make_double2(fma(c1, bfp_double_fp(sa), psi.x), fma(c1, bfp_double_int(sb), psi.y));
            if(ok) *reinterpret_cast<double2 *>(out + gi) = res;
            mag = max(mag, max(__double2hiint(res.x) & 0x7FFFFFFF, __double2hiint(res.y) & 0x7FFFFFFF));
            Mm = Mc;
            Mc = Mp;
        }
    }
    else {
        mag = bfp_slow_block<3>(psi_in, out, g.mask, g.log2N, c.c1, c.c2[0], c.lshift[2], blockIdx.x * BTX,
                                blockIdx.y * BTY, z0, BTX, BTY, zc);
    }
    bfp_fold_key<8>(mag, s_gen, st->key[parity ^ 1], blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z), tid);
}

// 3D: one kernel per step.  A CTA owns a 32 x 16 tile and marches it through
// `zc` planes: at plane z it stages X of plane z + 2, forms M of plane z + 1 on
// the tile and a halo of 1, and updates plane z.  Each of 360 threads has one
// pair of cells adjacent in x of the tile with a halo of 2 (18 pairs by 20
// rows): its column of three X, and of three M, stays in registers, two planes
// of X and two of M in shared memory serve the x and y neighbours, and there
// is one barrier a plane.  All 360 convert their X, the first 324 form M, the
// first 256 -- the tile -- update.  mu in integers made this the faster form: the
// halo's M costs 1.27 x 27 integer instructions where it used to cost FP64
// ones, and the step saves M's round trip through HBM (16 B a cell) and a
// launch.  N = 256 on GB300, us a step: the pair with FP64 in mu 172, the pair
// above 144, this kernel 116 (integer ALU 46 %, FP64 pipe 46 %, issue slots 59 %
// busy; the barrier a plane and the shared loads are the larger stalls).
constexpr int B3X = 32, B3Y = 16, B3P = B3X + 4, B3H = B3P / 2;   // tile, cells and pairs of a staged row
constexpr int B3THREADS = 384, B3CTAS = 3;   // CTAs per SM: 56 registers a thread
constexpr int B3OWN = B3X / 2 * B3Y, B3M = B3H * (B3Y + 2), B3ALL = B3H * (B3Y + 4);

__global__ void __launch_bounds__(B3THREADS, B3CTAS) euler3d_bfp_kernel(const double *__restrict__ in,
                                                                       double *__restrict__ out, Geom g, EulerConsts c,
                                                                       BfpConsts b, BfpState *st, int parity, int zc) {
    __shared__ __align__(16) long long sx[2][B3P * (B3Y + 4)], sm[2][B3P * (B3Y + 2)];
    const int tid = threadIdx.x;
    const int x0 = blockIdx.x * B3X, y0 = blockIdx.y * B3Y, z0 = blockIdx.z * zc;
    const int z1 = min(z0 + zc, g.N);
    pdl_begin();
    const unsigned long long key = bfp_read_key(st->key[parity], tid);
    const BfpScale sc = bfp_scale<3>((int) (key & 0xFFFFu), c, b);
    int mag = 0;
    if(sc.fast) {
        int px, row;   // this thread's pair and row of the staged region
        if(tid < B3OWN) {
            px = 1 + tid % (B3X / 2);
            row = 2 + tid / (B3X / 2);
        }
        else if(tid < B3OWN + 2 * B3H) {
            const int k = tid - B3OWN;
            px = k % B3H;
            row = k < B3H ? 1 : B3Y + 2;
        }
        else if(tid < B3M) {
            const int k = tid - (B3OWN + 2 * B3H);
            px = k < B3Y ? 0 : B3H - 1;
            row = 2 + k % B3Y;
        }
        else {
            const int k = tid - B3M;
            px = k % B3H;
            row = k < B3H ? 0 : B3Y + 3;
        }
        const bool has = tid < B3ALL;
        const int ix = row * B3P + 2 * px, im = ix - B3P;
        const unsigned off = ((x0 - 2 + 2 * px) & g.mask) + ((unsigned) ((y0 - 2 + row) & g.mask) << g.log2N);
        auto load = [&](int z) {
            const unsigned gi = off + ((unsigned) (z & g.mask) << (2 * g.log2N));   // below 2^30
            return has && CHGB_BC(11, gi + 1, g.bins) ? *reinterpret_cast<const double2 *>(in + gi) : make_double2(0.0, 0.0);
        };
        auto fixed = [&](double2 v) { return make_longlong2(bfp_fixed(v.x, sc.emax), bfp_fixed(v.y, sc.emax)); };
        auto stage = [&](int z, longlong2 X) {
            if(has && CHGB_BC(13, ix + 1, B3P * (B3Y + 4))) *reinterpret_cast<longlong2 *>(sx[z & 1] + ix) = X;
        };
        const double c1 = c.c1 * __hiloint2double((1023 + sc.lmu) << 20, 0);   // exact: |c1| is in [2^-100, 2^100] or 0
        longlong2 Xa = fixed(load(z0 - 2)), Xb = fixed(load(z0 - 1));
        stage(z0 - 1, Xb);
        longlong2 Ma = make_longlong2(0, 0), Mb = Ma;
        double2 next = load(z0), psi = make_double2(0.0, 0.0);
#pragma unroll 3   // the columns' three planes turn without moves
        for(int z = z0 - 2; z < z1; z++) {
            __syncthreads();   // plane z + 1 of X and plane z of M staged; the planes before them read by every warp
            const longlong2 Xc = fixed(next);
            stage(z + 2, Xc);
            if(z + 1 < z1) next = load(z + 3);
            if(z >= z0 && tid < B3OWN) psi = load(z);   // in L2 (and L1): fetched three planes ago
            longlong2 Mc = Ma;
            if(tid < B3M && CHGB_BC(14, ix - B3P, B3P * (B3Y + 4)) && CHGB_BC(14, ix + B3P + 1, B3P * (B3Y + 4))) {
                long long sa, sb;
                bfp_xy_sums<B3P>(sx[(z + 1) & 1], ix, Xb.x, Xb.y, sa, sb);
                Mc = make_longlong2(bfp_mu(Xb.x, sa + (Xa.x + Xc.x), sc), bfp_mu(Xb.y, sb + (Xa.y + Xc.y), sc));
                *reinterpret_cast<longlong2 *>(sm[(z + 1) & 1] + im) = Mc;
            }
            if(z >= z0 && tid < B3OWN) {
                const unsigned gi = off + ((unsigned) z << (2 * g.log2N));
                long long sa, sb;
                bfp_xy_sums<B3P>(sm[z & 1], im, Mb.x, Mb.y, sa, sb);
                sa += (Ma.x + Mc.x) - 6 * Mb.x;
                sb += (Ma.y + Mc.y) - 6 * Mb.y;
                const double2 res = make_double2(fma(c1, bfp_double_fp(sa), psi.x), fma(c1, bfp_double_fp(sb), psi.y));
                if(CHGB_BC(15, gi + 1, g.bins)) *reinterpret_cast<double2 *>(out + gi) = res;
                mag = max(mag, max(__double2hiint(res.x) & 0x7FFFFFFF, __double2hiint(res.y) & 0x7FFFFFFF));
            }
            Xa = Xb;
            Xb = Xc;
            Ma = Mb;
            Mb = Mc;
        }
    }
    else {
        mag = bfp_slow_block<3>(in, out, g.mask, g.log2N, c.c1, c.c2[0], c.lshift[2], x0, y0, z0, B3X, B3Y, z1 - z0);
    }
    bfp_fold_key<B3THREADS / 32>(mag, (key >> 16) + 1, st->key[parity ^ 1],
                                 blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z), tid);
}

// The key of the field psi (n values, n even): (gen << 16) | its largest biased exponent.
__global__ void __launch_bounds__(256) bfp_refresh_kernel(const double2 *__restrict__ psi, long long n2,
                                                          unsigned long long *bank, unsigned long long gen) {
    int mag = 0;
    for(long long i = (long long) blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += (long long) gridDim.x * blockDim.x) {
        const double2 v = psi[i];
        mag = max(mag, max(__double2hiint(v.x) & 0x7FFFFFFF, __double2hiint(v.y) & 0x7FFFFFFF));
    }
    bfp_fold_key<8>(mag, gen, bank, blockIdx.x, threadIdx.x);
}

// 2D: one kernel per step.  A CTA stages X of a TX x TY tile of psi with a halo
// of 2, forms M on the tile plus a halo of 1, then updates the tile, everywhere
// two cells adjacent in x at a time.  The halo's M is formed by each CTA that
// needs it from the same X, so every CTA sees the same integers; there is one
// launch per step and no M round trip through memory.  The key is read from
// bank `parity` and the step's exponents fold into the other bank (CTAs of one
// launch both read and fold).
template <int TX, int TY>
__global__ void __launch_bounds__(256, 4) euler2d_bfp_kernel(const double *__restrict__ in, double *__restrict__ out,
                                                             Geom g, EulerConsts c, BfpConsts b, BfpState *st,
                                                             int parity) {
    constexpr int P = TX + 4, H = P / 2;                // cells and pairs of a staged row
    constexpr int NX = H * (TY + 4), NM = H * (TY + 2), NU = TX / 2 * TY;
    // M is formed on whole pairs: the outermost cell of each row's ends reads
    // into the neighbouring row and is not used
    __shared__ __align__(16) long long sx[2 * NX], sm[2 * NM];
    const int tid = threadIdx.x;
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
    pdl_begin();
    const unsigned long long key = bfp_read_key(st->key[parity], tid);
    const BfpScale sc = bfp_scale<2>((int) (key & 0xFFFFu), c, b);
    int mag = 0;
    if(sc.fast) {
#pragma unroll
        for(int k = 0; k < (NX + 255) / 256; k++) {
            const int i = tid + 256 * k;
            if(i < NX) {
                const int y = i / H, x = 2 * (i - y * H);
                const unsigned gi = ((x0 - 2 + x) & g.mask) + ((unsigned) ((y0 - 2 + y) & g.mask) << g.log2N);
                const double2 v = CHGB_BC(21, gi + 1, g.bins) ? *reinterpret_cast<const double2 *>(in + gi)
                                                              : make_double2(0.0, 0.0);
                *reinterpret_cast<longlong2 *>(sx + 2 * i) = make_longlong2(bfp_fixed(v.x, sc.emax), bfp_fixed(v.y, sc.emax));
            }
        }
        __syncthreads();
#pragma unroll
        for(int k = 0; k < (NM + 255) / 256; k++) {
            const int i = tid + 256 * k;
            if(i < NM && CHGB_BC(22, 2 * i + 2 * P + 1, 2 * NX)) {
                const longlong2 X = *reinterpret_cast<const longlong2 *>(sx + 2 * i + P);
                long long sa, sb;
                bfp_xy_sums<P>(sx, 2 * i + P, X.x, X.y, sa, sb);
                *reinterpret_cast<longlong2 *>(sm + 2 * i) = make_longlong2(bfp_mu(X.x, sa, sc), bfp_mu(X.y, sb, sc));
            }
        }
        __syncthreads();
        const double c1 = c.c1 * __hiloint2double((1023 + sc.lmu) << 20, 0);   // exact: |c1| is in [2^-100, 2^100] or 0
#pragma unroll
        for(int k = 0; k < NU / 256; k++) {
            const int i = tid + 256 * k;
            const int y = i / (TX / 2), x = 2 * (i % (TX / 2));
            const int m = (y + 1) * P + x + 2;
            const unsigned gi = (unsigned) (x0 + x) + ((unsigned) (y0 + y) << g.log2N);
            if(!CHGB_BC(23, m - P, 2 * NM) || !CHGB_BC(23, m + P + 1, 2 * NM) || !CHGB_BC(24, gi + 1, g.bins)) continue;
            const double2 psi = *reinterpret_cast<const double2 *>(in + gi);
            const longlong2 M = *reinterpret_cast<const longlong2 *>(sm + m);
            long long sa, sb;
            bfp_xy_sums<P>(sm, m, M.x, M.y, sa, sb);
            const double2 res = make_double2(fma(c1, bfp_double_fp(sa - 4 * M.x), psi.x),
                                             fma(c1, bfp_double_int(sb - 4 * M.y), psi.y));
            *reinterpret_cast<double2 *>(out + gi) = res;
            mag = max(mag, max(__double2hiint(res.x) & 0x7FFFFFFF, __double2hiint(res.y) & 0x7FFFFFFF));
        }
    }
    else {
        mag = bfp_slow_block<2>(in, out, g.mask, g.log2N, c.c1, c.c2[0], c.lshift[1], x0, y0, 0, TX, TY, 1);
    }
    bfp_fold_key<8>(mag, (key >> 16) + 1, st->key[parity ^ 1], blockIdx.x + gridDim.x * blockIdx.y, tid);
}

}  // namespace chgb

extern "C" int chgb_bounds_report(unsigned long long *first) {
    if(!first) return CHGB_ERR_INVALID;
#ifdef CHGB_BOUNDS_CHECK
    // the explicit kernels' record (this file), then the transforms' (spectral.cu)
    unsigned long long a = 0, b = 0;
    if(chgb::bc_read_tu(&a) != cudaSuccess || chgb::bc_read_spectral(&b) != cudaSuccess) return CHGB_ERR_CUDA;
    *first = a ? a : b;
    return CHGB_OK;
#else
    *first = 0;
    chgb::record_error("chgb_bounds_report: not a bounds-check build (-DCHGB_BOUNDS_CHECK, lib/libchgb_bc.so)");
    return CHGB_ERR_UNSUPPORTED;
#endif
}

namespace chgb {

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
namespace {

template <int KIND, int MOB>
cudaError_t launch_1d(const Geom &g, const ModelDev &m, const EulerConsts &c, const double *in, double *out,
                      cudaStream_t st, bool configure) {
    if(configure) return cudaSuccess;
    if(g.N >= 256) {
        euler1d_kernel<KIND, MOB, 256><<<g.N / 256, 256, 0, st>>>(in, out, g, m, c);
    }
    else if(g.N >= 64) {
        euler1d_kernel<KIND, MOB, 64><<<g.N / 64, 64, 0, st>>>(in, out, g, m, c);
    }
    else if(g.N >= 16) {
        euler1d_kernel<KIND, MOB, 16><<<g.N / 16, 32, 0, st>>>(in, out, g, m, c);
    }
    else {
        euler1d_kernel<KIND, MOB, 4><<<g.N / 4, 32, 0, st>>>(in, out, g, m, c);
    }
    return cudaGetLastError();
}

template <int KIND, int MOB, int TX, int TY>
cudaError_t launch_2d_tile(const Geom &g, const ModelDev &m, const EulerConsts &c, const double *in, double *out,
                           cudaStream_t st, bool configure) {
    constexpr int S = NSpecies<KIND>::value;
    size_t smem = sizeof(double) * S * ((TX + 4) * (TY + 4) + (MOB ? 2 : 1) * (TX + 2) * (TY + 2));
    auto kern = euler2d_kernel<KIND, MOB, TX, TY>;
    if(configure) {
        return smem > 48 * 1024 ? cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem)
                                : cudaSuccess;
    }
    dim3 grid(g.N / TX, g.N / TY);
    kern<<<grid, dim3(32, 8), smem, st>>>(in, out, g, m, c);
    return cudaGetLastError();
}

template <int KIND, int MOB>
cudaError_t launch_2d(const Geom &g, const ModelDev &m, const EulerConsts &c, const double *in, double *out,
                      cudaStream_t st, bool configure) {
    // the largest tile that still gives >= 1024 CTAs (about 7 per SM): halo
    // recomputation favours big tiles, filling 152 SMs favours many (N=256:
    // 16x16 tiles run a step in 4.1 us, 32x32 tiles -- 64 CTAs -- in 6.4 us)
    const long long cells = (long long) g.N * g.N;
    if(g.N >= 32 && cells / (32 * 32) >= 1024) return launch_2d_tile<KIND, MOB, 32, 32>(g, m, c, in, out, st, configure);
    if(g.N >= 32 && cells / (32 * 16) >= 1024) return launch_2d_tile<KIND, MOB, 32, 16>(g, m, c, in, out, st, configure);
    if(g.N >= 16) return launch_2d_tile<KIND, MOB, 16, 16>(g, m, c, in, out, st, configure);
    if(g.N >= 8) return launch_2d_tile<KIND, MOB, 8, 8>(g, m, c, in, out, st, configure);
    return launch_2d_tile<KIND, MOB, 4, 4>(g, m, c, in, out, st, configure);
}

template <int KIND, int MOB, int TX, int TY>
cudaError_t launch_3d_tile(const Geom &g, const ModelDev &m, const EulerConsts &c, const double *in, double *out,
                           cudaStream_t st, bool configure) {
    constexpr int S = NSpecies<KIND>::value;
    size_t smem = sizeof(double) * S * (5 * (TX + 4) * (TY + 4) + (MOB ? 6 : 3) * (TX + 2) * (TY + 2));
    auto kern = euler3d_kernel<KIND, MOB, TX, TY>;
    if(configure) {
        return smem > 48 * 1024 ? cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem)
                                : cudaSuccess;
    }
    int zc = g.N < 32 ? g.N : 32;
    dim3 grid(g.N / TX, g.N / TY, g.N / zc);
    kern<<<grid, dim3(32, 8), smem, st>>>(in, out, g, m, c, zc);
    return cudaGetLastError();
}

template <int KIND, int MOB>
cudaError_t launch_3d(const Geom &g, const ModelDev &m, const EulerConsts &c, const double *in, double *out,
                      cudaStream_t st, bool configure) {
    if(g.N >= 32) return launch_3d_tile<KIND, MOB, 32, 16>(g, m, c, in, out, st, configure);
    if(g.N >= 16) return launch_3d_tile<KIND, MOB, 16, 16>(g, m, c, in, out, st, configure);
    if(g.N >= 8) return launch_3d_tile<KIND, MOB, 8, 8>(g, m, c, in, out, st, configure);
    return launch_3d_tile<KIND, MOB, 4, 4>(g, m, c, in, out, st, configure);
}

template <int KIND, int MOB>
cudaError_t launch_dims(const Geom &g, const ModelDev &m, const EulerConsts &c, const double *in, double *out,
                        cudaStream_t st, bool configure) {
    switch(g.dims) {
        case 1: return launch_1d<KIND, MOB>(g, m, c, in, out, st, configure);
        case 2: return launch_2d<KIND, MOB>(g, m, c, in, out, st, configure);
        default: return launch_3d<KIND, MOB>(g, m, c, in, out, st, configure);
    }
}

template <int KIND>
cudaError_t launch_mob(int mob, const Geom &g, const ModelDev &m, const EulerConsts &c, const double *in,
                       double *out, cudaStream_t st, bool configure) {
    // mob: 0 = plain euler, 1 = euler_mobility with constant M, 2 = free-energy M
    if(mob == 0) return launch_dims<KIND, 0>(g, m, c, in, out, st, configure);
    if(mob == 1) return launch_dims<KIND, 1>(g, m, c, in, out, st, configure);
    if(mob == 3) return launch_dims<KIND, 3>(g, m, c, in, out, st, configure);
    if constexpr(KIND == CHGB_MODEL_SIMPLE_WERTHEIM) return launch_dims<KIND, 2>(g, m, c, in, out, st, configure);
    return cudaErrorInvalidValue;
}

}  // namespace

namespace {

constexpr int SPLIT_CTAS = 2 * 152;

template <int KIND, int MOB, int DIMS>
cudaError_t launch_split_kind(const Geom &g, const ModelDev &m, const EulerConsts &c, const double *in, double *out,
                              double *mu, double *mob, cudaStream_t st, unsigned *key,
                              int parity) {
    constexpr int S = NSpecies<KIND>::value;
    // 8-plane z-chunks: the extra halo planes per chunk are cheap L2 loads,
    // and the many small CTAs keep every SM's FP64 pipe fed to the end of the
    // launch (N=256: 8192 CTAs, 7% faster than 32-plane chunks on GB300); fewer
    // planes where those would not give every SM two CTAs (N <= 64)
    int zc = (DIMS == 3) ? 8 : 1;
    while(zc > 1 && (g.N / STX) * (g.N / STY) * (g.N / zc) < SPLIT_CTAS) zc /= 2;
    dim3 grid(g.N / STX, g.N / STY, (DIMS == 3) ? g.N / zc : 1);
    dim3 block(STX, STY);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, mu_kernel<KIND, MOB, DIMS>, in, mu, mob, g, m, c, zc, key);
    if(e != cudaSuccess) return e;
    if constexpr(S == 1 && (MOB == 1 || MOB == 2))
        if(key) {
            // z chunks of 16 planes where that gives 1,000 CTAs (two and a half on each
            // SM at a time), of four below, fewer yet for every SM to have two.  3D N=128:
            // 4 planes 78.4 us a step, 8 planes 86.9, 2 planes 79.2; N=256: 16 538, 32 553
            const int tiles = (g.N / MTX) * (g.N / MTY);
            int uz = DIMS == 2 ? 1 : tiles * (g.N / 16) >= 1000 ? 16 : 4;
            while(uz > 1 && tiles * (g.N / uz) < SPLIT_CTAS) uz /= 2;
            cfg.gridDim = dim3(g.N / MTX, g.N / MTY, DIMS == 3 ? g.N / uz : 1);
            cfg.blockDim = dim3(MTHR);
            constexpr bool CONST = MOB == 1, DENSITY = KIND == CHGB_MODEL_SIMPLE_WERTHEIM;
            auto kernel = tiles * (g.N / uz) >= 5 * 152 ? update_mob_fx_kernel<DIMS, CONST, DENSITY, DIMS == 2 ? 8 : 5>
                                                        : update_mob_fx_kernel<DIMS, CONST, DENSITY, DIMS == 2 ? 8 : 1>;
            return cudaLaunchKernelEx(&cfg, kernel, in, (const double *) mu,
                                      (const double *) mob, out, g, c, uz, key - 2 * parity, parity);
        }
    return cudaLaunchKernelEx(&cfg, update_kernel<S, MOB, DIMS>, in, (const double *) mu, (const double *) mob, out, g,
                              c, zc);
}

template <int KIND, int MOB>
cudaError_t launch_split_mob(const Geom &g, const ModelDev &m, const EulerConsts &c, const double *in, double *out,
                             double *mu, double *mob, cudaStream_t st, unsigned *key,
                              int parity) {
    if(g.dims == 2) return launch_split_kind<KIND, MOB, 2>(g, m, c, in, out, mu, mob, st, key, parity);
    return launch_split_kind<KIND, MOB, 3>(g, m, c, in, out, mu, mob, st, key, parity);
}

template <int KIND>
cudaError_t launch_split_model(int mob_kind, const Geom &g, const ModelDev &m, const EulerConsts &c,
                               const double *in, double *out, double *mu, double *mob, cudaStream_t st, unsigned *key,
                              int parity) {
    if(mob_kind == 0) return launch_split_mob<KIND, 0>(g, m, c, in, out, mu, mob, st, key, parity);
    if(mob_kind == 1) return launch_split_mob<KIND, 1>(g, m, c, in, out, mu, mob, st, key, parity);
    // kind 3 reads the given field; mu_kernel writes `mob` only for kind 2
    if(mob_kind == 3) return launch_split_mob<KIND, 3>(g, m, c, in, out, mu, const_cast<double *>(c.mobf), st, key, parity);
    if constexpr(KIND == CHGB_MODEL_SIMPLE_WERTHEIM) return launch_split_mob<KIND, 2>(g, m, c, in, out, mu, mob, st, key, parity);
    return cudaErrorInvalidValue;
}

}  // namespace

bool euler_split_supported(const Geom &g) { return g.dims >= 2 && g.N >= 32; }

// Two steps per launch: plain `euler` in 2D boxes of 32 <= N <= 512, 16 x 16 tiles.
bool euler_two_supported(int integrator, const Geom &g) {
    return integrator == CHGB_INTEGRATOR_EULER && g.dims == 2 && g.N >= 32 && g.N <= 512;
}

namespace {
template <int KIND>
cudaError_t launch_two_kind(const Geom &g, const ModelDev &m, const EulerConsts &c, const double *in, double *out,
                            double *mid, cudaStream_t st, bool configure) {
    constexpr int S = NSpecies<KIND>::value, T = 16;
    const size_t smem = sizeof(double) * S * ((T + 8) * (T + 8) + (T + 6) * (T + 6) + (T + 4) * (T + 4) +
                                              (T + 2) * (T + 2));
    auto kern = euler2d_two_kernel<KIND, T, T>;
    if(configure) {
        return smem > 48 * 1024 ? cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem)
                                : cudaSuccess;
    }
    kern<<<dim3(g.N / T, g.N / T), dim3(32, 8), smem, st>>>(in, out, mid, g, m, c);
    return cudaGetLastError();
}
}  // namespace

cudaError_t launch_euler_two(const Geom &g, const ModelDev &m, const EulerConsts &c, const double *in, double *out,
                             cudaStream_t st, bool configure, double *mid) {
    switch(m.kind) {
        case CHGB_MODEL_LANDAU: return launch_two_kind<CHGB_MODEL_LANDAU>(g, m, c, in, out, mid, st, configure);
        case CHGB_MODEL_SIMPLE_WERTHEIM:
            return launch_two_kind<CHGB_MODEL_SIMPLE_WERTHEIM>(g, m, c, in, out, mid, st, configure);
        default: return launch_two_kind<CHGB_MODEL_SALEH>(g, m, c, in, out, mid, st, configure);
    }
}

bool euler_cluster_supported(int integrator, const Geom &g) {
    return integrator == CHGB_INTEGRATOR_EULER && g.dims == 2 && (g.N == 32 || g.N == 64);
}

namespace {
template <int KIND, int T>
cudaError_t launch_cluster_kind(const Geom &g, const ModelDev &m, const EulerConsts &c, const double *in,
                                double *out, int nsteps, cudaStream_t st, bool configure) {
    // at least four warps, one per SM sub-partition: each has its own FP64 unit
    constexpr int NTHR = T * T < 128 ? 128 : T * T;
    auto kern = euler2d_cluster_kernel<KIND, T, NTHR>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CLUSTER_TILES, CLUSTER_TILES, 1);
    cfg.blockDim = dim3(NTHR, 1, 1);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CLUSTER_TILES;
    attr[0].val.clusterDim.y = CLUSTER_TILES;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if(configure) {
        // 16 CTAs is above the portable cluster size of 8: opt in, then ask
        // whether the GPU can hold such a cluster at all
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if(e != cudaSuccess) return e;
        int clusters = 0;
        e = cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg);
        if(e != cudaSuccess) return e;
        return clusters > 0 ? cudaSuccess : cudaErrorInvalidConfiguration;
    }
    if(nsteps < 1) return cudaErrorInvalidValue;
    return cudaLaunchKernelEx(&cfg, kern, in, out, g, m, c, nsteps);
}

template <int KIND>
cudaError_t launch_cluster_tile(const Geom &g, const ModelDev &m, const EulerConsts &c, const double *in, double *out,
                                int nsteps, cudaStream_t st, bool configure) {
    if(g.N == 64) return launch_cluster_kind<KIND, 16>(g, m, c, in, out, nsteps, st, configure);
    if(g.N == 32) return launch_cluster_kind<KIND, 8>(g, m, c, in, out, nsteps, st, configure);
    return cudaErrorInvalidValue;
}
}  // namespace

cudaError_t launch_euler_cluster(const Geom &g, const ModelDev &m, const EulerConsts &c, const double *in,
                                 double *out, int nsteps, cudaStream_t st, bool configure) {
    switch(m.kind) {
        case CHGB_MODEL_LANDAU: return launch_cluster_tile<CHGB_MODEL_LANDAU>(g, m, c, in, out, nsteps, st, configure);
        case CHGB_MODEL_SIMPLE_WERTHEIM:
            return launch_cluster_tile<CHGB_MODEL_SIMPLE_WERTHEIM>(g, m, c, in, out, nsteps, st, configure);
        default: return launch_cluster_tile<CHGB_MODEL_SALEH>(g, m, c, in, out, nsteps, st, configure);
    }
}

namespace {
template <int KIND, int TX, int TY>
cudaError_t launch_batch_tile(const EulerBatchRep *reps, const int2 *items, int nitems, int parity, bool configure,
                              cudaStream_t st) {
    constexpr int S = NSpecies<KIND>::value;
    size_t smem = sizeof(double) * S * ((TX + 4) * (TY + 4) + (TX + 2) * (TY + 2));
    auto kern = euler2d_batch_kernel<KIND, TX, TY>;
    if(configure) {
        return smem > 48 * 1024 ? cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem)
                                : cudaSuccess;
    }
    if(nitems == 0) return cudaSuccess;
    kern<<<nitems, dim3(32, TX * TY >= 1024 ? 8 : 4), smem, st>>>(reps, items, parity);
    return cudaGetLastError();
}

template <int KIND>
cudaError_t launch_batch_kind(int tile, const EulerBatchRep *reps, const int2 *items, int nitems, int parity,
                              bool configure, cudaStream_t st) {
    switch(tile) {
        case 32: return launch_batch_tile<KIND, 32, 32>(reps, items, nitems, parity, configure, st);
        case 16: return launch_batch_tile<KIND, 16, 16>(reps, items, nitems, parity, configure, st);
        default: return launch_batch_tile<KIND, 64, 16>(reps, items, nitems, parity, configure, st);
    }
}
}  // namespace

cudaError_t launch_euler2d_batch(int kind, int tile, const EulerBatchRep *reps, const int2 *items, int nitems,
                                 int parity, bool configure, cudaStream_t st) {
    switch(kind) {
        case CHGB_MODEL_LANDAU:
            return launch_batch_kind<CHGB_MODEL_LANDAU>(tile, reps, items, nitems, parity, configure, st);
        case CHGB_MODEL_SIMPLE_WERTHEIM:
            return launch_batch_kind<CHGB_MODEL_SIMPLE_WERTHEIM>(tile, reps, items, nitems, parity, configure, st);
        default: return launch_batch_kind<CHGB_MODEL_SALEH>(tile, reps, items, nitems, parity, configure, st);
    }
}

bool euler_bfp_supported(int integrator, int model_kind, const Geom &g) {
    return integrator == CHGB_INTEGRATOR_EULER && model_kind == CHGB_MODEL_LANDAU && g.dims >= 2 && g.N >= 32;
}

// c2's mantissa and exponent, and elin, for the mu kernel of a DIMS-dimensional box.
static BfpConsts bfp_consts(const EulerConsts &c, int dims) {
    BfpConsts b;
    const double c2 = c.c2[0];
    unsigned long long u;
    std::memcpy(&u, &c2, sizeof u);
    const int e = (int) (u >> 52) & 0x7FF;
    const long long mag = (long long) ((u & 0xFFFFFFFFFFFFFull) | (e ? 1ull << 52 : 0ull));
    b.mc = (long long) ((u >> 63) ? -mag : mag) * 1024;   // |mc| < 2^63
    b.ec = e ? e : 1;
    const double lin = std::fabs(c.lshift[dims - 1]) + 2.0 * dims * std::fabs(c2);
    b.elin = lin > 0.0 && std::isfinite(lin) ? std::ilogb(lin) + 1 : -4000;   // lin < 2^elin
    // constants the integer step does not take (not finite, or so far from one
    // that its scales would leave the exponent range) put every step in mode 0
    const double a1 = std::fabs(c.c1);
    const bool c1_ok = a1 == 0.0 || (a1 >= std::ldexp(1.0, -100) && a1 <= std::ldexp(1.0, 100));
    if(!std::isfinite(lin) || (lin > 0.0 && b.elin < -800) || !c1_ok) b.elin = 100000;
    return b;
}

// Planes a CTA of the 3D step marches through: the chunk with the fewest plane
// iterations (two of each chunk are its halo's) over the waves of CTAs that the
// GPU holds.  Cell-steps/s on GB300: N = 256 37 planes (2 waves) 1.44e11, 32
// (2.2 waves) 1.36e11, 16 1.25e11; N = 128 10 planes 1.03e11, 8 9.2e10, 16
// 7.2e10; N = 512 64 planes 1.58e11, 32 1.52e11, 16 1.44e11.  N = 64, whose CTAs
// never fill a wave, 4 planes 4.3e10, 2 3.2e10.
static int bfp_zchunk(const Geom &g) {
    if(g.N <= 64) return 4;
    const long long tiles = (long long) (g.N / B3X) * (g.N / B3Y), slots = 152 * B3CTAS;
    long long best = 0;
    int pick = 8;
    for(int zc = 8; zc <= 64; zc++) {
        const long long ctas = tiles * ((g.N + zc - 1) / zc), cost = (ctas + slots - 1) / slots * (zc + 2);
        if(best == 0 || cost < best) {
            best = cost;
            pick = zc;
        }
    }
    return pick;
}

cudaError_t launch_euler_bfp(const Geom &g, const EulerConsts &c, const double *in, double *out, double *mu,
                             BfpState *st, int parity, cudaStream_t stream) {
    const BfpConsts b = bfp_consts(c, g.dims);
    const int pair_zc = g.N <= 64 ? 2 : g.N == 128 ? 4 : g.N == 256 ? 16 : 32;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e;
    if(g.dims == 2) {
        auto tile = [&](auto kernel, int tx, int ty) {
            cfg.gridDim = dim3(g.N / tx, g.N / ty);
            return cudaLaunchKernelEx(&cfg, kernel, in, out, g, c, b, st, parity);
        };
        // the largest tile that leaves every SM a CTA (halo work against
        // CTAs).  Cell-steps/s on GB300 with 64 x 32, 32 x 32 and 64 x 16 tiles:
        // N = 512 6.3e10 each, N = 1024 1.26, 1.18, 1.19e11; with 64 x 32
        // and 64 x 16, N = 2048 1.78, 1.45e11, N = 4096 1.91, 1.48e11
        if(g.N >= 1024) e = tile(euler2d_bfp_kernel<64, 32>, 64, 32);
        else e = tile(euler2d_bfp_kernel<32, 32>, 32, 32);
    }
    else {
        if(mu) {
            cfg.gridDim = dim3(g.N / BTX, g.N / BTY, g.N / pair_zc);
            long long *m = reinterpret_cast<long long *>(mu);
            e = cudaLaunchKernelEx(&cfg, mu_bfp_kernel, in, m, g, c, b, st, parity, pair_zc);
            if(e == cudaSuccess)
                e = cudaLaunchKernelEx(&cfg, update_bfp_kernel, in, (const long long *) m, out, g, c, st, parity, pair_zc);
        }
        else {
            const int zc = bfp_zchunk(g);
            cfg.gridDim = dim3(g.N / B3X, g.N / B3Y, (g.N + zc - 1) / zc);
            cfg.blockDim = dim3(B3THREADS);
            e = cudaLaunchKernelEx(&cfg, euler3d_bfp_kernel, in, out, g, c, b, st, parity, zc);
        }
    }
    return e;
}

cudaError_t launch_bfp_refresh(const double *psi, long long n, BfpState *st, int parity, unsigned long long gen,
                               cudaStream_t stream) {
    const long long n2 = n / 2;
    const long long blocks = std::min<long long>((n2 + 255) / 256, 152 * 8);
    bfp_refresh_kernel<<<(unsigned) blocks, 256, 0, stream>>>(reinterpret_cast<const double2 *>(psi), n2, st->key[parity], gen);
    return cudaGetLastError();
}

cudaError_t launch_euler_split(int integrator, const Geom &g, const ModelDev &m, const EulerConsts &c,
                               const double *in, double *out, double *mu, double *mob, cudaStream_t st, unsigned *key,
                               int parity) {
    if(key) key += 2 * parity;   // the entries mu_kernel folds into
    int mob_kind = 0;
    if(integrator == CHGB_INTEGRATOR_EULER_MOBILITY) mob_kind = mobility_kind(c.mobility_type);
    switch(m.kind) {
        case CHGB_MODEL_LANDAU: return launch_split_model<CHGB_MODEL_LANDAU>(mob_kind, g, m, c, in, out, mu, mob, st, key, parity);
        case CHGB_MODEL_SIMPLE_WERTHEIM:
            return launch_split_model<CHGB_MODEL_SIMPLE_WERTHEIM>(mob_kind, g, m, c, in, out, mu, mob, st, key, parity);
        default: return launch_split_model<CHGB_MODEL_SALEH>(mob_kind, g, m, c, in, out, mu, mob, st, key, parity);
    }
}

bool euler_mob_fx_supported(int integrator, int model, int mobility_type, const Geom &g) {
    return integrator == CHGB_INTEGRATOR_EULER_MOBILITY && model != CHGB_MODEL_SALEH && g.dims >= 2 && g.N >= 32 &&
           (mobility_type == CHGB_MOBILITY_CONSTANT ||
            (mobility_type == CHGB_MOBILITY_FREE_ENERGY && model == CHGB_MODEL_SIMPLE_WERTHEIM));
}

cudaError_t launch_euler_step(int integrator, const Geom &g, const ModelDev &m, const EulerConsts &c,
                              const double *in, double *out, cudaStream_t st, bool configure) {
    int mob = 0;
    if(integrator == CHGB_INTEGRATOR_EULER_MOBILITY) mob = mobility_kind(c.mobility_type);
    switch(m.kind) {
        case CHGB_MODEL_LANDAU: return launch_mob<CHGB_MODEL_LANDAU>(mob, g, m, c, in, out, st, configure);
        case CHGB_MODEL_SIMPLE_WERTHEIM: return launch_mob<CHGB_MODEL_SIMPLE_WERTHEIM>(mob, g, m, c, in, out, st, configure);
        default: return launch_mob<CHGB_MODEL_SALEH>(mob, g, m, c, in, out, st, configure);
    }
}

}  // namespace chgb
