// spectral.cu — the `pseudospectral` semi-implicit step, FP64, own FFT.
//
// Reference: src/integrators/PseudospectralCPU.cpp:13-136 (FFTW r2c/c2r,
// per-mode update) and its CUDA mirror src/CUDA/integrators/PseudospectralCUDA.cu
// (single-precision cuFFT for f'; not followed).
//
// State.  The master copy is the half spectrum psi_t = rho_hat / N^dims (axis x
// halved, as FFTW's r2c), along the last transformed axis (spectral_line_index);
// the transforms' work array has the reference's layout
// [species][n0]..[n_{d-2}][N/2+1].  Storing psi_t pre-divided by N^dims makes the inverse
// transform produce rho directly, so the per-mode update of
// PseudospectralCPU.cpp:119-131 folds to
//     psi_t' = alpha * psi_t - beta * F[f'(rho)],
//     alpha = (1 + c S) / denom,  beta = c * dealias / denom / N^dims,
//     c = dt M q^2,  denom = 1 + dt M (S q^2 + 2 k q^4),
// with q^2 and the dealiasing mask tabulated on the host exactly as the
// reference computes them (their 1D/2D/3D formulas differ in rounding and in
// `<` vs `<=` at the cut).
//
// One time step is:
//   ROW  (x, contiguous rows): half spectrum row -> c2r -> rho row -> f'(rho)
//        -> r2c -> half spectrum row, all in shared memory (one kernel);
//   COL  (each slower axis): complex FFT along the axis of column bundles in
//        shared memory; on the slowest axis the forward transform, the per-mode
//        update and the inverse transform run in one kernel.
// 2D: ROW + COL_y(fwd, update, inv).  3D: ROW + COL_y(fwd) + COL_z(fwd, update,
// inv) + COL_y(inv).  1D: ROW + an elementwise update.
// The real r2c/c2r of a row of L = 2M values is a complex FFT of length M on
// the even/odd packing z[n] = x[2n] + i x[2n+1] plus one pre/post-processing
// sweep.  The transforms run in 64-bit block floating point (bfp.cuh): each
// line is converted to fixed point with one exponent, transformed with integer
// arithmetic and converted back; the state, f' and the mode update stay FP64.
// A line's values live in registers, two, four or eight to a thread, from the load
// of the row or column to the store of its transform; they cross between
// threads through shared memory once per radix-2, -4 or -8 pass.
#include <cmath>
#include <vector>

#include "bfp.cuh"
#include "bounds.cuh"
#include "kernels.h"
#include "spectral.h"

namespace chgb {

#ifdef CHGB_BOUNDS_CHECK
cudaError_t bc_read_spectral(unsigned long long *first) { return bc_read_tu(first); }
#endif

namespace {

// ---------------------------------------------------------------------------
// Pseudospectral line transforms, bfp.cuh.
// ---------------------------------------------------------------------------

// The CTA's share of a row pass: `lines` = rows * S lines of length M = 2^lgM,
// one after another, T = max(1, M / E) threads each; a column pass: C lines,
// interleaved in groups of at most FX_MAX_INTERLEAVE.
constexpr int FX_MAX_INTERLEAVE = 8;
constexpr int FX_MAX_WARPS = 32;

inline int fx_line_threads(int L, int E) { return L > E ? L / E : 1; }

template <int E>
__device__ __forceinline__ FxLine fx_line(int lg, int lgC, bool whole_block) {
    constexpr int lgE = E == 8 ? 3 : E == 4 ? 2 : 1;
    FxLine ln;
    ln.lg = lg;
    ln.lgC = lgC;
    const int lgT = lg > lgE ? lg - lgE : 0;
    ln.T = 1 << lgT;
    ln.c = threadIdx.x & ((1 << lgC) - 1);
    ln.lane = (threadIdx.x >> lgC) & (ln.T - 1);
    const int nthr = blockDim.x, wbase = threadIdx.x & ~31;
    // 0: the barriers are the block's
    ln.warp_mask = whole_block || lgT + lgC > 5 ? 0u : nthr - wbase >= 32 ? 0xffffffffu : (1u << (nthr - wbase)) - 1u;
    return ln;
}

enum { ROW_IN_REAL = 0, ROW_IN_HAT = 1 };
// Flux stage of the variable-mobility step between a row's c2r and r2c:
// g <- (M - M0[s]) (g / N^d) (FLUX_DM) or M (g / N^d) (FLUX_M).
enum { FLUX_NONE = 0, FLUX_DM = 1, FLUX_M = 2 };

// c2r of one row from its half spectrum src[0..M] to the packed real row
// z[n] = x[2n] + i x[2n+1], n = lane + i T, in r[i].  The pre-processing
//     Z[k] = (X[k] + conj X[M-k]) + i conj(w^k) (X[k] - conj X[M-k])
// takes the modes k and M - k together: with T = conj(w^k) (X[k] - conj X[M-k])
// and E = X[k] + conj X[M-k], Z[k] = E + i T and Z[M-k] = conj(E - i T), one
// twiddle product for two modes.  The imaginary parts of the k = 0 and k = M
// bins do not reach the real row (FFTW's c2r contract; they are not round-off
// zeros when the spectrum is i k times a field).  Headroom G = log2 M + 3.
template <int E>
__device__ __forceinline__ void fx_row_c2r(double2 (&r)[E], const double2 *__restrict__ src, bool active,
                                           const FxLine &ln, fx2 *&cur, fx2 *&oth, const int4 *__restrict__ twf,
                                           int *sm_w) {
    const int M = 1 << ln.lg, np = min(E, M) / 2;
    double2 xa[E / 2], xb[E / 2], xm = make_double2(0.0, 0.0);
    int mag = 0;
#pragma unroll
    for(int i = 0; i < E / 2; i++) {
        const int k = ln.lane + i * ln.T;
        xa[i] = xb[i] = make_double2(0.0, 0.0);
        if(active && i < np) {
            xa[i] = src[k];
            xb[i] = src[M - k];
            if(k == 0) xa[i].y = xb[i].y = 0.0;
        }
        mag = max(mag, max(max(fx_mag(xa[i].x), fx_mag(xa[i].y)), max(fx_mag(xb[i].x), fx_mag(xb[i].y))));
    }
    if(ln.lane == 0 && active) {
        xm = src[M / 2];
        mag = max(mag, max(fx_mag(xm.x), fx_mag(xm.y)));
    }
    mag = fx_line_max(mag, 1, ln.T, sm_w);
    const FxScale s = fx_line_scale(mag, ln.lg + 3);
    double2 all[E + 1];
#pragma unroll
    for(int i = 0; i < E / 2; i++) {
        all[i] = xa[i];
        all[E / 2 + i] = xb[i];
    }
    all[E] = xm;
    fx_scale_by(all, s.odd, s.pre);
    // stored with real and imaginary parts swapped: the inverse transform
    const int a0 = ln.at(ln.lane);
#pragma unroll
    for(int i = 0; i < E / 2; i++) {
        if(i < np) {
            const int k = ln.lane + i * ln.T;
            const fx2 a = fx_in(all[i], s), b = fx_in(all[E / 2 + i], s);
            const fx2 e = fx2{a.x + b.x, a.y - b.y};
            const fx2 t = fx_cmul<true>(fx2{a.x - b.x, a.y + b.y}, __ldg(&twf[k]));
            cur[a0 + i * ln.step(ln.T)] = fx2{e.y + t.x, e.x - t.y};
            if(k > 0) cur[ln.at(M - k)] = fx2{t.x - e.y, e.x + t.y};
        }
    }
    if(ln.lane == 0 && M > 1) {
        const fx2 a = fx_in(all[E], s);
        cur[ln.at(M / 2)] = fx2{-2 * a.y, 2 * a.x};
    }
    ln.sync();
    fx2 v[E];
#pragma unroll
    for(int i = 0; i < E; i++) v[i] = (i < M) ? cur[a0 + i * ln.step(ln.T)] : fx2{0, 0};
    fx_swap_buf(cur, oth);
    fx_fft(v, ln, cur, oth, twf, ln.lg + 1);
#pragma unroll
    for(int i = 0; i < E; i++) r[i] = fx_out(fx_swap(v[i]), s);
    fx_scale_by(r, s.odd, s.post);
}

// r2c of one packed real row r[i] to its half spectrum dst[0..M], the
// post-processing X[k] = (a + t) / 2, X[M-k] = conj(a - t) / 2 with
// a = Z[k] + conj Z[M-k], t = w^k (-i) (Z[k] - conj Z[M-k]), two modes to a
// product as above; the halving is folded into the output scale, and 2^-down.
template <int E>
__device__ __forceinline__ void fx_row_r2c(double2 (&r)[E], double2 *__restrict__ dst, bool active,
                                           const FxLine &ln, fx2 *&cur, fx2 *&oth, const int4 *__restrict__ twf,
                                           int *sm_w, int down = 0) {
    const int M = 1 << ln.lg, np = min(E, M) / 2;
    int mag = 0;
#pragma unroll
    for(int i = 0; i < E; i++)
        if(i < M) mag = max(mag, max(fx_mag(r[i].x), fx_mag(r[i].y)));
    mag = fx_line_max(mag, 1, ln.T, sm_w);
    FxScale s = fx_line_scale(mag, ln.lg + 3);
    fx_scale_by(r, s.odd, s.pre);
    fx2 v[E];
#pragma unroll
    for(int i = 0; i < E; i++) v[i] = (i < M) ? fx_in(r[i], s) : fx2{0, 0};
    fx_fft(v, ln, cur, oth, twf, ln.lg + 1);
    const int a0 = ln.at(ln.lane);
#pragma unroll
    for(int i = 0; i < E; i++)
        if(i < M) cur[a0 + i * ln.step(ln.T)] = v[i];
    ln.sync();
    s.sh += 1 + down;
    double2 x[E + 1];
#pragma unroll
    for(int i = 0; i < E / 2; i++) {
        x[i] = x[E / 2 + i] = make_double2(0.0, 0.0);
        if(i < np) {
            const int k = ln.lane + i * ln.T;
            const fx2 zk = v[i], zc = cur[k ? ln.at(M - k) : a0];
            const fx2 a = fx2{zk.x + zc.x, zk.y - zc.y};
            const fx2 t = fx_cmul<false>(fx2{zk.y + zc.y, zc.x - zk.x}, __ldg(&twf[k]));
            x[i] = fx_out(fx2{a.x + t.x, a.y + t.y}, s);
            x[E / 2 + i] = fx_out(fx2{a.x - t.x, t.y - a.y}, s);
            if(k == 0) x[i].y = x[E / 2 + i].y = 0.0;
        }
    }
    x[E] = make_double2(0.0, 0.0);
    if(ln.lane == 0) {
        const fx2 z = cur[ln.at(M / 2)];
        x[E] = fx_out(fx2{2 * z.x, -2 * z.y}, s);
    }
    fx_scale_by(x, s.odd, s.post);
    if(active) {
#pragma unroll
        for(int i = 0; i < E / 2; i++) {
            if(i < np) {
                const int k = ln.lane + i * ln.T;
                dst[k] = x[i];
                dst[M - k] = x[E / 2 + i];
            }
        }
        if(ln.lane == 0) dst[M / 2] = x[E];
    }
    fx_swap_buf(cur, oth);
}

// f'(rho) of a line's cells in registers.  The formula of one cell inlines
// once, not eight times: the values of the longer models go through the
// thread's own slots of shared memory in a loop.
template <int KIND, int E>
__device__ __forceinline__ void row_fprime(double2 (&r)[E], const ModelDev &m, const FxLine &ln, fx2 *&cur, fx2 *&oth,
                                           int s, int line_size, bool active) {
    const int ne = min(E, 1 << ln.lg), a0 = ln.at(ln.lane), as = ln.step(ln.T);
    if constexpr(KIND == CHGB_MODEL_LANDAU) {
#pragma unroll
        for(int i = 0; i < E; i++) {
            der_bulk<KIND>(m, &r[i].x, &r[i].x);
            der_bulk<KIND>(m, &r[i].y, &r[i].y);
        }
    }
    else {
        double2 *A = reinterpret_cast<double2 *>(cur);
#pragma unroll
        for(int i = 0; i < E; i++)
            if(i < ne) A[a0 + i * as] = r[i];
        if constexpr(KIND == CHGB_MODEL_SIMPLE_WERTHEIM) {
#pragma unroll 1
            for(int i = 0; i < ne; i++) {
                double2 v = A[a0 + i * as];
                der_bulk<KIND>(m, &v.x, &v.x);
                der_bulk<KIND>(m, &v.y, &v.y);
                A[a0 + i * as] = v;
            }
        }
        else {
            // der_bulk<CHGB_MODEL_SALEH>, term by term, each species' line its own:
            // the first two lines form the log X of their pairs in their second
            // buffer, the linker's adds them up in its own, then every line adds
            // its logarithm and writes f' over that
            double2 *B = reinterpret_cast<double2 *>(oth);
            __syncthreads();
            if(active && s < 2) {
                const double2 *R2 = A + (2 - s) * line_size;
                const double delta = s == 0 ? m.dAA : m.dBB, sv = s == 0 ? m.sv0 : m.sv1;
#pragma unroll 1
                for(int i = 0; i < ne; i++) {
                    const int p = a0 + i * as;
                    const double2 o = A[p], c = R2[p];
                    B[p] = make_double2(saleh_log_X(delta, sv, o.x, m.half, c.x, m.logtab),
                                        saleh_log_X(delta, sv, o.y, m.half, c.y, m.logtab));
                }
            }
            __syncthreads();
            if(active && s == 2) {
#pragma unroll 1
                for(int i = 0; i < ne; i++) {
                    const int p = a0 + i * as;
                    const double2 l0 = B[p - 2 * line_size], l1 = B[p - line_size];
                    B[p] = make_double2(l0.x + l1.x, l0.y + l1.y);
                }
            }
            __syncthreads();
            if(active) {
                const double2 *R = A - s * line_size;
                const double v = s == 0 ? m.sv0 : s == 1 ? m.sv1 : m.half;
#pragma unroll 1
                for(int i = 0; i < ne; i++) {
                    const int p = a0 + i * as;
                    const double2 r0 = R[p], r1 = R[p + line_size], r2 = R[p + 2 * line_size], o = A[p], l = B[p];
                    double2 d;
#pragma unroll
                    for(int h = 0; h < 2; h++) {
                        const double rho_tot = ((0. + (h ? r0.y : r0.x)) + (h ? r1.y : r1.x)) + (h ? r2.y : r2.x);
                        const double b2 = m.two_B2 * rho_tot, b3 = 3.0 * m.B3 * (rho_tot * rho_tot);
                        const double own = h ? o.y : o.x;
                        const double f = (own != 0.) ? ((fx_log(own, m.logtab) + b2) + b3) + v * (h ? l.y : l.x) : 0.0;
                        if(h) d.y = f;
                        else d.x = f;
                    }
                    B[p] = d;
                }
            }
            // the other lines may still read this one's A: the next exchange writes B first
            A = B;
            fx_swap_buf(cur, oth);
        }
#pragma unroll
        for(int i = 0; i < E; i++)
            if(i < ne) r[i] = A[a0 + i * as];
    }
}

// ROW pass: line li of the CTA is species li % S of row row0 + li / S.
// Half-spectrum rows live at work[s * hat + row * H]; real rows at
// real[s * bins + row * N].  The shared memory holds two buffers of the CTA's
// blockDim / T lines.  The transforms run in fixed point; f' and the stored
// values are FP64.  FLUX: the mobility stage
// applied to the real row between the two transforms (mob, M0 as
// psm_flux_kernel's).
template <int KIND, int E, int IN, bool FPRIME, bool WRITE_REAL, bool R2C, int FLUX = FLUX_NONE>
__device__ __forceinline__ void row_body(double2 *__restrict__ work, const double *__restrict__ real_in,
                                         double *__restrict__ real_out, int lgM, int rows_per_cta, long long bins,
                                         long long hat, const int4 *__restrict__ twf, const ModelDev &m,
                                         long long row0, fx2 *sm, const double *__restrict__ mob = nullptr,
                                         const double *__restrict__ M0 = nullptr) {
    constexpr int S = NSpecies<KIND>::value;
    __shared__ int sm_w[2][FX_MAX_WARPS];
    const FxLine ln = fx_line<E>(lgM, 0, S > 1);
    const int M = 1 << lgM, N = 2 * M, H = M + 1;
    const int LS = fx_line_size(M), lines = rows_per_cta * S;
    const int li = threadIdx.x / ln.T, nl = blockDim.x / ln.T;
    const int s = li % S;
    const long long row = row0 + li / S;
    const bool active = li < lines && CHGB_BC(106, row * N + N - 1, bins) && CHGB_BC(107, row * H + H - 1, hat);
    fx2 *cur = sm + li * LS, *oth = sm + (nl + li) * LS;
    double2 r[E];

    if constexpr(IN == ROW_IN_REAL) {
        const double2 *src = reinterpret_cast<const double2 *>(real_in + s * bins + row * N);
#pragma unroll
        for(int i = 0; i < E; i++)
            r[i] = (active && i < M) ? src[ln.lane + i * ln.T] : make_double2(0.0, 0.0);
    }
    else {
        fx_row_c2r(r, work + s * hat + row * H, active, ln, cur, oth, twf, sm_w[0]);
    }
    if constexpr(WRITE_REAL) {
        double2 *dst = reinterpret_cast<double2 *>(real_out + s * bins + row * N);
#pragma unroll
        for(int i = 0; i < E; i++)
            if(active && i < M) dst[ln.lane + i * ln.T] = r[i];
    }
    if constexpr(FLUX != FLUX_NONE) {
        const double2 *mrow = reinterpret_cast<const double2 *>(mob + s * bins + row * N);
        const double m0 = (FLUX == FLUX_DM && active) ? M0[s] : 0.0;
#pragma unroll
        for(int i = 0; i < E; i++) {
            if(active && i < M) {
                const double2 mm = mrow[ln.lane + i * ln.T];
                if(FLUX == FLUX_DM) r[i] = make_double2((mm.x - m0) * r[i].x, (mm.y - m0) * r[i].y);
                else r[i] = make_double2(mm.x * r[i].x, mm.y * r[i].y);
            }
        }
    }
    if constexpr(FPRIME) row_fprime<KIND, E>(r, m, ln, cur, oth, s, LS, active);
    // the flux's division by N^d, a power of two, is one of the scale
    if constexpr(R2C)
        fx_row_r2c(r, work + s * hat + row * H, active, ln, cur, oth, twf, sm_w[1],
                   FLUX != FLUX_NONE ? 63 - __clzll(bins) : 0);
}

// Threads of a row CTA: at most 256 a line (E = 8: N = 4096).
template <int KIND>
struct RowThreads {
    static constexpr int value = 256 * NSpecies<KIND>::value;
};

template <int KIND, int E, int IN, bool FPRIME, bool WRITE_REAL, bool R2C, int FLUX = FLUX_NONE>
__global__ void __launch_bounds__(RowThreads<KIND>::value) row_kernel(double2 *__restrict__ work,
                                                                      const double *__restrict__ real_in,
                                                                      double *__restrict__ real_out, int lgM,
                                                                      int rows_per_cta, long long bins, long long hat,
                                                                      const int4 *__restrict__ twf, ModelDev m,
                                                                      const double *__restrict__ mob,
                                                                      const double *__restrict__ M0) {
    extern __shared__ fx2 sm2[];
    pdl_begin();
    row_body<KIND, E, IN, FPRIME, WRITE_REAL, R2C, FLUX>(work, real_in, real_out, lgM, rows_per_cta, bins, hat, twf, m,
                                                      (long long) blockIdx.x * rows_per_cta, sm2, mob, M0);
}

// Batched row pass of one time step: CTA b takes rows items[b].y.. of replica items[b].x.
template <int KIND>
__global__ void __launch_bounds__(256) row_batch_kernel(const PsBatchRep *__restrict__ reps,
                                                        const int2 *__restrict__ items) {
    extern __shared__ fx2 sm2[];
    const int2 it = items[blockIdx.x];
    const PsBatchRep &r = reps[it.x];
    if(r.E == 2)
        row_body<KIND, 2, ROW_IN_HAT, true, false, true>(r.work, nullptr, nullptr, r.log2N - 1, r.row_rpc, r.bins, r.hat,
                                                         r.twf, r.m, it.y, sm2);
    else
        row_body<KIND, 4, ROW_IN_HAT, true, false, true>(r.work, nullptr, nullptr, r.log2N - 1, r.row_rpc, r.bins, r.hat,
                                                         r.twf, r.m, it.y, sm2);
}

enum { COL_FWD = 0, COL_INV = 1, COL_STEP = 2, COL_INIT = 3, COL_GRAD_INV = 4, COL_FWD_DIV = 5, COL_FWD_MU = 6,
       COL_UPD_INV = 7, COL_LOAD_INV = 8, COL_STEP_REC = 9 };

// The pointwise stages of the variable-mobility step that ride on the last
// axis' column pass (src/integrators/PseudospectralMobilityCPU.cpp:249-306).
// Their spectra and tables lie column by column (species-major), `work` by rows;
// kd holds 0 for the modes that dealiasing drops; fields a mode does not use
// stay null.
//   COL_GRAD_INV (load):  i k_d src                                    (:258-263)
//   COL_FWD_DIV (store):  div (= if first, += otherwise) i k_d f       (:284-293)
//   COL_FWD_MU (store):   psi_hat = f'_hat; out = f'_hat + two_k q2 rho (:249-254)
//   COL_UPD_INV (load):   rho <- the semi-implicit update with f'_hat = psi_hat; rho N^-d (:296-306)
struct ColOps {
    const double *kd, *q2, *M0;
    const double2 *src, *div_in;
    double2 *out, *rho;
    int first, with_div;
    int log2_bins;
    double two_k, dt, inv_dt, Ssplit;
};

// dt / x: the reciprocal in integers (relative 2^-58, then one rounding) where
// both are in its range.
__device__ __noinline__ static double div_fallback(double a, double x) { return a / x; }
__device__ __forceinline__ double dt_over(double dt, double x) {
    if(!un_takes(x) || !un_takes(dt)) return div_fallback(dt, x);
    return __longlong_as_double((long long) un_to_bits(un_mul(un_of(dt), un_rcp(un_of(x)))));
}

// One transform of a column line: r[i] = values at positions lane + i T, INV
// the unnormalised inverse, times 2^-down.  Headroom G = log2 L + 1.
template <bool INV, int E>
__device__ __forceinline__ void fx_col_fft(double2 (&r)[E], const FxLine &ln, int C, fx2 *&cur, fx2 *&oth,
                                           const int4 *__restrict__ twf, int *sm_w, int down = 0) {
    const int L = 1 << ln.lg;
    int mag = 0;
#pragma unroll
    for(int i = 0; i < E; i++)
        if(i < L) mag = max(mag, max(fx_mag(r[i].x), fx_mag(r[i].y)));
    mag = fx_line_max(mag, C, ln.T * C, sm_w);
    FxScale s = fx_line_scale(mag, ln.lg + 1);
    fx_scale_by(r, s.odd, s.pre);
    fx2 v[E];
#pragma unroll
    for(int i = 0; i < E; i++) {
        v[i] = (i < L) ? fx_in(r[i], s) : fx2{0, 0};
        if(INV) v[i] = fx_swap(v[i]);
    }
    fx_fft(v, ln, cur, oth, twf, ln.lg);
    s.sh += down;
#pragma unroll
    for(int i = 0; i < E; i++) r[i] = fx_out(INV ? fx_swap(v[i]) : v[i], s);
    fx_scale_by(r, s.odd, s.post);
}

// COL pass: C lines (adjacent half-spectrum columns kx0..) of one species and
// one plane per CTA, in groups of at most FX_MAX_INTERLEAVE interleaved lines;
// element pos of column kx at
//   off = species * hat + plane * plane_stride + kx + pos * elem_stride.
// The shared memory holds two buffers of C lines.
template <int MODE, int E>
__device__ __forceinline__ void col_body(double2 *__restrict__ work, double2 *__restrict__ psi_hat,
                                         const double2 *__restrict__ ab, int lgL, int H, int lgC, long long elem_stride, long long plane_stride, long long hat,
                                         const int4 *__restrict__ twf, double scale, int kx0, long long plane,
                                         long long species, fx2 *sm, const ColOps &ops = ColOps()) {
    __shared__ int sm_w[2][FX_MAX_WARPS * FX_MAX_INTERLEAVE];
    const int lgI = min(lgC, 3), I = 1 << lgI;   // interleaved lines of a group
    const FxLine ln = fx_line<E>(lgL, lgI, false);
    const int L = 1 << lgL, LS = fx_line_size(L) << lgI;
    const int group = threadIdx.x / (ln.T << lgI), groups = 1 << (lgC - lgI);
    const int kx = kx0 + (group << lgI) + ln.c;
    const bool active = group < groups && kx < H;
    fx2 *cur = sm + group * LS, *oth = sm + (blockDim.x / (ln.T << lgI) + group) * LS;
    const long long off0 = species * hat + plane * plane_stride + kx + ln.lane * elem_stride;
    const long long dT = ln.T * elem_stride;
    // the same mode in a spectrum that is kept column by column
    const long long line0 = species * hat + ((plane * H + kx) << lgL) + ln.lane;
    double2 r[E];
    const double m0 = MODE == COL_UPD_INV ? ops.M0[species] : 0.0;
#pragma unroll
    for(int i = 0; i < E; i++) {
        r[i] = make_double2(0.0, 0.0);
        const long long off = off0 + i * dT;
        if(!active || i >= L || !CHGB_BC(101, off - species * hat, hat)) continue;
        double2 v;
        if(MODE == COL_LOAD_INV) {
            v = psi_hat[line0 + i * ln.T];
        }
        else if(MODE == COL_GRAD_INV) {
            v = mul_ik(ops.kd[line0 + i * ln.T], ops.src[line0 + i * ln.T]);
        }
        else if(MODE == COL_UPD_INV) {
            // the reference's (rho + dt div - c (f' - S rho)) / (1 + c (S + 2 k q^2)), c =
            // dt M0 q^2, with its numerator less rho times its denominator where that is
            // below 2: rho + dt / (1 + ...) (div - M0 q^2 (f' + 2 k q^2 rho)), whose
            // rounding is rho's alone.  A mode that is damped further would keep the
            // rounding of the larger value it had: there as it stands, dt taken out.  12
            // FP64 instructions a mode either way and a reciprocal in integers, against 22
            // with a corrected division of each part.  The two forms against the first
            // alone, us a step: 2D N=1024 176.6 -> 177.6, 3D N=128 428.6 -> 432.5 (as
            // operands selected for the same FMAs 179.6 and 433.5)
            const long long lo = line0 + i * ln.T;
            const double k2 = ops.q2[lo], t = ops.two_k * k2, mk = m0 * k2;
            const double den = fma(ops.dt * mk, ops.Ssplit + t, 1.0), g = dt_over(ops.dt, den);
            const double2 q = ops.rho[lo], f = psi_hat[lo];
            const double2 d = ops.with_div ? ops.div_in[lo] : make_double2(0.0, 0.0);
            if(den < 2.0) {
                v.x = fma(g, fma(-mk, fma(t, q.x, f.x), d.x), q.x);
                v.y = fma(g, fma(-mk, fma(t, q.y, f.y), d.y), q.y);
            }
            else {
                const double a = fma(mk, ops.Ssplit, ops.inv_dt);
                v.x = g * fma(a, q.x, fma(-mk, f.x, d.x));
                v.y = g * fma(a, q.y, fma(-mk, f.y, d.y));
            }
            ops.rho[lo] = v;
        }
        else {
            v = work[off];
        }
        r[i] = v;
    }
    constexpr bool INV = MODE == COL_INV || MODE == COL_LOAD_INV || MODE == COL_GRAD_INV || MODE == COL_UPD_INV;
    fx_col_fft<INV>(r, ln, I, cur, oth, twf, sm_w[0], MODE == COL_UPD_INV ? ops.log2_bins : 0);
    if constexpr(MODE == COL_STEP || MODE == COL_STEP_REC) {
#pragma unroll
        for(int i = 0; i < E; i++) {
            const long long off = line0 + i * ln.T;
            if(!active || i >= L || !CHGB_BC(101, off - species * hat, hat)) continue;
            const double2 ph = psi_hat[off], c = ab[off];
            const double2 nv = make_double2(fma(c.x, ph.x, -c.y * r[i].x), fma(c.x, ph.y, -c.y * r[i].y));
            psi_hat[off] = nv;
            // a trajectory's record (a mode of its own: as a test of the pointer it cost the
            // plain step 2 %)
            if(MODE == COL_STEP_REC) ops.out[off] = nv;
            r[i] = nv;
        }
        fx_col_fft<true>(r, ln, I, cur, oth, twf, sm_w[1]);
    }
#pragma unroll
    for(int i = 0; i < E; i++) {
        const long long off = off0 + i * dT;
        if(!active || i >= L || !CHGB_BC(101, off - species * hat, hat)) continue;
        double2 f = r[i];
        if(MODE == COL_INIT) {
            psi_hat[line0 + i * ln.T] = make_double2(f.x * scale, f.y * scale);
        }
        else if(MODE == COL_FWD_MU) {
            const long long lo = line0 + i * ln.T;
            psi_hat[lo] = f;
            const double t = ops.two_k * ops.q2[lo];
            const double2 q = ops.rho[lo];
            ops.out[lo] = make_double2(fma(t, q.x, f.x), fma(t, q.y, f.y));
        }
        else if(MODE == COL_FWD_DIV) {
            const long long lo = line0 + i * ln.T;
            const double k = ops.kd[lo];
            if(ops.first) {
                ops.out[lo] = mul_ik(k, f);
            }
            else {
                const double2 d = ops.out[lo];
                ops.out[lo] = make_double2(fma(-k, f.y, d.x), fma(k, f.x, d.y));
            }
        }
        else {
            work[off] = f;
        }
    }
}

template <int MODE, int E>
__global__ void __launch_bounds__(512, E == 8 ? 1 : 2) col_kernel(double2 *__restrict__ work, double2 *__restrict__ psi_hat,
                                                  const double2 *__restrict__ ab, int lgL, int H, int lgC,
                                                  long long elem_stride,
                                                  long long plane_stride, long long hat,
                                                  const int4 *__restrict__ twf, double scale, ColOps ops) {
    extern __shared__ fx2 sm2[];
    pdl_begin();
    col_body<MODE, E>(work, psi_hat, ab, lgL, H, lgC, elem_stride, plane_stride, hat, twf, scale,
                   (int) blockIdx.x << lgC, blockIdx.y, blockIdx.z, sm2, ops);
}

// Batched 2D column pass (forward, update, inverse) of one time step:
// CTA b takes columns items[b].z.. of species items[b].y of replica items[b].x.
__global__ void __launch_bounds__(256, 4) col_batch_kernel(const PsBatchRep *__restrict__ reps,
                                                           const int4 *__restrict__ items) {
    extern __shared__ fx2 sm2[];
    const int4 it = items[blockIdx.x];
    const PsBatchRep &r = reps[it.x];
    if(r.E == 2)
        col_body<COL_STEP, 2>(r.work, r.psi_hat, r.ab, r.log2N, r.H, r.log2C, r.H, 0, r.hat, r.twf, 0.0, it.z, 0, it.y, sm2);
    else
        col_body<COL_STEP, 4>(r.work, r.psi_hat, r.ab, r.log2N, r.H, r.log2C, r.H, 0, r.hat, r.twf, 0.0, it.z, 0, it.y, sm2);
}

// 1D: elementwise init (psi_t = F[rho] / N) or update on the half spectrum.
__global__ void update1d_kernel(double2 *__restrict__ work, double2 *__restrict__ psi_hat,
                                const double2 *__restrict__ ab, long long n, int init, double scale) {
    for(long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < n; i += (long long) gridDim.x * blockDim.x) {
        double2 f = work[i];
        if(init) {
            psi_hat[i] = make_double2(f.x * scale, f.y * scale);
        }
        else {
            double2 ph = psi_hat[i];
            const double2 c = ab[i];
            double2 nv = make_double2(fma(c.x, ph.x, -c.y * f.x), fma(c.x, ph.y, -c.y * f.y));
            psi_hat[i] = nv;
            work[i] = nv;
        }
    }
}

int ilog2(int n) {
    int l = 0;
    while((1 << l) < n) l++;
    return l;
}

}  // namespace

// A column pass's launch shape: values per thread, log2 of the columns per CTA.
struct ColShape {
    int E = 8, lgC = 0, threads = 1;
    size_t smem = 0;
};

struct SpectralState {
    chgb_params p;
    Geom g;
    ModelDev m;
    int H = 0;
    long long hat = 0;       // complex values per species
    double2 *psi_hat = nullptr, *work = nullptr;
    int4 *twf = nullptr;      // the twiddles in fixed point (bfp.cuh): limbs of round(w 2^62)
    double2 *ab = nullptr;    // the update's coefficients (alpha, beta) of every mode
    const double *real_buf = nullptr;  // the handle's real-space density buffer
    bool real_valid = false;  // the real buffer holds the current rho
    bool hat_valid = false;   // work holds the x-half-spectrum rows of the current rho
    // launch shapes: rows per row CTA; the column passes, and COL_STEP's
    int row_rpc = 1, row_threads = 1;
    size_t row_smem = 0;
    ColShape col, step;
    bool pdl = true;          // programmatic dependent launch of the passes
    int row_E = 8;            // values per thread of the row transforms
};

// Where a mode stands in the spectra kept column by column (psi_hat, ab and the
// adjoint's), by its place in the rows' order.  The transforms' own buffer
// `work` is written by rows; the arrays that only the last axis' column pass
// touches lie along its columns, where a warp reads 512 contiguous bytes instead
// of 16 from each of 32 rows.
long long spectral_line_index(const Geom &g, long long mode) {
    if(g.dims == 1) return mode;
    const long long lines = (long long) (g.N / 2 + 1) * (g.dims == 3 ? g.N : 1);
    return mode % lines * g.N + mode / lines;
}

// Wave-vector tables of src/integrators/PseudospectralCPU.cpp:32-86, folded
// into the update coefficients.
static void build_tables(const SpectralState &s, std::vector<double2> &ab) {
    const int N = s.g.N, dims = s.g.dims, S = s.g.S;
    const double dx = s.p.dx, dt = s.p.dt, M = s.p.M, Ssplit = s.p.splitting_S;
    const double bins = (double) s.g.bins;
    std::vector<double> k2v(s.hat), mask(s.hat);
    double k_cut = N * M_PI / (N * dx) * 2.0 / 3.0;
    long long idx = 0;
    if(dims == 1) {
        for(int i = 0; i < s.H; i++, idx++) {
            double k = 2.0 * M_PI * i / (N * dx);
            mask[idx] = (k <= k_cut) ? 1.0 : 0.0;
            k2v[idx] = k * k;
        }
    }
    else if(dims == 2) {
        for(int kx_idx = 0; kx_idx < N; kx_idx++) {
            int kx = (kx_idx < N / 2) ? kx_idx : N - kx_idx;
            for(int ky = 0; ky < N / 2 + 1; ky++, idx++) {
                double k = 2.0 * M_PI * std::sqrt((double) (kx * kx + ky * ky)) / (N * dx);
                mask[idx] = (k < k_cut) ? 1.0 : 0.0;
                k2v[idx] = k * k;
            }
        }
    }
    else {
        for(int kx_idx = 0; kx_idx < N; kx_idx++) {
            int kx_i = (kx_idx < N / 2) ? kx_idx : (kx_idx - N);
            double kx = 2.0 * M_PI * kx_i / (N * dx);
            for(int ky_idx = 0; ky_idx < N; ky_idx++) {
                int ky_i = (ky_idx < N / 2) ? ky_idx : (ky_idx - N);
                double ky = 2.0 * M_PI * ky_i / (N * dx);
                for(int kz_idx = 0; kz_idx < N / 2 + 1; kz_idx++, idx++) {
                    double kz = 2.0 * M_PI * kz_idx / (N * dx);
                    double k2 = kx * kx + ky * ky + kz * kz;
                    double k = std::sqrt(k2);
                    mask[idx] = (k <= k_cut) ? 1.0 : 0.0;
                    k2v[idx] = k2;
                }
            }
        }
    }
    ab.resize((size_t) S * s.hat);
    for(int sp = 0; sp < S; sp++) {
        for(long long i = 0; i < s.hat; i++) {
            double k2 = k2v[i], k4 = k2 * k2;
            double denom = 1.0 + dt * M * (Ssplit * k2 + 2.0 * s.p.k[sp] * k4);
            double c = dt * M * k2;
            double dm = s.p.use_dealias ? mask[i] : 1.0;
            ab[sp * s.hat + spectral_line_index(s.g, i)] = make_double2((1.0 + c * Ssplit) / denom, c * dm / denom / bins);
        }
    }
}

// One fixed-point twiddle component: W = round(v 2^62) = hi 2^32 + lo, both
// signed (bfp.cuh).  lo = -2^31 becomes -2^31 + 1: the kernels negate limbs.
static void fx_limbs(long double v, int &hi, int &lo) {
    const long long W = llroundl(v * 4611686018427387904.0L);   // 2^62
    lo = (int) (uint32_t) (W & 0xFFFFFFFFll);
    hi = (int) ((W - lo) >> 32);
    if(lo == INT32_MIN) lo = -INT32_MAX;
}

// W[q] = exp(-2 pi i q / N), q < N, in fixed point for the transforms of
// bfp.cuh: built from one octant in long double so that the table is exactly
// symmetric (W[N/4] = -i, W[N/2] = -1 exactly), then rounded to 2^-62.
static void build_twiddles(int N, std::vector<int4> &wf) {
    wf.resize(N);
    for(int q = 0; q < N; q++) {
        // reduce q to the first octant with exact symmetries
        long double c, s;
        int oct = (int) (((long long) q * 8) / N);
        int r = q - oct * (N / 8);
        auto cs = [&](long double num, long double &co, long double &si) {
            long double a = 2.0L * 3.141592653589793238462643383279502884L * num / (long double) N;
            co = cosl(a);
            si = sinl(a);
        };
        long double co, si;
        if(N < 8) {
            cs((long double) q, co, si);
            c = co;
            s = si;
            if(q * 4 == N) { c = 0; s = 1; }
            if(q * 2 == N) { c = -1; s = 0; }
            if(q * 4 == 3 * N) { c = 0; s = -1; }
        }
        else {
            int e = N / 8;
            // angle = (oct * e + r) * 2pi/N = oct * pi/4 + r * 2pi/N
            switch(oct) {
                case 0: cs(r, co, si); c = co; s = si; break;
                case 1: cs(e - r, co, si); c = si; s = co; break;       // pi/2 - t
                case 2: cs(r, co, si); c = -si; s = co; break;          // pi/2 + t
                case 3: cs(e - r, co, si); c = -co; s = si; break;      // pi - t
                case 4: cs(r, co, si); c = -co; s = -si; break;         // pi + t
                case 5: cs(e - r, co, si); c = -si; s = -co; break;     // 3pi/2 - t
                case 6: cs(r, co, si); c = si; s = -co; break;          // 3pi/2 + t
                default: cs(e - r, co, si); c = co; s = -si; break;     // 2pi - t
            }
        }
        int4 f;
        fx_limbs(c, f.x, f.y);
        fx_limbs(-s, f.z, f.w);
        wf[q] = f;
    }
}

static void tune_col_shape(SpectralState *s);

// Values per thread of a box's line transforms.  The fewer, the more warps and
// the shorter each one's chain of products, which hides the latencies of loads
// and exchanges; the more, the fewer exchanges and twiddle products.  Two where
// one box leaves most of the GPU's schedulers idle (2D N <= 256, 3D N <= 64),
// four up to N = 1024, eight for longer lines, whose 512 threads of four would
// leave two CTAs to an SM.
// GB300, us per `pseudospectral` step of one box alone / of three at once:
//          2D N=64     N=256      N=512      N=1024     N=2048     3D N=32    N=64       N=128      N=256
//   two    10.7/4.1   13.6/5.8   22.6/12.1                         18.0/6.7   33.0/13.5  92.0/74.8
//   four   14.9/5.2   14.8/5.7   19.7/10.7  45.4/35.1  196/183     22.0/8.3   34.5/14.6  91.2/75.2  675/649
//   eight                        24.8/11.4  47.2/36.3  196/173                46.1/21.2  108 /83.1  778/718
// (2D N=256 with two: the adjoint's 200 steps 9080 -> 7685 us, two GMRES steps
// 2062 -> 1715; a batch of 33 boxes up to N=512 2742 -> 2778.)
static int fx_line_elems(const Geom &g) { return g.N <= (g.dims == 3 ? 64 : 256) ? 2 : g.N <= 1024 ? 4 : 8; }

// The shape with C columns per CTA.
static ColShape col_shape(const Geom &g, int E, int C) {
    ColShape c;
    c.E = E;
    c.lgC = ilog2(C);
    c.threads = C * fx_line_threads(g.N, E);
    c.smem = sizeof(fx2) * 2 * (size_t) C * fx_line_size(g.N);
    return c;
}

// Let a kernel take `smem` bytes of dynamic shared memory.  The limit is one of
// the kernel, not of a handle: it is only ever set to the largest a CTA can
// have beside the kernels' static arrays, so that no handle lowers another's.
static cudaError_t allow_smem(const void *f, size_t smem) {
    if(smem <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024);
}

int spectral_create(const chgb_params &p, const Geom &g, const ModelDev &m, SpectralState **out, std::string &err) {
    *out = nullptr;
    if(g.N > 4096) {
        err = "pseudospectral supports N <= 4096";
        return CHGB_ERR_INVALID;
    }
    SpectralState *s = new SpectralState();
    s->p = p;
    s->g = g;
    s->m = m;
    s->H = g.N / 2 + 1;
    s->hat = s->H;
    for(int d = 1; d < g.dims; d++) s->hat *= g.N;
    size_t hat_bytes = sizeof(double2) * (size_t) s->hat * g.S;
    bool ok = cudaMalloc(&s->psi_hat, hat_bytes) == cudaSuccess && cudaMalloc(&s->work, hat_bytes) == cudaSuccess &&
              cudaMalloc(&s->ab, hat_bytes) == cudaSuccess &&
              cudaMalloc(&s->twf, sizeof(int4) * g.N) == cudaSuccess;
    if(!ok) {
        cudaGetLastError();
        spectral_destroy(s);
        err = "device allocation failed";
        return CHGB_ERR_ALLOC;
    }
    std::vector<double2> ab;
    build_tables(*s, ab);
    std::vector<int4> wf;
    build_twiddles(g.N, wf);
    ok = cudaMemcpy(s->ab, ab.data(), hat_bytes, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(s->twf, wf.data(), sizeof(int4) * wf.size(), cudaMemcpyHostToDevice) == cudaSuccess;
    if(!ok) {
        spectral_destroy(s);
        err = "table upload failed";
        return CHGB_ERR_CUDA;
    }
    s->row_E = fx_line_elems(g);
    s->pdl = g.dims == 3;
    // launch shapes.  A CTA takes at least a warp's worth of lines, then more up
    // to 128 threads while ~2 CTAs per SM are left: small boxes want their few
    // lines spread over as many SMs as possible
    constexpr long long kSpreadCtas = 2 * 152;
    const int M = g.N / 2;
    const long long rows = (long long) g.bins / g.N;
    const int row_T = fx_line_threads(M, s->row_E);
    s->row_rpc = 1;
    while(s->row_rpc * 2 * row_T * g.S <= 128 && s->row_rpc * 2 <= rows &&
          (s->row_rpc * row_T * g.S < 32 || rows / (s->row_rpc * 2) >= kSpreadCtas))
        s->row_rpc *= 2;
    s->row_threads = s->row_rpc * g.S * row_T;
    s->row_smem = sizeof(fx2) * 2 * (size_t) (s->row_threads / row_T) * fx_line_size(M);
    const long long col_lines = (long long) s->H * (g.dims == 3 ? g.N : 1) * g.S;
    auto spread = [&](int E) {
        const int T = fx_line_threads(g.N, E);
        int C = 1;
        while(C * 2 * T <= 256 && C * 2 <= FX_MAX_INTERLEAVE && (C * T < 32 || col_lines / (C * 2) >= kSpreadCtas))
            C *= 2;
        return col_shape(g, E, C);
    };
    s->col = spread(fx_line_elems(g));
    s->step = spread(fx_line_elems(g));
    // shared-memory attributes, once
    auto setattr = [](const void *f, size_t smem) { allow_smem(f, smem); };
#define SETROW(K, E)                                                                            \
    setattr((const void *) row_kernel<K, E, ROW_IN_REAL, false, false, true>, s->row_smem);     \
    setattr((const void *) row_kernel<K, E, ROW_IN_REAL, true, false, true>, s->row_smem);      \
    setattr((const void *) row_kernel<K, E, ROW_IN_HAT, true, false, true>, s->row_smem);       \
    setattr((const void *) row_kernel<K, E, ROW_IN_HAT, false, true, false>, s->row_smem);      \
    setattr((const void *) row_kernel<K, E, ROW_IN_HAT, true, true, true>, s->row_smem);        \
    setattr((const void *) row_kernel<K, E, ROW_IN_HAT, false, false, true, FLUX_DM>, s->row_smem); \
    setattr((const void *) row_kernel<K, E, ROW_IN_HAT, false, false, true, FLUX_M>, s->row_smem);
    SETROW(CHGB_MODEL_LANDAU, 8)
    SETROW(CHGB_MODEL_SIMPLE_WERTHEIM, 8)
    SETROW(CHGB_MODEL_SALEH, 8)
    SETROW(CHGB_MODEL_LANDAU, 4)
    SETROW(CHGB_MODEL_SIMPLE_WERTHEIM, 4)
    SETROW(CHGB_MODEL_SALEH, 4)
    SETROW(CHGB_MODEL_LANDAU, 2)
    SETROW(CHGB_MODEL_SIMPLE_WERTHEIM, 2)
    SETROW(CHGB_MODEL_SALEH, 2)
#undef SETROW
#define SETCOL(E)                                                                                                  \
    for(const void *f : {(const void *) col_kernel<COL_FWD, E>, (const void *) col_kernel<COL_INV, E>,             \
                         (const void *) col_kernel<COL_STEP, E>, (const void *) col_kernel<COL_INIT, E>,           \
                         (const void *) col_kernel<COL_GRAD_INV, E>, (const void *) col_kernel<COL_FWD_DIV, E>,    \
                         (const void *) col_kernel<COL_FWD_MU, E>, (const void *) col_kernel<COL_UPD_INV, E>,      \
                         (const void *) col_kernel<COL_LOAD_INV, E>, (const void *) col_kernel<COL_STEP_REC, E>})  \
        setattr(f, 224 * 1024);   // whatever shape the timing below picks
    SETCOL(8)
    SETCOL(4)
    SETCOL(2)
#undef SETCOL
    cudaError_t e = cudaGetLastError();
    if(e != cudaSuccess) {
        spectral_destroy(s);
        err = std::string("kernel configuration: ") + cudaGetErrorString(e);
        return CHGB_ERR_CUDA;
    }
    tune_col_shape(s);
    *out = s;
    return CHGB_OK;
}

void spectral_destroy(SpectralState *s) {
    if(!s) return;
    if(s->psi_hat) cudaFree(s->psi_hat);
    if(s->work) cudaFree(s->work);
    if(s->ab) cudaFree(s->ab);
    if(s->twf) cudaFree(s->twf);
    delete s;
}

void spectral_set_pdl(SpectralState *s, bool on) { s->pdl = s->pdl && on; }

namespace {

// A pass as a programmatic dependent launch (pdl_begin in the kernels): the
// next pass's CTAs are placed while the last ones of this pass drain.
template <typename... Params, typename... Args>
cudaError_t launch_pass(const SpectralState *s, void (*kernel)(Params...), dim3 grid, int threads, size_t smem,
                        cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned) threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = s->pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

dim3 row_grid(const SpectralState *s) { return dim3((unsigned) ((long long) s->g.bins / s->g.N / s->row_rpc)); }

template <int KIND, int IN, bool FPRIME, bool WRITE_REAL, bool R2C>
cudaError_t launch_row_kind(SpectralState *s, const double *real_in, double *real_out, cudaStream_t st) {
    auto kernel = s->row_E == 8   ? row_kernel<KIND, 8, IN, FPRIME, WRITE_REAL, R2C>
                  : s->row_E == 4 ? row_kernel<KIND, 4, IN, FPRIME, WRITE_REAL, R2C>
                                  : row_kernel<KIND, 2, IN, FPRIME, WRITE_REAL, R2C>;
    return launch_pass(s, kernel, row_grid(s), s->row_threads, s->row_smem, st, s->work, real_in, real_out, ilog2(s->g.N) - 1, s->row_rpc, s->g.bins, s->hat, s->twf, s->m,
                       nullptr, nullptr);
}

// Row pass of the variable-mobility flux: c2r of work's rows, the flux stage, r2c back into work.
template <int KIND, int FLUX>
cudaError_t launch_row_flux_kind(SpectralState *s, const double *mob, const double *M0, cudaStream_t st) {
    auto kernel = s->row_E == 8   ? row_kernel<KIND, 8, ROW_IN_HAT, false, false, true, FLUX>
                  : s->row_E == 4 ? row_kernel<KIND, 4, ROW_IN_HAT, false, false, true, FLUX>
                                  : row_kernel<KIND, 2, ROW_IN_HAT, false, false, true, FLUX>;
    return launch_pass(s, kernel, row_grid(s), s->row_threads, s->row_smem, st, s->work, nullptr, nullptr, ilog2(s->g.N) - 1, s->row_rpc, s->g.bins, s->hat,
                       s->twf, s->m, mob, M0);
}

template <int FLUX>
cudaError_t launch_row_flux(SpectralState *s, const double *mob, const double *M0, cudaStream_t st) {
    switch(s->m.kind) {
        case CHGB_MODEL_LANDAU: return launch_row_flux_kind<CHGB_MODEL_LANDAU, FLUX>(s, mob, M0, st);
        case CHGB_MODEL_SIMPLE_WERTHEIM: return launch_row_flux_kind<CHGB_MODEL_SIMPLE_WERTHEIM, FLUX>(s, mob, M0, st);
        default: return launch_row_flux_kind<CHGB_MODEL_SALEH, FLUX>(s, mob, M0, st);
    }
}

template <int IN, bool FPRIME, bool WRITE_REAL, bool R2C>
cudaError_t launch_row(SpectralState *s, const double *real_in, double *real_out, cudaStream_t st) {
    switch(s->m.kind) {
        case CHGB_MODEL_LANDAU:
            return launch_row_kind<CHGB_MODEL_LANDAU, IN, FPRIME, WRITE_REAL, R2C>(s, real_in, real_out, st);
        case CHGB_MODEL_SIMPLE_WERTHEIM:
            return launch_row_kind<CHGB_MODEL_SIMPLE_WERTHEIM, IN, FPRIME, WRITE_REAL, R2C>(s, real_in, real_out, st);
        default: return launch_row_kind<CHGB_MODEL_SALEH, IN, FPRIME, WRITE_REAL, R2C>(s, real_in, real_out, st);
    }
}

// axis: 1 = y, 2 = z (3D only).  planes/strides follow the [z][y][kx] layout.
// `spec`: the spectrum, column by column, that the pass loads or stores in place
// of the state's psi (COL_INIT then keeps the transform unscaled).
template <int MODE>
cudaError_t launch_col(SpectralState *s, int axis, cudaStream_t st, const ColOps &ops = ColOps(),
                       double2 *spec = nullptr) {
    const int N = s->g.N, H = s->H;
    long long elem_stride, plane_stride;
    int planes;
    if(s->g.dims == 2) {
        elem_stride = H;
        plane_stride = 0;
        planes = 1;
    }
    else if(axis == 1) {
        elem_stride = H;
        plane_stride = (long long) N * H;
        planes = N;
    }
    else {
        elem_stride = (long long) N * H;
        plane_stride = H;
        planes = N;
    }
    const ColShape &c = MODE == COL_STEP || MODE == COL_STEP_REC ? s->step : s->col;
    const int C = 1 << c.lgC;
    auto kernel = c.E == 8 ? col_kernel<MODE, 8> : c.E == 4 ? col_kernel<MODE, 4> : col_kernel<MODE, 2>;
    return launch_pass(s, kernel, dim3((unsigned) ((H + C - 1) / C), (unsigned) planes, (unsigned) s->g.S), c.threads,
                       c.smem, st, s->work, spec ? spec : s->psi_hat, s->ab, ilog2(N), H, c.lgC, elem_stride, plane_stride, s->hat,
                       s->twf, spec ? 1.0 : 1.0 / (double) s->g.bins, ops);
}

}  // namespace

// Columns per CTA of the column passes, timed at create.  Adjacent columns in
// one CTA use whole 32-byte sectors of the strided column loads, while fewer,
// larger CTAs spread the lines over fewer SMs; which wins depends on the box.
// So boxes of 2^18 cells and more time one column step and one forward pass
// with 1, 2, 4 and 8 columns per CTA (those that fit 512 threads and the shared
// memory) on a state filled with noise, and keep the fastest of each.  Every
// shape gives the same bits: a line's transform does not depend on its CTA.
// The state is zeroed afterwards (an upload sets it).
template <int MODE>
static void tune_col_mode(SpectralState *s, ColShape &shape, cudaStream_t st, cudaEvent_t ev0, cudaEvent_t ev1) {
    const int axis = s->g.dims - 1;
    ColShape pick = shape;
    float best = 0.0f;
    for(int C : {1, 2, 4, 8}) {
        shape = col_shape(s->g, shape.E, C);
        if(shape.threads > 512 || shape.threads < 32 || shape.smem > 224 * 1024) continue;
        cudaError_t e = launch_col<MODE>(s, axis, st);   // warm-up
        if(e == cudaSuccess) e = cudaEventRecord(ev0, st);
        for(int r = 0; r < 5 && e == cudaSuccess; r++) e = launch_col<MODE>(s, axis, st);
        if(e == cudaSuccess) e = cudaEventRecord(ev1, st);
        if(e == cudaSuccess) e = cudaEventSynchronize(ev1);
        float ms = 0.0f;
        if(e == cudaSuccess) e = cudaEventElapsedTime(&ms, ev0, ev1);
        if(e != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        if(best == 0.0f || ms < best) {
            best = ms;
            pick = shape;
        }
    }
    shape = pick;
}

static void tune_col_shape(SpectralState *s) {
    if(s->g.dims < 2 || (long long) s->g.bins < (1ll << 18)) return;
    cudaStream_t st = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    if(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess ||
       cudaEventCreate(&ev0) != cudaSuccess || cudaEventCreate(&ev1) != cudaSuccess) {
        cudaGetLastError();
        if(ev0) cudaEventDestroy(ev0);
        if(st) cudaStreamDestroy(st);
        return;
    }
    const long long nd = s->hat * s->g.S * 2;   // doubles of psi_hat / work
    if(launch_fill_noise(reinterpret_cast<double *>(s->psi_hat), 0.0, 1e-2, nd, st) == cudaSuccess &&
       launch_fill_noise(reinterpret_cast<double *>(s->work), 0.0, 1e-2, nd, st) == cudaSuccess) {
        tune_col_mode<COL_STEP>(s, s->step, st, ev0, ev1);
        tune_col_mode<COL_FWD>(s, s->col, st, ev0, ev1);
    }
    cudaMemsetAsync(s->psi_hat, 0, sizeof(double) * nd, st);
    cudaMemsetAsync(s->work, 0, sizeof(double) * nd, st);
    cudaStreamSynchronize(st);
    cudaGetLastError();
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
    cudaStreamDestroy(st);
}

namespace {

cudaError_t launch_update1d(SpectralState *s, int init, cudaStream_t st) {
    long long n = s->hat * s->g.S;
    int grid = (int) std::min<long long>((n + 255) / 256, 152 * 8);
    update1d_kernel<<<grid, 256, 0, st>>>(s->work, s->psi_hat, s->ab, n, init, 1.0 / (double) s->g.bins);
    return cudaGetLastError();
}

}  // namespace

int spectral_set_rho(SpectralState *s, const double *d_rho, cudaStream_t st, int64_t *launches, std::string &err) {
    s->real_buf = d_rho;
    cudaError_t e = launch_row<ROW_IN_REAL, false, false, true>(s, d_rho, nullptr, st);
    int n = 1;
    if(e == cudaSuccess) {
        if(s->g.dims == 1) {
            e = launch_update1d(s, 1, st);
            n++;
        }
        else if(s->g.dims == 2) {
            e = launch_col<COL_INIT>(s, 1, st);
            n++;
        }
        else {
            e = launch_col<COL_FWD>(s, 1, st);
            if(e == cudaSuccess) e = launch_col<COL_INIT>(s, 2, st);
            n += 2;
        }
    }
    *launches += n;
    if(e != cudaSuccess) {
        err = std::string("pseudospectral init: ") + cudaGetErrorString(e);
        return CHGB_ERR_CUDA;
    }
    s->real_valid = true;
    s->hat_valid = false;
    return CHGB_OK;
}

int spectral_step(SpectralState *s, int64_t nsteps, cudaStream_t st, int64_t *launches, std::string &err) {
    // The real buffer is only an input of the first step after an upload.
    for(int64_t t = 0; t < nsteps; t++) {
        cudaError_t e;
        if(s->hat_valid) e = launch_row<ROW_IN_HAT, true, false, true>(s, nullptr, nullptr, st);
        else e = launch_row<ROW_IN_REAL, true, false, true>(s, s->real_buf, nullptr, st);
        int n = 1;
        if(e == cudaSuccess) {
            if(s->g.dims == 1) {
                e = launch_update1d(s, 0, st);
                n++;
            }
            else if(s->g.dims == 2) {
                e = launch_col<COL_STEP>(s, 1, st);
                n++;
            }
            else {
                e = launch_col<COL_FWD>(s, 1, st);
                if(e == cudaSuccess) e = launch_col<COL_STEP>(s, 2, st);
                if(e == cudaSuccess) e = launch_col<COL_INV>(s, 1, st);
                n += 3;
            }
        }
        *launches += n;
        if(e != cudaSuccess) {
            err = std::string("pseudospectral step: ") + cudaGetErrorString(e);
            return CHGB_ERR_CUDA;
        }
        s->hat_valid = true;
        s->real_valid = false;
    }
    return CHGB_OK;
}

int spectral_real(SpectralState *s, double *d_rho, cudaStream_t st, int64_t *launches, std::string &err) {
    if(s->real_valid) return CHGB_OK;
    cudaError_t e = launch_row<ROW_IN_HAT, false, true, false>(s, nullptr, d_rho, st);
    *launches += 1;
    if(e != cudaSuccess) {
        err = std::string("pseudospectral real field: ") + cudaGetErrorString(e);
        return CHGB_ERR_CUDA;
    }
    s->real_valid = true;
    return CHGB_OK;
}

}  // namespace chgb

// ---------------------------------------------------------------------------
// batched 2D steps
// ---------------------------------------------------------------------------
namespace chgb {

// A batch CTA takes at least one whole row of every species, and one whole
// column.  (Three species need 384 threads a row at N = 1024: such a box runs on
// its own, where it fills the GPU alone.)
bool spectral_batchable(const SpectralState *s) {
    return s->g.dims == 2 && s->g.N >= 8 && s->g.N <= 1024 &&
           fx_line_threads(s->g.N / 2, s->row_E) * s->g.S <= PS_BATCH_THREADS &&
           fx_line_threads(s->g.N, s->step.E) <= PS_BATCH_THREADS;
}

bool spectral_hat_valid(const SpectralState *s) { return s->hat_valid; }

void spectral_mark_stepped(SpectralState *s) {
    s->hat_valid = true;
    s->real_valid = false;
}

void spectral_batch_rep(const SpectralState *s, PsBatchRep *r, size_t *row_smem, size_t *col_smem) {
    const int N = s->g.N, M = N / 2, S = s->g.S;
    r->work = s->work;
    r->psi_hat = s->psi_hat;
    r->ab = s->ab;
    r->twf = s->twf;
    r->m = s->m;
    r->N = N;
    r->log2N = ilog2(N);
    r->H = s->H;
    r->bins = s->g.bins;
    r->hat = s->hat;
    r->E = s->row_E;   // the columns' as well
    const int row_T = fx_line_threads(M, s->row_E), col_T = fx_line_threads(N, s->step.E);
    r->row_rpc = 1;
    while(r->row_rpc * 2 * row_T * S <= PS_BATCH_THREADS && r->row_rpc * 2 <= N) r->row_rpc *= 2;
    r->col_C = std::max(1, std::min(PS_BATCH_THREADS / col_T, 16));
    r->log2C = ilog2(r->col_C);
    *row_smem = sizeof(fx2) * 2 * (size_t) (PS_BATCH_THREADS / row_T) * fx_line_size(M);
    *col_smem = sizeof(fx2) * 2 * (size_t) (PS_BATCH_THREADS / col_T) * fx_line_size(N);
}

namespace {
template <int KIND>
cudaError_t configure_kind(size_t row_smem, size_t col_smem) {
    cudaError_t e = allow_smem((const void *) row_batch_kernel<KIND>, row_smem);
    if(e == cudaSuccess) e = allow_smem((const void *) col_batch_kernel, col_smem);
    return e;
}
}  // namespace

cudaError_t configure_ps2d_batch(int kind, size_t row_smem, size_t col_smem) {
    switch(kind) {
        case CHGB_MODEL_LANDAU: return configure_kind<CHGB_MODEL_LANDAU>(row_smem, col_smem);
        case CHGB_MODEL_SIMPLE_WERTHEIM: return configure_kind<CHGB_MODEL_SIMPLE_WERTHEIM>(row_smem, col_smem);
        default: return configure_kind<CHGB_MODEL_SALEH>(row_smem, col_smem);
    }
}

cudaError_t launch_ps2d_batch(int kind, const PsBatchRep *reps, const int2 *row_items, int nrow, const int4 *col_items,
                              int ncol, size_t row_smem, size_t col_smem, cudaStream_t st) {
    if(nrow > 0) {
        switch(kind) {
            case CHGB_MODEL_LANDAU:
                row_batch_kernel<CHGB_MODEL_LANDAU><<<nrow, PS_BATCH_THREADS, row_smem, st>>>(reps, row_items);
                break;
            case CHGB_MODEL_SIMPLE_WERTHEIM:
                row_batch_kernel<CHGB_MODEL_SIMPLE_WERTHEIM><<<nrow, PS_BATCH_THREADS, row_smem, st>>>(reps, row_items);
                break;
            default: row_batch_kernel<CHGB_MODEL_SALEH><<<nrow, PS_BATCH_THREADS, row_smem, st>>>(reps, row_items); break;
        }
        cudaError_t e = cudaGetLastError();
        if(e != cudaSuccess) return e;
    }
    if(ncol > 0) col_batch_kernel<<<ncol, PS_BATCH_THREADS, col_smem, st>>>(reps, col_items);
    return cudaGetLastError();
}

}  // namespace chgb

namespace chgb {
const double2 *spectral_psi_hat(const SpectralState *s, int species) { return s->psi_hat + (size_t) species * s->hat; }
}  // namespace chgb

// ---------------------------------------------------------------------------
// Adjoint of the 2D Landau pseudospectral step (backward pass of chgb_adjoint_*)
//
// Forward, in real space: psi' = A psi - B f'(psi), A = C2R diag(alpha) R2C / N^2,
// B = C2R diag(beta) R2C (both symmetric).  Adjoint, kept in Fourier space
// (lam_hat = R2C(lam)):
//     lam_hat_n = alpha lam_hat_{n+1} - R2C( f''(psi_n) * C2R(beta lam_hat_{n+1}) ),
// the same two-kernel structure as the forward step, with the same
// fixed-point transforms.  Parameter gradients,
// with <u, C2R(X)> = sum_full X_k conj(R2C(u)_k):
//   dL/deps += <B lam_{n+1}, psi_n>                          (row pass)
//   dL/dk   += sum_k w_k Re(conj lam_hat_{n+1} * tk * psi_t_{n+1})
//   dL/dM   += sum_k w_k Re(conj lam_hat_{n+1} * (tm1 psi_t_{n+1} - tm2 psi_t_n))
// with tk = -2 dt M q^4 / den, tm1 = 1 / (M den), tm2 = 2 k q^4 dt / den^2 + alpha / (M den)
// (dalpha/dk, dbeta/dk are -2 dt M q^4/den times alpha, beta; dbeta/dM = beta/(M den)
// and beta f_hat_n = alpha psi_t_n - psi_t_{n+1}).
// ---------------------------------------------------------------------------
namespace chgb {

namespace {

// Sum over the block; the result is valid in thread 0.
__device__ __forceinline__ double block_sum(double v, double *red) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    const int n = min(32, (int) blockDim.x - w * 32);
    const unsigned mask = n == 32 ? 0xffffffffu : (1u << n) - 1u;
    for(int o = 16; o > 0; o >>= 1) {
        const double t = __shfl_down_sync(mask, v, o);
        if(lane + o < n) v += t;
    }
    __syncthreads();
    if(lane == 0) red[w] = v;
    __syncthreads();
    double t = 0.0;
    if(threadIdx.x == 0)
        for(int i = 0; i < nw; i++) t += red[i];
    return t;
}

// Row pass of the adjoint step: work rows (x half spectrum of beta lam_hat after
// the inverse y transform) -> C2R -> B lam; geps += <B lam, psi_n>; * f''(psi_n) -> R2C.
template <int E>
__global__ void __launch_bounds__(256) row_adj_kernel(double2 *__restrict__ work, const double *__restrict__ psi_n,
                                                     int lgM, int rows_per_cta, const int4 *__restrict__ twf,
                                                     double eps, double *__restrict__ geps) {
    extern __shared__ fx2 sm2[];
    __shared__ double red[32];
    __shared__ int sm_w[2][FX_MAX_WARPS];
    const FxLine ln = fx_line<E>(lgM, 0, false);
    const int M = 1 << lgM, N = 2 * M, LS = fx_line_size(M);
    const int li = threadIdx.x / ln.T, nl = blockDim.x / ln.T;
    const long long row = (long long) blockIdx.x * rows_per_cta + li;
    fx2 *cur = sm2 + li * LS, *oth = sm2 + (nl + li) * LS;
    double2 r[E];
    fx_row_c2r(r, work + row * (M + 1), true, ln, cur, oth, twf, sm_w[0]);
    double acc = 0.0;
    const double2 *pr = reinterpret_cast<const double2 *>(psi_n + row * N);
#pragma unroll
    for(int i = 0; i < E; i++) {
        if(i < M) {
            const double2 b = r[i], p = pr[ln.lane + i * ln.T];
            acc = fma(b.x, p.x, acc);
            acc = fma(b.y, p.y, acc);
            r[i] = make_double2(b.x * fma(3.0 * p.x, p.x, -eps), b.y * fma(3.0 * p.y, p.y, -eps));
        }
    }
    const double t = block_sum(acc, red);
    if(threadIdx.x == 0) geps[blockIdx.x] += t;
    fx_row_r2c(r, work + row * (M + 1), true, ln, cur, oth, twf, sm_w[1]);
}

enum { ADJ_A = 1, ADJ_B = 2, ADJ_BA = 3 };

// Column pass of the adjoint: B part (forward y FFT of the row result, lam_hat
// update) and/or A part (gradient sums with psi_next = psi_t_{n+1} and
// psi_cur = psi_t_n, then beta * lam_hat and the inverse y FFT into work).
template <int MODE, int E>
__global__ void __launch_bounds__(512) col_adj_kernel(double2 *__restrict__ work, double2 *__restrict__ lam,
                                                     const double2 *__restrict__ ab,
                                                     const double *__restrict__ tk, const double *__restrict__ tm1,
                                                     const double *__restrict__ tm2,
                                                     const double2 *__restrict__ psi_next,
                                                     const double2 *__restrict__ psi_cur, int lgL, int H, int lgC,
                                                     const int4 *__restrict__ twf, double *__restrict__ gk,
                                                     double *__restrict__ gm) {
    extern __shared__ fx2 sm2[];
    __shared__ double red[32];
    __shared__ int sm_w[2][FX_MAX_WARPS * FX_MAX_INTERLEAVE];
    const int C = 1 << lgC;   // at most FX_MAX_INTERLEAVE: one group
    const FxLine ln = fx_line<E>(lgL, lgC, false);
    const int L = 1 << lgL;
    const int kx = blockIdx.x * C + ln.c;
    const bool active = kx < H;
    fx2 *cur = sm2, *oth = sm2 + (fx_line_size(L) << lgC);
    // work by rows, lam, psi and the tables by columns
    const long long off0 = kx + (long long) ln.lane * H, dT = (long long) ln.T * H;
    const long long line0 = ((long long) kx << lgL) + ln.lane;
    double2 r[E];
#pragma unroll
    for(int i = 0; i < E; i++)
        r[i] = (!active || i >= L) ? make_double2(0.0, 0.0) : (MODE & ADJ_B) ? work[off0 + i * dT] : lam[line0 + i * ln.T];
    if(MODE & ADJ_B) {
        fx_col_fft<false>(r, ln, C, cur, oth, twf, sm_w[0]);
#pragma unroll
        for(int i = 0; i < E; i++) {
            if(active && i < L) {
                const long long off = line0 + i * ln.T;
                const double2 l = lam[off];
                const double al = ab[off].x;
                r[i] = make_double2(fma(al, l.x, -r[i].x), fma(al, l.y, -r[i].y));
                lam[off] = r[i];
            }
        }
    }
    if(MODE & ADJ_A) {
        double ak = 0.0, am = 0.0;
        const double w = (kx == 0 || kx == L / 2) ? 1.0 : 2.0;
#pragma unroll
        for(int i = 0; i < E; i++) {
            if(active && i < L) {
                const long long off = line0 + i * ln.T;
                const double2 l = r[i], pn = psi_next[off], pc = psi_cur[off];
                const double dn = fma(l.x, pn.x, l.y * pn.y);
                const double dc = fma(l.x, pc.x, l.y * pc.y);
                ak = fma(w * tk[off], dn, ak);
                am = fma(w, fma(tm1[off], dn, -tm2[off] * dc), am);
                const double be = ab[off].y;
                r[i] = make_double2(be * l.x, be * l.y);
            }
        }
        double t = block_sum(ak, red);
        if(threadIdx.x == 0) gk[blockIdx.x] += t;
        t = block_sum(am, red);
        if(threadIdx.x == 0) gm[blockIdx.x] += t;
        fx_col_fft<true>(r, ln, C, cur, oth, twf, sm_w[1]);
#pragma unroll
        for(int i = 0; i < E; i++)
            if(active && i < L) work[off0 + i * dT] = r[i];
    }
}

__global__ void axpy_hat_kernel(double2 *__restrict__ y, const double2 *__restrict__ x, double a, long long n) {
    for(long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < n; i += (long long) gridDim.x * blockDim.x) {
        double2 v = x[i], w = y[i];
        y[i] = make_double2(fma(a, v.x, w.x), fma(a, v.y, w.y));
    }
}

}  // namespace

struct SpectralAdj {
    double *tk = nullptr, *tm1 = nullptr, *tm2 = nullptr;
    double2 *lam = nullptr;
    double2 *work = nullptr;   // the adjoint sweep's own transform scratch (the state's stays free for recomputation)
    double *geps = nullptr, *gk = nullptr, *gm = nullptr;   // per-CTA partial sums
    int n_row_cta = 0, n_col_cta = 0;
};

// The kernels for the state's values per thread.
static auto row_adj_kernel_of(const SpectralState *s) {
    return s->row_E == 8 ? row_adj_kernel<8> : s->row_E == 4 ? row_adj_kernel<4> : row_adj_kernel<2>;
}

template <int E>
static auto col_adj_kernel_of(int mode) {
    return mode == ADJ_A ? col_adj_kernel<ADJ_A, E> : mode == ADJ_B ? col_adj_kernel<ADJ_B, E> : col_adj_kernel<ADJ_BA, E>;
}

static auto col_adj_kernel_of(const SpectralState *s, int mode) {
    return s->col.E == 8 ? col_adj_kernel_of<8>(mode) : s->col.E == 4 ? col_adj_kernel_of<4>(mode) : col_adj_kernel_of<2>(mode);
}

bool spectral_adjoint_supported(const SpectralState *s) {
    return s->g.dims == 2 && s->g.S == 1 && s->m.kind == CHGB_MODEL_LANDAU && s->g.N >= 8;
}

SpectralAdj *spectral_adj_create(SpectralState *s, std::string &err) {
    SpectralAdj *a = new SpectralAdj();
    const int N = s->g.N;
    const double dx = s->p.dx, dt = s->p.dt, M = s->p.M, Ssplit = s->p.splitting_S, k = s->p.k[0];
    std::vector<double> tk(s->hat), tm1(s->hat), tm2(s->hat);
    // the same wave vectors as build_tables (src/integrators/PseudospectralCPU.cpp:44-57)
    for(int kx_idx = 0; kx_idx < N; kx_idx++) {
        int kx = (kx_idx < N / 2) ? kx_idx : N - kx_idx;
        for(int ky = 0; ky < N / 2 + 1; ky++) {
            double kk = 2.0 * M_PI * std::sqrt((double) (kx * kx + ky * ky)) / (N * dx);
            double k2 = kk * kk, k4 = k2 * k2;
            double denom = 1.0 + dt * M * (Ssplit * k2 + 2.0 * k * k4);
            double c = dt * M * k2;
            double alpha = (1.0 + c * Ssplit) / denom;
            const long long at = (long long) ky * N + kx_idx;
            tk[at] = -2.0 * dt * M * k4 / denom;
            tm1[at] = 1.0 / (M * denom);
            tm2[at] = 2.0 * k * k4 * dt / (denom * denom) + alpha / (M * denom);
        }
    }
    a->n_row_cta = (int) (((long long) s->g.bins / N) / s->row_rpc);
    a->n_col_cta = (s->H + (1 << s->col.lgC) - 1) >> s->col.lgC;
    bool ok = cudaMalloc(&a->tk, sizeof(double) * s->hat) == cudaSuccess &&
              cudaMalloc(&a->tm1, sizeof(double) * s->hat) == cudaSuccess &&
              cudaMalloc(&a->tm2, sizeof(double) * s->hat) == cudaSuccess &&
              cudaMalloc(&a->lam, sizeof(double2) * s->hat) == cudaSuccess &&
              cudaMalloc(&a->work, sizeof(double2) * s->hat) == cudaSuccess &&
              cudaMalloc(&a->geps, sizeof(double) * a->n_row_cta) == cudaSuccess &&
              cudaMalloc(&a->gk, sizeof(double) * a->n_col_cta) == cudaSuccess &&
              cudaMalloc(&a->gm, sizeof(double) * a->n_col_cta) == cudaSuccess;
    ok = ok && cudaMemcpy(a->tk, tk.data(), sizeof(double) * s->hat, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(a->tm1, tm1.data(), sizeof(double) * s->hat, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(a->tm2, tm2.data(), sizeof(double) * s->hat, cudaMemcpyHostToDevice) == cudaSuccess;
    if(ok) {
        size_t rs = s->row_smem, cs = s->col.smem;
        allow_smem((const void *) row_adj_kernel_of(s), rs);
        for(int mode : {ADJ_A, ADJ_B, ADJ_BA}) allow_smem((const void *) col_adj_kernel_of(s, mode), cs);
        ok = cudaGetLastError() == cudaSuccess;
    }
    if(!ok) {
        cudaGetLastError();
        spectral_adj_destroy(a);
        err = "adjoint allocation failed";
        return nullptr;
    }
    return a;
}

void spectral_adj_destroy(SpectralAdj *a) {
    if(!a) return;
    cudaFree(a->tk);
    cudaFree(a->tm1);
    cudaFree(a->tm2);
    cudaFree(a->lam);
    cudaFree(a->work);
    cudaFree(a->geps);
    cudaFree(a->gk);
    cudaFree(a->gm);
    delete a;
}

double2 *spectral_adj_lam(SpectralAdj *a) { return a->lam; }

cudaError_t spectral_adj_zero(SpectralAdj *a, const SpectralState *s, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(a->geps, 0, sizeof(double) * a->n_row_cta, st);
    if(e == cudaSuccess) e = cudaMemsetAsync(a->gk, 0, sizeof(double) * a->n_col_cta, st);
    if(e == cudaSuccess) e = cudaMemsetAsync(a->gm, 0, sizeof(double) * a->n_col_cta, st);
    if(e == cudaSuccess) e = cudaMemsetAsync(a->lam, 0, sizeof(double2) * s->hat, st);
    return e;
}

cudaError_t spectral_adj_add_seed(SpectralAdj *a, const SpectralState *s, const double2 *x, double scale,
                                  cudaStream_t st) {
    int grid = (int) std::min<long long>((s->hat + 255) / 256, 152 * 8);
    axpy_hat_kernel<<<grid, 256, 0, st>>>(a->lam, x, scale, s->hat);
    return cudaGetLastError();
}

// mode: 1 = A only (start of a segment), 2 = B only (end), 3 = B then A
cudaError_t spectral_adj_col(SpectralAdj *a, SpectralState *s, int mode, const double2 *psi_next,
                             const double2 *psi_cur, cudaStream_t st) {
    const int N = s->g.N;
    dim3 grid((unsigned) a->n_col_cta);
#define ADJ_COL_ARGS                                                                                                   \
    a->work, a->lam, s->ab, a->tk, a->tm1, a->tm2, psi_next, psi_cur, ilog2(N), s->H, s->col.lgC, s->twf,      \
        a->gk, a->gm
    col_adj_kernel_of(s, mode)<<<grid, s->col.threads, s->col.smem, st>>>(ADJ_COL_ARGS);
#undef ADJ_COL_ARGS
    return cudaGetLastError();
}

cudaError_t spectral_adj_row(SpectralAdj *a, SpectralState *s, const double *psi_n, cudaStream_t st) {
    row_adj_kernel_of(s)<<<a->n_row_cta, s->row_threads, s->row_smem, st>>>(a->work, psi_n, ilog2(s->g.N) - 1, s->row_rpc,
                                                                            s->twf, s->m.epsilon, a->geps);
    return cudaGetLastError();
}

// Sum the per-CTA partials in a fixed order: g3 = {sum geps, sum gk, sum gm}.
int spectral_adj_grads(SpectralAdj *a, double *g3) {
    std::vector<double> ge(a->n_row_cta), gk(a->n_col_cta), gm(a->n_col_cta);
    if(cudaMemcpy(ge.data(), a->geps, sizeof(double) * ge.size(), cudaMemcpyDeviceToHost) != cudaSuccess ||
       cudaMemcpy(gk.data(), a->gk, sizeof(double) * gk.size(), cudaMemcpyDeviceToHost) != cudaSuccess ||
       cudaMemcpy(gm.data(), a->gm, sizeof(double) * gm.size(), cudaMemcpyDeviceToHost) != cudaSuccess)
        return CHGB_ERR_CUDA;
    double s0 = 0, s1 = 0, s2 = 0;
    for(double v : ge) s0 += v;
    for(double v : gk) s1 += v;
    for(double v : gm) s2 += v;
    g3[0] = s0;
    g3[1] = s1;
    g3[2] = s2;
    return CHGB_OK;
}

// psi_hat <- hat; work <- inverse y transform of hat (the state a step starts from).
cudaError_t spectral_load_hat(SpectralState *s, const double2 *hat, cudaStream_t st) {
    size_t bytes = sizeof(double2) * (size_t) s->hat * s->g.S;
    cudaError_t e = cudaSuccess;
    if(hat != s->psi_hat) e = cudaMemcpyAsync(s->psi_hat, hat, bytes, cudaMemcpyDeviceToDevice, st);
    if(e == cudaSuccess) e = launch_col<COL_LOAD_INV>(s, 1, st, ColOps(), s->psi_hat);
    s->hat_valid = true;
    s->real_valid = false;
    return e;
}

// One forward step from the half-spectrum state that also writes rho_n (real) to
// real_out and psi_{n+1} to hat_out.
cudaError_t spectral_step_record(SpectralState *s, double *real_out, double2 *hat_out, cudaStream_t st) {
    cudaError_t e = launch_row<ROW_IN_HAT, true, true, true>(s, nullptr, real_out, st);
    ColOps o{};
    o.out = hat_out;
    if(e == cudaSuccess) e = launch_col<COL_STEP_REC>(s, 1, st, o);
    s->hat_valid = true;
    s->real_valid = false;
    return e;
}

// real_out = C2R(hat_scaled) (unnormalised: a scaled state gives the field).
cudaError_t spectral_inverse(SpectralState *s, const double2 *hat_scaled, double *real_out, cudaStream_t st) {
    cudaError_t e = launch_col<COL_LOAD_INV>(s, 1, st, ColOps(), const_cast<double2 *>(hat_scaled));   // read only in this mode
    if(e == cudaSuccess) e = launch_row<ROW_IN_HAT, false, true, false>(s, nullptr, real_out, st);
    s->hat_valid = false;
    return e;
}

double2 *spectral_psi_hat_mut(SpectralState *s) { return s->psi_hat; }

// Plain transforms on caller buffers, FFTW's unnormalised r2c / c2r, S species:
// the row and column passes of a step without the model or the update.  The
// passes run in the state's work array; the last axis' stores and loads the
// spectrum column by column.  1D: `hat` is the work array.
cudaError_t spectral_r2c(SpectralState *s, const double *real, double2 *hat, cudaStream_t st, int *launches) {
    double2 *saved = s->work;
    if(s->g.dims == 1) s->work = hat;
    cudaError_t e = launch_row<ROW_IN_REAL, false, false, true>(s, real, nullptr, st);
    if(e == cudaSuccess && s->g.dims == 3) e = launch_col<COL_FWD>(s, 1, st);
    if(e == cudaSuccess && s->g.dims >= 2) e = launch_col<COL_INIT>(s, s->g.dims - 1, st, ColOps(), hat);
    s->work = saved;
    *launches += s->g.dims;
    return e;
}

cudaError_t spectral_c2r(SpectralState *s, double2 *hat, double *real, cudaStream_t st, int *launches) {
    double2 *saved = s->work;
    if(s->g.dims == 1) s->work = hat;
    cudaError_t e = cudaSuccess;
    if(s->g.dims >= 2) e = launch_col<COL_LOAD_INV>(s, s->g.dims - 1, st, ColOps(), hat);
    if(e == cudaSuccess && s->g.dims == 3) e = launch_col<COL_INV>(s, 1, st);
    if(e == cudaSuccess) e = launch_row<ROW_IN_HAT, false, true, false>(s, nullptr, real, st);
    s->work = saved;
    *launches += s->g.dims;
    return e;
}
long long spectral_hat_size(const SpectralState *s) { return s->hat; }

// ---- the variable-mobility step with its pointwise stages on the passes -----
// dims >= 2.  The stage rides on the slowest axis's column pass (y in 2D, z in
// 3D): the first inverse pass of a c2r loads through it, the last forward pass
// of an r2c stores through it.

cudaError_t spectral_psmob_fprime(SpectralState *s, const double *rho, double2 *fder_hat, double2 *mu,
                                  const double2 *rho_hat, const double *q2, double two_k, cudaStream_t st,
                                  int *launches) {
    const int last = s->g.dims - 1;
    cudaError_t e = launch_row<ROW_IN_REAL, true, false, true>(s, rho, nullptr, st);
    if(e == cudaSuccess && s->g.dims == 3) e = launch_col<COL_FWD>(s, 1, st);
    ColOps o{};
    o.q2 = q2;
    o.rho = const_cast<double2 *>(rho_hat);   // read only in this mode
    o.out = mu;
    o.two_k = two_k;
    if(e == cudaSuccess)
        e = mu ? launch_col<COL_FWD_MU>(s, last, st, o, fder_hat) : launch_col<COL_INIT>(s, last, st, o, fder_hat);
    *launches += s->g.dims;
    return e;
}

cudaError_t spectral_psmob_flux(SpectralState *s, const double2 *src, const double *kd, const double *mob,
                                const double *M0, double2 *div, bool first, cudaStream_t st, int *launches) {
    const int last = s->g.dims - 1;
    ColOps o{};
    o.kd = kd;
    o.src = src;
    o.out = div;
    o.first = first ? 1 : 0;
    cudaError_t e = launch_col<COL_GRAD_INV>(s, last, st, o);
    if(e == cudaSuccess && s->g.dims == 3) e = launch_col<COL_INV>(s, 1, st);
    if(e == cudaSuccess)
        e = M0 ? launch_row_flux<FLUX_DM>(s, mob, M0, st) : launch_row_flux<FLUX_M>(s, mob, nullptr, st);
    if(e == cudaSuccess && s->g.dims == 3) e = launch_col<COL_FWD>(s, 1, st);
    if(e == cudaSuccess) e = launch_col<COL_FWD_DIV>(s, last, st, o);
    *launches += 2 * s->g.dims - 1;
    return e;
}

cudaError_t spectral_psmob_update(SpectralState *s, double2 *rho_hat, const double2 *fder_hat, const double2 *div_hat,
                                  const double *q2, const double *M0, double dt, double Ssplit, double k0,
                                  double *rho, cudaStream_t st, int *launches) {
    ColOps o{};
    o.q2 = q2;
    o.M0 = M0;
    o.rho = rho_hat;
    o.div_in = div_hat;
    o.with_div = div_hat ? 1 : 0;
    o.dt = dt;
    o.inv_dt = 1.0 / dt;
    o.Ssplit = Ssplit;
    o.two_k = 2.0 * k0;
    o.log2_bins = s->g.dims * s->g.log2N;
    cudaError_t e = launch_col<COL_UPD_INV>(s, s->g.dims - 1, st, o, const_cast<double2 *>(fder_hat));   // read only
    if(e == cudaSuccess && s->g.dims == 3) e = launch_col<COL_INV>(s, 1, st);
    if(e == cudaSuccess) e = launch_row<ROW_IN_HAT, false, true, false>(s, nullptr, rho, st);
    *launches += s->g.dims;
    return e;
}

}  // namespace chgb
