// common.cuh — shared device-side definitions of the chgb CUDA library
// (sm_103a, FP64 throughout).
//
// Layout of every field in HBM: species-major, data[s * bins + idx] with
// idx = x + N*y + N*N*z (the reference's MultiField, src/utils/MultiField.h:59-63),
// periodic wrap by bit mask (src/CahnHilliard.cpp:50-56).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/chgb.h"
#include "wertheim_fx.cuh"

namespace chgb {

// Free-energy model constants, derived once on the host from chgb_model_params
// the way the model constructors derive them (src/models/SimpleWertheim.cpp:20-34,
// src/models/SalehWertheim.cpp:19-41).
struct ModelDev {
    int kind;
    int S;
    double epsilon;                 // landau
    double valence;                 // simple_wertheim valence as double
    double B2, B3;
    double two_valence_delta;       // 2 * valence * delta
    double four_valence_delta;      // 2 * two_valence_delta (exact: a power-of-two multiple)
    double two_B2;                  // 2 * B2 (exact)
    double reg_delta, log_delta;    // regularisation_delta and log(regularisation_delta)
    double reg_slope, reg_base;     // below it f' is reg_slope rho + reg_base + valence log X
    double sv0, sv1, half;          // saleh valences of A and B, linker half valence
    double dAA, dBB;
    double dcf;                     // density conversion factor
    int ivalence;
    int sw_fx;                      // simple_wertheim: the integer path (sw_cell) takes the constants
    // table of un_log in device memory; nullptr: the FP64 formulas and the
    // library's log instead
    const UnLogEntry *logtab;
};

// with_log_table = false never allocates (the table is used if an earlier
// call made it for the current device).
ModelDev make_model_dev(const chgb_model_params &m, bool with_log_table = true);

// Grid geometry and the step constants folded once per handle.
struct Geom {
    int dims, N, log2N, mask;
    int bins;                       // N^dims
    int S;
};

struct EulerConsts {
    double c2[CHGB_MAX_SPECIES];    // 2 k_s / dx^2  (surface term of mu)
    double c1;                      // dt * M / dx^2 (constant-mobility update)
    double dt;
    double half_inv_dx2;            // 0.5 / dx^2   (face flux and divergence folded)
    double M;                       // constant mobility / M0
    double lshift[3];               // Landau: 2 d c2 - eps for d = 1, 2, 3 (species 0)
    int mobility_type;
    const double *mobf;             // regularised / gel: the mobility field of this step
};

// Per-step mobility update of the `regularised` and `gel` types
// (src/mobility/RegularisedMobility.h:26-33, src/mobility/GelMobility.h:41-58).
struct MobilityDev {
    int type;                       // CHGB_MOBILITY_REGULARISED or CHGB_MOBILITY_GEL
    double M, rho_min;              // regularised
    double c0;                      // gel
    // gel, folded: g = g_a rho + g_b is (p phi - phi_c) / (1 - phi_c) with phi =
    // (rho + 1) / 2, the order parameter's step c + Mdt c (g - c)
    double g_a, g_b, Mdt;
    Un K;                           // 1 / (c0 ln 2)
    const uint64_t *exptab;         // table of un_expneg (null: the library's exp)
};

// Maximum of a mobility field per species, max(0, max M): the values' bits in
// order as unsigned integers (M > 0; negative ones and NaN are passed over, as
// m < v ? v : m from m = 0 does).  Each block adds its maximum to acc; the last
// one, counted per species, hands it to M0 and clears both for the next launch.
struct M0Sink {
    unsigned long long *acc;
    unsigned *count;
    double *M0;                     // null: no maximum is wanted
};

__device__ __forceinline__ void m0_take(unsigned long long &m, double v) {
    const long long b = __double_as_longlong(v);
    if(b > (long long) m && b <= 0x7FF0000000000000ll) m = (unsigned long long) b;
}

// All threads of a block; species s0 .. s1 - 1 share the value.
__device__ __forceinline__ void m0_commit(unsigned long long m, const M0Sink &sink, int s0, int s1) {
    __shared__ unsigned long long red[32];
#pragma unroll
    for(int o = 16; o > 0; o >>= 1) {
        const unsigned long long v = __shfl_xor_sync(0xFFFFFFFFu, m, o);
        m = m < v ? v : m;
    }
    if((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if(threadIdx.x == 0) {
        for(int w = 1; w < (int) (blockDim.x + 31) / 32; w++) m = m < red[w] ? red[w] : m;
        for(int s = s0; s < s1; s++) {
            atomicMax(&sink.acc[s], m);
            __threadfence();   // the maximum is in before the count says so
            if(atomicAdd(&sink.count[s], 1u) == gridDim.x - 1) {
                __threadfence();
                sink.M0[s] = __longlong_as_double((long long) __ldcg(&sink.acc[s]));
                sink.acc[s] = 0;
                sink.count[s] = 0;
            }
        }
    }
    __syncthreads();   // red is free again
}

// i k z: the wave-vector factor of a spectral derivative
// (src/integrators/PseudospectralMobilityCPU.cpp:258-263)
__device__ __forceinline__ double2 mul_ik(double k, double2 z) { return make_double2(-k * z.y, k * z.x); }

// ---------------------------------------------------------------------------
// Models.  Each formula follows the reference's CPU code (the oracle); the
// reference's own CUDA kernels are single precision and are not followed.
// ---------------------------------------------------------------------------

// x^n for the model's integer valence n >= 0, by repeated squaring: the
// reference's std::pow(X, (double) valence) to within a few ulp at a fraction
// of a general pow's FP64 work.
__device__ __forceinline__ double ipow(double x, int n) {
    double r = 1.0;
    while(n > 0) {
        if(n & 1) r *= x;
        x *= x;
        n >>= 1;
    }
    return r;
}

// 1/x: the hardware's approximate reciprocal (relative error below 2^-20,
// measured on GB300) refined by two Newton steps y <- y + y (1 - x y), each
// squaring the error.  Within 2 ulp of 1/x, for four FMAs instead of the ten
// or so FP64 instructions of a correctly rounded division.  Subnormal x is
// flushed to zero (1/x = inf, then NaN), as for x = 0.
__device__ __forceinline__ double fast_rcp(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double e = fma(-x, y, 1.0);
    y = fma(y, e, y);
    e = fma(-x, y, 1.0);
    return fma(y, e, y);
}

// ln a in units of 2^-53 (wertheim_fx.cuh) through the device's table.
__device__ __forceinline__ int64_t un_log_tab(Un a, const UnLogEntry *__restrict__ tab) {
    return un_log(a, [tab](int j, uint32_t &inv, int64_t &ln) {
        const int4 t = __ldg(reinterpret_cast<const int4 *>(tab + j));
        inv = (uint32_t) t.x;
        ln = (int64_t) (((uint64_t) (uint32_t) t.w << 32) | (uint32_t) t.z);
    });
}
constexpr double UNLOG_UNIT = 1.1102230246251565e-16;   // 2^-53

// A double the integer path takes: positive, finite, normal, its exponent far
// from the range's ends (products of a few stay normal).
__device__ __forceinline__ bool un_takes(double x) {
    return (unsigned) (__double2hiint(x) >> 20) - 600u < 900u;   // 2^-423 .. 2^476; the sign bit fails it
}
__device__ __forceinline__ Un un_of(double x) { return un_from_bits((uint64_t) __double_as_longlong(x)); }

// ln x: one FP64-pipe conversion and a product; 13 FP64 instructions in FP64
// with a table, 29 in the library's log.  Within 2^-52 absolute, and half an
// ulp of the rounding.
__device__ __noinline__ static double log_fallback(double x) { return log(x); }

__device__ __forceinline__ double fx_log(double x, const UnLogEntry *__restrict__ tab) {
    if(tab == nullptr || !un_takes(x)) return log_fallback(x);
    return (double) un_log_tab(un_of(x), tab) * UNLOG_UNIT;
}

// e^(-c/c0) of the gel mobility: in integers (wertheim_fx.cuh) up to c/c0 of
// at least 177 (t below 512 by its exponent, so at most 354), 1 where |c/c0| is below 2^-59, the
// library's exp for the rest: larger ones, negative c, NaN.
__device__ __noinline__ static double exp_fallback(double x) { return exp(x); }

__device__ __forceinline__ double gel_exp(const MobilityDev &md, double c) {
    const uint64_t *tab = md.exptab;
    const int e = ((__double2hiint(c) >> 20) & 0x7FF) - 1023 + md.K.e;   // c/c0 < 2^(e+2) ln 2
    if(tab != nullptr && un_takes(c) && e <= 7)
        return __longlong_as_double((long long) un_to_bits(un_expneg(un_of(c), md.K, [tab](int j) { return __ldg(tab + j); })));
    if(tab != nullptr && e < -60) return 1.0;
    return exp_fallback(-(c / md.c0));
}

// X(rho) of src/models/SimpleWertheim.cpp:88-90 (the division by the fast
// reciprocal above).
__device__ __forceinline__ double sw_X(const ModelDev &m, double rho) {
    return (-1.0 + sqrt(1.0 + m.four_valence_delta * rho)) * fast_rcp(m.two_valence_delta * rho);
}

// X of one Saleh species pair, src/models/SalehWertheim.cpp:80-85; returns log X.
__device__ __noinline__ static double saleh_log_X_fp(double rho_factor) {
    const double X = (-1.0 + sqrt(1.0 + 4.0 * rho_factor)) * fast_rcp(2.0 * rho_factor);
    return (rho_factor >= 0) ? log(X) : 0.0;
}

__device__ __forceinline__ double saleh_log_X(double delta, double v, double rho_s, double half, double rho_linker,
                                              const UnLogEntry *tab) {
    const double rho_factor = delta * (v * rho_s + half * rho_linker);
    // the exponent also bounds 4 rho_factor below 2^60
    if(tab == nullptr || !un_takes(rho_factor) || rho_factor >= 0x1p57) return saleh_log_X_fp(rho_factor);
    const double t = 4.0 * rho_factor;
    Un X;
    if(!un_X((uint64_t) __double_as_longlong(1.0 + t), un_of(t), X)) return saleh_log_X_fp(rho_factor);
    return (double) un_log_tab(X, tab) * UNLOG_UNIT;
}

// f'(rho) of all S species of one cell: r[s] in, d[s] out.
template <int KIND>
__device__ __forceinline__ void der_bulk(const ModelDev &m, const double *r, double *d);

// src/models/Landau.cpp:46-53: f' = -eps psi + psi^3
template <>
__device__ __forceinline__ void der_bulk<CHGB_MODEL_LANDAU>(const ModelDev &m, const double *r, double *d) {
    double op = r[0];
    d[0] = op * fma(op, op, -m.epsilon);   // two FP64 instructions, two roundings
}

// f' of a simple_wertheim cell (src/models/SimpleWertheim.cpp:40-53) and rho
// X^v, which the free-energy mobility takes (:104-111).
struct SwCell {
    double der, rhoXv;
};

// The cell in integers (wertheim_fx.cuh) where the path takes the density: 5 FP64
// instructions instead of 40.  log(rho) + valence log(X) as one logarithm,
// log(rho X^valence); BELOW the regularisation log(X) alone.
template <bool BELOW>
__device__ __forceinline__ bool sw_cell_fx(const ModelDev &m, double rho, SwCell &c) {
    const double t = m.four_valence_delta * rho;
    Un X;
    if(!un_takes(t) || t >= 0x1p59 || !un_X((uint64_t) __double_as_longlong(1.0 + t), un_of(t), X)) return false;
    const Un P = un_mul(un_of(rho), un_pow(X, m.ivalence));
    if(P.e < -1000) return false;
    c.rhoXv = __longlong_as_double((long long) un_to_bits(P));
    if constexpr(BELOW)
        c.der = fma((double) un_log_tab(X, m.logtab), m.valence * UNLOG_UNIT, fma(m.reg_slope, rho, m.reg_base));
    else c.der = fma((double) un_log_tab(P, m.logtab), UNLOG_UNIT, m.two_B2 * rho);
    return true;
}

// Cells below the regularisation and those in FP64, out of the others' way: with
// the ones below in the inlined path, as operands selected, a 3D N=128
// euler_mobility step that has none took 75.8 us instead of 72.2.  In FP64 they
// made `euler` boxes slower than FP64 for every cell did: 2D N=32 with half of
// them below 7.1 -> 8.4 us a step, here 5.9; N=1024 with all below 135 -> 148,
// here 31.
__device__ __noinline__ static SwCell sw_cell_other(const ModelDev &m, double rho) {
    SwCell c;
    if(m.sw_fx && m.logtab != nullptr && un_takes(rho) && rho < m.reg_delta && sw_cell_fx<true>(m, rho, c)) return c;
    const double X = sw_X(m, rho);
    c.rhoXv = rho * ipow(X, m.ivalence);
    c.der = m.two_B2 * rho;
    if(rho < m.reg_delta) {
        c.der += m.log_delta + (rho - m.reg_delta) / m.reg_delta;
        c.der += (rho > 0.) ? m.valence * log(X) : 0.0;
    }
    else c.der += log(c.rhoXv);
    return c;
}

__device__ __forceinline__ SwCell sw_cell(const ModelDev &m, double rho) {
    SwCell c;
    if(!m.sw_fx || m.logtab == nullptr || !un_takes(rho) ||
       __double_as_longlong(rho) < __double_as_longlong(m.reg_delta) || !sw_cell_fx<false>(m, rho, c))
        return sw_cell_other(m, rho);
    return c;
}

// src/models/SimpleWertheim.cpp:40-53
template <>
__device__ __forceinline__ void der_bulk<CHGB_MODEL_SIMPLE_WERTHEIM>(const ModelDev &m, const double *r, double *d) {
    d[0] = sw_cell(m, r[0]).der;
}

// src/models/SalehWertheim.cpp:87-109.  A species whose density is exactly
// zero gets f' = 0 (the reference leaves the previous scratch value there).
template <>
__device__ __forceinline__ void der_bulk<CHGB_MODEL_SALEH>(const ModelDev &m, const double *r, double *d) {
    double rho_tot = ((0. + r[0]) + r[1]) + r[2];
    double b2 = m.two_B2 * rho_tot;
    double b3 = 3.0 * m.B3 * (rho_tot * rho_tot);
    double lx0 = saleh_log_X(m.dAA, m.sv0, r[0], m.half, r[2], m.logtab);
    double lx1 = saleh_log_X(m.dBB, m.sv1, r[1], m.half, r[2], m.logtab);
    d[0] = (r[0] != 0.) ? ((fx_log(r[0], m.logtab) + b2) + b3) + m.sv0 * lx0 : 0.0;
    d[1] = (r[1] != 0.) ? ((fx_log(r[1], m.logtab) + b2) + b3) + m.sv1 * lx1 : 0.0;
    d[2] = (r[2] != 0.) ? ((fx_log(r[2], m.logtab) + b2) + b3) + m.half * (lx0 + lx1) : 0.0;
}

// Free-energy mobility M0 * rho * X^valence, src/models/SimpleWertheim.cpp:104-111.
__device__ __forceinline__ double sw_mobility(const ModelDev &m, double M0, double rho) {
    return M0 * sw_cell(m, rho).rhoXv;
}

// Bulk free-energy density f(rho) of one cell (r[s] for all species).
template <int KIND>
__device__ __forceinline__ double bulk_fe(const ModelDev &m, const double *r);

// src/models/Landau.cpp:55-58
template <>
__device__ __forceinline__ double bulk_fe<CHGB_MODEL_LANDAU>(const ModelDev &m, const double *r) {
    double op = r[0];
    return -0.5 * m.epsilon * (op * op) + 0.25 * ((op * op) * (op * op));
}

// src/models/SimpleWertheim.cpp:71-86
template <>
__device__ __forceinline__ double bulk_fe<CHGB_MODEL_SIMPLE_WERTHEIM>(const ModelDev &m, const double *r) {
    double rho = r[0];
    double reg = m.reg_delta;
    double f_ref = m.B2 * (rho * rho);
    if(rho < reg) {
        double a = 1 / (2.0 * reg);
        double b = m.log_delta - 1.0;
        double c = reg * (m.log_delta - 1.0) - a * (reg * reg) - b * reg;
        f_ref += a * (rho * rho) + b * rho + c;
    }
    else {
        f_ref += rho * (log(rho * m.dcf) - 1.0);
    }
    double f_bond = 0.0;
    if(rho > 0.) {
        double X = sw_X(m, rho);
        f_bond = m.valence * rho * (log(X) + 0.5 * (1. - X));
    }
    return f_ref + f_bond;
}

// src/models/SalehWertheim.cpp:47-78
template <>
__device__ __forceinline__ double bulk_fe<CHGB_MODEL_SALEH>(const ModelDev &m, const double *r) {
    double rho = ((0. + r[0]) + r[1]) + r[2];
    double mixing_S = 0.;
    for(int i = 0; i < 3; i++) {
        double x_i = r[i] / rho;
        mixing_S += (x_i > 0) ? x_i * log(x_i) : 0;
    }
    double B2_contrib = m.B2 * rho;
    double B3_contrib = 0.5 * m.B3 * (rho * rho);
    double f_ref = rho * (log(rho * m.dcf) - 1.0 + mixing_S + B2_contrib + B3_contrib);

    double rf = m.dAA * (m.sv0 * r[0] + m.half * r[2]);
    double X_1A = (-1.0 + sqrt(1.0 + 4.0 * rf)) / (2.0 * rf);
    double fe1 = log(X_1A) - X_1A / 2.0 + 0.5;
    rf = m.dBB * (m.sv1 * r[1] + m.half * r[2]);
    double X_2B = (-1.0 + sqrt(1.0 + 4.0 * rf)) / (2.0 * rf);
    double fe2 = log(X_2B) - X_2B / 2.0 + 0.5;
    double bonding = r[0] * m.sv0 * fe1 + r[1] * m.sv1 * fe2 + r[2] * m.half * (fe1 + fe2);
    return f_ref + bonding;
}

// Programmatic dependent launch: wait for the stream's previous kernel (its
// writes have landed), then let the next kernel's CTAs be placed on the SMs
// this grid no longer needs.  Without the launch attribute the wait returns at
// once.
__device__ __forceinline__ void pdl_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}

struct KArr {
    double v[CHGB_MAX_SPECIES];
};

template <int KIND>
struct NSpecies {
    static constexpr int value = (KIND == CHGB_MODEL_SALEH) ? 3 : 1;
};

}  // namespace chgb
