// wertheim_fx.cuh — X, X^v, logarithms and their products for the Wertheim
// models, and the gel mobility's exponential, in 64-bit integers (device code;
// also compiles on the host, where the CPU tests run it against extended
// precision).
//
// On GB300 an FP64 instruction takes the pipe time of 32 integer-ALU ones, and a
// simple_wertheim cell took 51 of them for mu (a square root, a reciprocal, a
// power, a logarithm).  Here those four run on mantissas: a positive value is
// m 2^(e-63) with m's leading one at bit 63 (Un).  Products keep the upper word
// of 64 x 64 bits from three 32 x 32 -> 64-bit ones (IMAD.WIDE); the square
// root and the reciprocal start from the hardware's single-precision estimates
// (relative error below 2^-20.5 is enough) and take one correction of third
// order, whose residual is formed exactly enough in integers; the logarithm is
// table-driven after P. T. P. Tang (ACM TOMS 16 (1990)), with 256 entries whose
// reciprocals have 32 bits, so that r = y / c_j - 1 is one product.  Floors
// throughout: the errors below are one-sided, a few units each.
//   un_mul    relative 3 2^-63
//   un_rcp    relative 2^-59
//   un_sqrt   correctly rounded to double
//   un_X      relative 2^-58 of (-1 + sqrt(1 + t)) / (t / 2) with the sum and
//             the square root rounded to double
//   un_log    absolute 1.1 2^-53, and |log2 a| 2^-64 of ln 2's last place
//   un_expneg relative 2^-58 + t 2^-61.5
// Measured, 3D N=128 euler_mobility: the mu kernel 180 -> 59 us (FP64 pipe 64 %
// busy from the interface's conversions and sums), a step 265 -> 116 us.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define CHGB_FX __device__ __forceinline__
#else
#include <cmath>
#include <cstring>
#define CHGB_FX inline
#endif

namespace chgb {

#ifdef __CUDACC__
CHGB_FX uint64_t fxw(uint32_t a, uint32_t b) {
    uint64_t r;
    asm("mul.wide.u32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
CHGB_FX int64_t fxws(int32_t a, int32_t b) {
    int64_t r;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
// a >> n for any n >= 0 (PTX clamps the shift)
CHGB_FX uint64_t fx_down(uint64_t a, int n) {
    uint64_t r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(a), "r"(n));
    return r;
}
CHGB_FX uint32_t fx_est_rsqrt(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return __float_as_uint(r);
}
CHGB_FX uint32_t fx_est_rcp(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return __float_as_uint(r);
}
CHGB_FX int fx_lead(uint32_t hi) { return __clz((int) hi); }
#else
CHGB_FX uint64_t fxw(uint32_t a, uint32_t b) { return (uint64_t) a * b; }
CHGB_FX int64_t fxws(int32_t a, int32_t b) { return (int64_t) a * b; }
CHGB_FX uint64_t fx_down(uint64_t a, int n) { return n > 63 ? 0 : a >> n; }
// the device's estimates are within 2 ulp; the test adds that error either way
extern int fx_est_ulps;
CHGB_FX uint32_t fx_est(float r) {
    uint32_t u;
    std::memcpy(&u, &r, sizeof u);
    return u + (uint32_t) fx_est_ulps;
}
CHGB_FX uint32_t fx_est_rsqrt(float x) { return fx_est((float) (1.0 / std::sqrt((double) x))); }
CHGB_FX uint32_t fx_est_rcp(float x) { return fx_est((float) (1.0 / (double) x)); }
CHGB_FX int fx_lead(uint32_t hi) { return __builtin_clz(hi); }
#endif

struct Un {
    uint64_t m;
    int e;
};

// Table of un_log: entry j holds inv = round(2^31 / c_j), c_j = 1 + (j + 1/2) /
// 256, and -ln(inv / 2^31) in units of 2^-60.
constexpr int UNLOG_N = 256;
struct UnLogEntry {
    uint32_t inv, pad;
    int64_t ln;
};

// A normal positive double's bits.
CHGB_FX Un un_from_bits(uint64_t b) {
    return Un{(1ull << 63) | (b << 11), (int) (b >> 52) - 1023};
}

// The nearest double's bits (ties up); the exponent has to stay normal.
CHGB_FX uint64_t un_to_bits(Un a) { return ((uint64_t) (uint32_t) (a.e + 1022) << 52) + ((a.m >> 11) + ((a.m >> 10) & 1)); }

// Upper word of a b, short of it by less than 3.
CHGB_FX uint64_t un_high(uint64_t a, uint64_t b) {
    const uint32_t ah = (uint32_t) (a >> 32), al = (uint32_t) a, bh = (uint32_t) (b >> 32), bl = (uint32_t) b;
    return fxw(ah, bh) + (fxw(ah, bl) >> 32) + (fxw(al, bh) >> 32);
}

CHGB_FX Un un_mul(Un a, Un b) {
    Un r{un_high(a.m, b.m), a.e + b.e + 1};
    if((int64_t) r.m >= 0) {
        r.m <<= 1;
        r.e--;
    }
    return r;
}

CHGB_FX Un un_pow(Un x, int n) {   // n >= 1
    while(!(n & 1)) {
        x = un_mul(x, x);
        n >>= 1;
    }
    Un r = x;
    while(n >>= 1) {
        x = un_mul(x, x);
        if(n & 1) r = un_mul(r, x);
    }
    return r;
}

// A float of [1/4, 2) in units of 2^-24.  The estimates of a value in (1/2, 1]
// may fall just outside.
CHGB_FX uint32_t fx_mant24(uint32_t b) { return (((b & 0x7FFFFFu) | 0x800000u) << 1) >> (127u - (b >> 23)); }

// 1 / x, short of it by less than 2^-59 relative.
CHGB_FX Un un_rcp(Un x) {
    const uint64_t D = x.m >> 1;   // tau = D / 2^62 in [1, 2)
    const uint32_t dh = (uint32_t) (D >> 32), dl = (uint32_t) D;
    const uint32_t vb = fx_est_rcp((float) dh * 9.3132257461547852e-10f);
    const uint32_t v = fx_mant24(vb);   // ~ 1 / tau in units of 2^-24
    // f = 1 - tau v in units of 2^-62, below 2^-20; 1 / tau = v (1 + f + f^2)
    const int64_t f = (int64_t) ((1ull << 62) - ((fxw(dh, v) << 8) + (fxw(dl, v) >> 24)));
    const int32_t fh = (int32_t) (f >> 12);
    const int64_t g = f + (fxws(fh, fh) >> 38);
    const uint64_t R = ((uint64_t) v << 37) + (uint64_t) (fxws((int32_t) v, (int32_t) (g >> 32)) << 7) +
                       (fxw(v, (uint32_t) g) >> 25);   // units of 2^-61
    const int s = fx_lead((uint32_t) (R >> 32));
    return Un{R << s, 2 - s - x.e};
}

// sqrt(a), correctly rounded (to nearest), of a double 1 <= a < 2^60 given by
// its bits: y = Y 2^(k-52), 2^52 <= Y < 2^53.
CHGB_FX int64_t un_sqrt(uint64_t abits, int &k) {
    const int ea = (int) (abits >> 52) - 1023, odd = ea & 1;
    k = ea >> 1;
    const uint64_t ma = ((abits & 0xFFFFFFFFFFFFFull) | (1ull << 52)) << odd;   // alpha = a / 2^2k = ma 2^-52 in [1, 4)
    const uint64_t A = ma << 10;                                               // in units of 2^-62
    const uint32_t ah = (uint32_t) (A >> 32), al = (uint32_t) A;
    const uint32_t wb = fx_est_rsqrt((float) ah * 9.3132257461547852e-10f);
    const uint32_t w = fx_mant24(wb) - 4u;   // ~ 1 / sqrt(alpha) in units of 2^-24, and below it: B < 2^63
    // e = 1 - alpha w^2 in units of 2^-62, below 2^-19
    const uint64_t w2 = fxw(w, w) << 14;
    const uint32_t w2h = (uint32_t) (w2 >> 32), w2l = (uint32_t) w2;
    const int64_t e = (int64_t) ((1ull << 62) - ((fxw(ah, w2h) << 2) + (fxw(ah, w2l) >> 30) + (fxw(al, w2h) >> 30)));
    // sqrt(alpha) = alpha w (1 - e)^(-1/2) = alpha w (1 + c), c = e / 2 + 3 e^2 / 8
    const int32_t eh = (int32_t) (e >> 12);
    const int64_t c = (e >> 1) + (int64_t) ((3u * (uint32_t) ((uint64_t) fxws(eh, eh) >> 32)) >> 9);
    const uint64_t B = (fxw(ah, w) << 8) + (fxw(al, w) >> 24);
    const int32_t ch = (int32_t) (c >> 32);
    const uint32_t bh = (uint32_t) (B >> 32);
    const uint64_t S = B + (uint64_t) (fxws((int32_t) bh, ch) << 2) + (fxw(bh, (uint32_t) c) >> 30) +
                       (uint64_t) (fxws((int32_t) ((uint32_t) B >> 1), ch) >> 29);
    // the nearest integer of units of 2^-52 up to one, then exactly: ma 2^52 - Y^2
    // (its low word is the whole difference) against Y, which is where the
    // square root lies halfway to the next
    const int64_t Y = (int64_t) ((S + 512) >> 10);
    const int64_t d = (int64_t) ((ma << 52) - (uint64_t) Y * (uint64_t) Y);
    return Y + (d > Y ? 1 : 0) - (d <= -Y ? 1 : 0);
}

// X = (-1 + sqrt(a)) / (t / 2) with a = 1 + t and the square root rounded to
// double, as the reference's FP64 expression rounds them: for small t their
// rounding, not the division's, is what X carries.  abits: the bits of a;
// t < 2^60.  Returns false where sqrt(a) = 1.
CHGB_FX bool un_X(uint64_t abits, Un t, Un &X) {
    int k;
    const int64_t y = un_sqrt(abits, k);                     // sets k, which the next line reads
    const int64_t z = y - (int64_t) ((1ull << 52) >> k);     // y - 1, exact
    if(z == 0) return false;
    const uint32_t zh = (uint32_t) ((uint64_t) z >> 32);
    const int s = zh ? fx_lead(zh) : 32 + fx_lead((uint32_t) z);
    t.e -= 1;
    X = un_mul(Un{(uint64_t) z << s, 11 - s + k}, un_rcp(t));
    return true;
}

// ln(a) in units of 2^-53.
template <typename Entry>
CHGB_FX int64_t un_log(Un a, Entry entry) {
    uint32_t inv;
    int64_t lnc;
    entry((int) (a.m >> 55) & (UNLOG_N - 1), inv, lnc);
    // r = y inv - 1 in units of 2^-62, |r| < 2^-9; r^2 in 2^-80, r^3 in 2^-58
    const int64_t r = (int64_t) (fxw((uint32_t) (a.m >> 32), inv) + (fxw((uint32_t) a.m, inv) >> 32) - (1ull << 62));
    const int32_t rh = (int32_t) (r >> 22), rl = (int32_t) r & 0x3FFFFF;
    const int64_t r2 = fxws(rh, rh) + (fxws(rh, rl) >> 21);
    const int32_t r2h = (int32_t) (r2 >> 31);
    const int32_t r3 = (int32_t) (fxws(r2h, rh) >> 31);
    // 1/3 - r/4 + r^2/5 in units of 2^-31
    const int32_t s = 715827883 - (rh >> 11) + ((r2h >> 10) * 205 >> 18);
    const int64_t p = (r >> 2) - (r2 >> 21) + (fxws(r3, s) >> 29);
    // e ln 2: ln 2 = 0x58B90BFC 2^-31 - 0x1718432A 2^-63
    return (int64_t) ((uint64_t) fxws(a.e, 0x58B90BFC) << 22) - (fxws(a.e, 0x1718432A) >> 10) + ((lnc + p) >> 7);
}

// e^(-c/c0) = 2^(-t), t = c K < 512 with K = 1 / (c0 ln 2): t = n + j / 256 +
// r, 2^(-j/256) from a table (units of 2^-63, UNEXP_N entries), 2^(-r) by its
// Taylor polynomial in w = r ln 2 < 2^-8.5 to w^5.
constexpr int UNEXP_N = 256;
template <typename Entry>
CHGB_FX Un un_expneg(Un c, Un K, Entry entry) {
    const Un t = un_mul(c, K);
    const int n = t.e < 0 ? 0 : (int) (t.m >> (63 - t.e));
    const uint64_t F = t.e < 0 ? fx_down(t.m, -1 - t.e) : t.m << (t.e + 1);   // the fraction, units of 2^-64
    const uint64_t q = entry((int) (F >> 56));
    const uint32_t rh = (uint32_t) (F >> 32) & 0xFFFFFFu, rl = (uint32_t) F;
    // w in units of 2^-62, w^2 in 2^-80, w^3 in 2^-57; ln 2 = 0xB17217F7 2^-32 + 0xD1CF79AC 2^-64
    const uint64_t w = (fxw(rh, 0xB17217F7u) >> 2) + (fxw(rh, 0xD1CF79ACu) >> 34) + (fxw(rl, 0xB17217F7u) >> 34);
    const uint32_t wh = (uint32_t) (w >> 22), wl = (uint32_t) w & 0x3FFFFFu;
    const uint64_t w2 = fxw(wh, wh) + (fxw(wh, wl) >> 21);
    const uint32_t w2h = (uint32_t) (w2 >> 31);
    const uint32_t w3 = (uint32_t) (fxw(w2h, wh) >> 32);
    // 1/6 - w/24 + w^2/120 in units of 2^-34
    const uint32_t s = 2863311531u - (wh >> 6) / 24u + (w2h >> 15) / 120u;
    const uint64_t p = (1ull << 62) - w + (w2 >> 19) - (fxw(w3, s) >> 29);
    const uint64_t h = un_high(q, p << 1);   // in (2^61, 2^62]
    const int z = fx_lead((uint32_t) (h >> 32));
    return Un{h << z, 1 - z - n};
}

}  // namespace chgb
