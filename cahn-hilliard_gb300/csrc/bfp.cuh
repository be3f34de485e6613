// bfp.cuh — block floating point for the pseudospectral FFTs: 64-bit integer
// arithmetic with one exponent per transform line.
//
// On GB300 the FP64 pipe issues at 1/64 of the FP32 rate, while 32-bit
// integer multiply-adds (IMAD.WIDE, 64 lanes a clock and SM, measured) and
// 64-bit adds on the integer ALU run tens of times faster.  An FFT butterfly
// is additions and twiddle products, so the transforms run in fixed point:
//
//   * A line (one row or column being transformed) of FP64 values is scaled
//     by one power of two 2^sh, chosen from the largest exponent field in the
//     line, so that every value the transform can produce keeps its complex
//     magnitude below 2^62: a length-L DFT grows magnitudes by at most L, the
//     real-transform pre/post-processing by at most 4, and a complex value's
//     magnitude is at most sqrt(2) times its largest component.  The largest
//     input component therefore keeps 62 - G bits, G = log2 L + 1 (column
//     transforms) or log2 L + 3 (the real-row transforms), 49 to 51 bits for
//     the boxes of the benchmark.  Values go in by integer operations (round
//     to nearest, ties away from zero) and come out through the FP64 pipe's int64 ->
//     double conversion (round to nearest even), that pipe's only work in a
//     transform.
//   * Additions are exact.  A twiddle w is stored as W = round(w 2^62), split
//     into signed 32-bit limbs W = h 2^32 + l, as each factor X is (its low
//     limb is its low word, its high limb one instruction), so a component of
//     a complex product is two 32 x 32 -> 64-bit products of high limbs, four
//     cross products and one rounding, accumulated by IMAD.WIDE with no
//     additions of their own.  The products of two low limbs are left out:
//     each is at most one unit of the result in magnitude and of either sign.
//     Per component the error is one rounding and two such terms, a root mean
//     square of 0.55 units of 2^-62 against 0.29 units of 2^-61 for exact
//     31-bit limbs in a 2^61 range.  Whole 1024-point transforms of random
//     lines: relative rms error 2.7e-16 against 4.8e-16 (CPU model against
//     113-bit arithmetic); with the low products 2.5e-16.
//   * A line holding a NaN or an infinity yields NaN for the whole line, as a
//     floating-point transform would.
//
// Bounds that keep every 64-bit intermediate in range, with |X| < 2^62 for
// every complex magnitude: high limbs are at most 2^30 in magnitude, low limbs
// 2^31, so a component's cross products stay below (2 sqrt(2) + 4) 2^60 <
// 2^63, and its high products below 2^61 (4 times that is the result, < 2^62).
#pragma once

#include <cuda_runtime.h>

namespace chgb {

// A complex value of a line in fixed point; same size and alignment as double2.
struct __align__(16) fx2 {
    long long x, y;
};

constexpr int FX_TOP = 62;   // every complex magnitude stays below 2^FX_TOP

// v = fx_hi(v) 2^32 + fx_lo(v), both signed.
__device__ __forceinline__ int fx_hi(long long v) { return (int) (v >> 32) + (int) ((unsigned) v >> 31); }
__device__ __forceinline__ int fx_lo(long long v) { return (int) v; }
// a b and a b + c, one IMAD.WIDE each.  In C++ a product of sign-extended low
// words, (long long) (int) v * ..., is compiled as a full 64-bit product, five
// instructions.
__device__ __forceinline__ long long wide(int a, int b) {
    long long r;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ long long wide(int a, int b, long long c) {
    long long r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}

// a w / 2^62 (CONJ = false) or a conj(w) / 2^62 (CONJ = true), rounded;
// w = {hx, lx, hy, ly}, the limbs of the twiddle's real and imaginary parts
// (no limb is -2^31, so the negations are exact).
template <bool CONJ>
__device__ __forceinline__ fx2 fx_cmul(fx2 a, int4 w) {
    const int xh = fx_hi(a.x), xl = fx_lo(a.x), yh = fx_hi(a.y), yl = fx_lo(a.y);
    const int nz = -w.z, nw = -w.w;
    const int rz = CONJ ? w.z : nz, rw = CONJ ? w.w : nw;   // Y's factor in the real part
    const int iz = CONJ ? nz : w.z, iw = CONJ ? nw : w.w;   // X's factor in the imaginary part
    const long long half = 1ll << 29;
    const long long hx = wide(xh, w.x, wide(yh, rz));
    const long long mx = wide(xh, w.y, wide(xl, w.x, wide(yh, rw, wide(yl, rz, half))));
    const long long hy = wide(yh, w.x, wide(xh, iz));
    const long long my = wide(yh, w.y, wide(yl, w.x, wide(xh, iw, wide(xl, iz, half))));
    return fx2{4 * hx + (mx >> 30), 4 * hy + (my >> 30)};
}

// X / sqrt(2), rounded the same way.
__device__ __forceinline__ long long fx_mul_sqrt_half(long long X) {
    constexpr long long C = 3260954456333195553ll;   // round(2^62 / sqrt(2))
    constexpr int Cl = (int) (C & 0xFFFFFFFFll), Ch = (int) ((C - Cl) >> 32);
    const int xh = fx_hi(X), xl = fx_lo(X);
    const long long mid = wide(xh, Cl, wide(xl, Ch, 1ll << 29));
    return 4 * wide(xh, Ch) + (mid >> 30);
}

__device__ __forceinline__ fx2 fx_add(fx2 a, fx2 b) { return fx2{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ fx2 fx_sub(fx2 a, fx2 b) { return fx2{a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ fx2 fx_swap(fx2 a) { return fx2{a.y, a.x}; }

// Forward 4-point DFT of (a, b, c, d) in place, in order.
__device__ __forceinline__ void fx_dft4(fx2 &a, fx2 &b, fx2 &c, fx2 &d) {
    const fx2 s0 = fx_add(a, c), d0 = fx_sub(a, c), s1 = fx_add(b, d), d1 = fx_sub(b, d);
    a = fx_add(s0, s1);
    c = fx_sub(s0, s1);
    b = fx2{d0.x + d1.y, d0.y - d1.x};
    d = fx2{d0.x - d1.y, d0.y + d1.x};
}

// Forward 8-point DFT in place, in order: two 4-point DFTs, the odd one's
// inputs turned by the eighth roots of unity (four products by 1/sqrt(2)).
__device__ __forceinline__ void fx_dft8(fx2 (&v)[8]) {
    fx2 e0 = fx_add(v[0], v[4]), e1 = fx_add(v[1], v[5]), e2 = fx_add(v[2], v[6]), e3 = fx_add(v[3], v[7]);
    fx2 o0 = fx_sub(v[0], v[4]), o1 = fx_sub(v[1], v[5]), o2 = fx_sub(v[2], v[6]), o3 = fx_sub(v[3], v[7]);
    o1 = fx2{fx_mul_sqrt_half(o1.x + o1.y), fx_mul_sqrt_half(o1.y - o1.x)};
    o2 = fx2{o2.y, -o2.x};
    o3 = fx2{fx_mul_sqrt_half(o3.y - o3.x), fx_mul_sqrt_half(-(o3.x + o3.y))};
    fx_dft4(e0, e1, e2, e3);
    fx_dft4(o0, o1, o2, o3);
    v[0] = e0;
    v[2] = e1;
    v[4] = e2;
    v[6] = e3;
    v[1] = o0;
    v[3] = o1;
    v[5] = o2;
    v[7] = o3;
}

// The high word of |v|: its exponent field and leading mantissa bits, ordered as |v|.
__device__ __forceinline__ int fx_mag(double v) { return __double2hiint(v) & 0x7FFFFFFF; }

// The scale of a line whose largest value has the high word `mag`, for
// headroom G: the largest component stays below 2^(FX_TOP - G) after
// multiplying by 2^sh (a value with exponent field e is below 2^(e - 1022)).
// Lines near either end of the double range (`odd`) are multiplied by a power
// of two, pre^3, before fx_in and by its inverse post^3 after fx_out, which
// keeps the conversions free of special cases; the line of a NaN or an
// infinity has post = NaN.
struct FxScale {
    int sh;
    bool odd;
    double pre, post;
};
__device__ __forceinline__ FxScale fx_line_scale(int mag, int G) {
    int e = mag >> 20;
    FxScale s;
    s.odd = (unsigned) (e - 128) > 1984u - 128u;
    s.pre = s.post = 1.0;
    if(s.odd) {
        const int k = e < 128 ? 200 : -200;
        s.pre = __hiloint2double((1023 + k) << 20, 0);
        s.post = e == 2047 ? __hiloint2double(0x7FF80000, 0) : __hiloint2double((1023 - k) << 20, 0);
        e = (e < 1 ? 1 : e) + 3 * k;
    }
    s.sh = FX_TOP - G + 1022 - e;
    return s;
}

// a >> t, 0 for t >= 64 (PTX clamps the shift).
__device__ __forceinline__ unsigned long long fx_shr(unsigned long long a, int t) {
    unsigned long long r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(a), "r"(t));
    return r;
}

// round(v 2^sh) to nearest (ties away from zero), 0 for zeros and what
// underflows.  The 53-bit mantissa sits at the top of a word and moves right by
// at least 3, one bit short of its place: the last bit is the rounding's.
__device__ __forceinline__ long long fx_in(double v, const FxScale &s) {
    const int hi = __double2hiint(v);
    const unsigned lo = (unsigned) __double2loint(v);
    const int t = 1085 - s.sh - ((hi >> 20) & 0x7FF);
    const unsigned mh = __funnelshift_l(lo, (unsigned) hi, 11) | 0x80000000u;
    const unsigned long long m = fx_shr(((unsigned long long) mh << 32) | (lo << 11), t);
    const long long sg = (long long) (hi >> 31);
    return (long long) (((m + 1) >> 1) ^ (unsigned long long) sg) - sg;
}
__device__ __forceinline__ fx2 fx_in(double2 v, const FxScale &s) { return fx2{fx_in(v.x, s), fx_in(v.y, s)}; }

// X 2^-sh as the nearest double, ties to even: on the FP64 pipe (x) or, the
// same value, in integers (y).  A warp's int64 -> double conversion holds that
// pipe for 64 cycles of its scheduler; the twenty integer instructions take 40
// of the integer ALU's, so a complex value takes one of each.
__device__ __forceinline__ double fx_out_fp(long long X, const FxScale &s) {
    const double d = __ll2double_rn(X);
    return X == 0 ? 0.0 : __hiloint2double(__double2hiint(d) - (s.sh << 20), __double2loint(d));
}
__device__ __forceinline__ double fx_nearest(long long X, int sh) {   // |X| < 2^63, a normal result
    const long long sg = X >> 63;
    const unsigned long long a = (unsigned long long) ((X ^ sg) - sg);
    const int lz = __clzll((long long) a);                     // 1 or more; 64 for 0
    const unsigned long long m = a << ((lz - 1) & 63);         // leading one at bit 62
    const unsigned long long q = (m + 0x1FF + ((m >> 10) & 1)) >> 10;   // 53 bits, or 2^53
    // the leading one adds 1 to the exponent field below it, a carry out of the mantissa 2
    const unsigned long long bits = ((unsigned long long) (unsigned) (1085 - lz - sh) << 52) + q;
    const unsigned long long r = X == 0 ? 0ull : bits | ((unsigned long long) sg << 63);
    return __longlong_as_double((long long) r);
}
__device__ __forceinline__ double2 fx_out(fx2 v, const FxScale &s) {
    return make_double2(fx_out_fp(v.x, s), fx_nearest(v.y, s.sh));
}

// v times f^3 where the line is `odd`.  The three products a value make the
// body long enough to be branched around: as one product each it was
// predicated, and predicated-off FP64 instructions hold that pipe all the same
// (3 of the row pass's 6 FP64 instructions a cell, ncu on GB300).
template <int E>
__device__ __forceinline__ void fx_scale_by(double2 (&v)[E], bool odd, double f) {
    if(odd) {
#pragma unroll
        for(int i = 0; i < E; i++) v[i] = make_double2(v[i].x * f * f * f, v[i].y * f * f * f);
    }
}

// ---------------------------------------------------------------------------
// One line's forward Stockham FFT of length 2^lg on T = max(1, 2^lg / E)
// threads, E = 2, 4 or 8 values a thread: v[i] is position lane + i T, on the way
// in and on the way out (2^lg < E: the first 2^lg entries).  The inverse
// transform is the same with real and imaginary parts swapped on both ways.
//
// E = 2: radix 2.  E = 4: radix 4, after one radix-2 pass (two butterflies a
// thread) where lg is odd.  E = 8: radix 8, with one radix-4 pass (two butterflies) where lg is 2
// modulo 3 and two where it is 1.  Values stay in registers; between two passes
// they cross through shared memory, which the line's loads and stores do not
// touch.  The boxes' lines are of 64 values and more with E = 4 and of 1024 and more
// with E = 8 (fx_line_elems, spectral.cu).  The tests for shorter ones stay: without
// them the compiler takes 128 registers for the rows with E = 8 instead of 100 (2D
// N = 2048 197.9 -> 201.6 us a step).
//
// The lines of a CTA lie in groups of C = 2^lgC interleaved lines (adjacent
// columns: a warp's loads then take whole sectors): element p of line c is at
// (p + p / 8) C + c of the group's buffer -- one element of padding in eight
// keeps the first pass's strided stores off one bank (lines shorter than 64
// are not padded).  `cur` and `oth` are two such buffers: an exchange writes
// cur, synchronises, reads it and swaps the two, so that one barrier an
// exchange is enough.
// ---------------------------------------------------------------------------
struct FxLine {
    int lg, lgC;     // log2 of the length and of the interleaved lines
    int T, lane, c;  // threads of the line, this thread's index among them, the line's index in its group
    unsigned warp_mask;   // the warp's threads, where the group lies in one warp: its barriers are warp barriers; else 0
    __device__ __forceinline__ bool pad() const { return lg >= 6; }
    // index of element p, and the distance of elements n apart (n and, when padded, their positions' remainders
    // modulo 8 such that no carry crosses: n a multiple of 8)
    __device__ __forceinline__ int at(int p) const { return ((p + (pad() ? p >> 3 : 0)) << lgC) + c; }
    __device__ __forceinline__ int step(int n) const { return (n + (pad() ? n >> 3 : 0)) << lgC; }
    __device__ __forceinline__ void sync() const {
        if(warp_mask) __syncwarp(warp_mask);
        else __syncthreads();
    }
};

// Elements of one line in a buffer.
__host__ __device__ __forceinline__ int fx_line_size(int L) { return L + (L >= 64 ? L >> 3 : 0); }

__device__ __forceinline__ void fx_swap_buf(fx2 *&a, fx2 *&b) {
    fx2 *t = a;
    a = b;
    b = t;
}

// tw[q] = exp(-2 pi i q / 2^lgtab), lgtab >= lg.
template <int E>
__device__ __forceinline__ void fx_fft(fx2 (&v)[E], const FxLine &ln, fx2 *&cur, fx2 *&oth,
                                       const int4 *__restrict__ tw, int lgtab) {
    const int lg = ln.lg, lane = ln.lane;
    if(lg < (E == 8 ? 3 : E == 4 ? 2 : 1)) {   // one thread per line
        if(E == 2) return;
        if(E == 8 && lg == 2) fx_dft4(v[0], v[1], v[2], v[3]);
        else {
            const fx2 s = fx_add(v[0], v[1]);
            v[1] = fx_sub(v[0], v[1]);
            v[0] = s;
        }
        return;
    }
    const int g0 = ln.at(lane), gs = ln.step(ln.T);
    int ns = 0;
    // the first pass: no twiddles
    if constexpr(E == 8) {
        if(lg != 4) {
            fx_dft8(v);
            ns = 3;
            if(lg > 3) {
                const int o = ln.at(lane << 3);
#pragma unroll
                for(int m = 0; m < 8; m++) cur[o + (m << ln.lgC)] = v[m];
            }
        }
    }
    else if(E == 2) {
        const fx2 s = fx_add(v[0], v[1]);
        v[1] = fx_sub(v[0], v[1]);
        v[0] = s;
        ns = 1;
        if(lg > 1) {
            const int o = ln.at(lane << 1);
            cur[o] = v[0];
            cur[o + (1 << ln.lgC)] = v[1];
        }
    }
    else if(lg & 1) {
        ns = 1;
#pragma unroll
        for(int b = 0; b < 2; b++) {
            const fx2 s = fx_add(v[b], v[b + 2]), d = fx_sub(v[b], v[b + 2]);
            const int o = ln.at((lane + b * ln.T) << 1);
            cur[o] = s;
            cur[o + (1 << ln.lgC)] = d;
        }
    }
    else {
        fx_dft4(v[0], v[1], v[2], v[3]);
        ns = 2;
        if(lg > 2) {
            const int o = ln.at(lane << 2);
#pragma unroll
            for(int m = 0; m < 4; m++) cur[o + (m << ln.lgC)] = v[m];
        }
    }
    while(ns < lg) {
        const int left = lg - ns;
        if(ns > 0) {
            ln.sync();
#pragma unroll
            for(int i = 0; i < E; i++) v[i] = cur[g0 + i * gs];
            fx_swap_buf(cur, oth);
        }
        if constexpr(E == 8) {
            if(left >= 3 && left != 4) {
                const int k = lane & ((1 << ns) - 1);
                const int q = k << (lgtab - ns - 3);
#pragma unroll
                for(int m = 1; m < 8; m++) v[m] = fx_cmul<false>(v[m], __ldg(&tw[m * q]));
                fx_dft8(v);
                if(left > 3) {
                    const int o = ln.at(((lane - k) << 3) + k), os = ln.step(1 << ns);
#pragma unroll
                    for(int m = 0; m < 8; m++) cur[o + m * os] = v[m];
                }
                ns += 3;
                continue;
            }
        }
        if constexpr(E == 2) {
            const int k = lane & ((1 << ns) - 1);
            const fx2 t = fx_cmul<false>(v[1], __ldg(&tw[k << (lgtab - ns - 1)])), s = fx_add(v[0], t);
            v[1] = fx_sub(v[0], t);
            v[0] = s;
            if(left > 1) {
                const int p = ((lane - k) << 1) + k;
                cur[ln.at(p)] = v[0];
                cur[ln.at(p + (1 << ns))] = v[1];
            }
            ns += 1;
            continue;
        }
        constexpr int B = E >= 4 ? E / 4 : 1;   // butterflies a thread
#pragma unroll
        for(int b = 0; b < (E >= 4 ? B : 0); b++) {
            const int j = lane + b * ln.T;
            const int k = j & ((1 << ns) - 1);
            const int q = k << (lgtab - ns - 2);
#pragma unroll
            for(int m = 1; m < 4; m++) v[b + B * m] = fx_cmul<false>(v[b + B * m], __ldg(&tw[m * q]));
            fx_dft4(v[b], v[b + B], v[b + 2 * B], v[b + 3 * B]);
            if(left > 2) {
                const int p = ((j - k) << 2) + k;
                if(E == 4 && ns < 3) {
#pragma unroll
                    for(int m = 0; m < 4; m++) cur[ln.at(p + (m << ns))] = v[b + B * m];
                }
                else {
                    const int o = ln.at(p), os = ln.step(1 << ns);
#pragma unroll
                    for(int m = 0; m < 4; m++) cur[o + m * os] = v[b + B * m];
                }
            }
        }
        ns += 2;
    }
}

// Maximum of `e` over the threads of each line: groups of W = T C consecutive
// threads (powers of two) with the C lines interleaved.  sm_w holds one int
// per warp and interleaved line.  Every thread of the block calls it.
__device__ __forceinline__ int fx_line_max(int e, int C, int W, int *sm_w) {
    const int nthr = blockDim.x;
    const int wbase = threadIdx.x & ~31;
    const unsigned mask = (nthr - wbase >= 32) ? 0xffffffffu : ((1u << (nthr - wbase)) - 1u);
    if(C == 1 && W >= 32) e = __reduce_max_sync(mask, e);
    else
        for(int o = C; o < 32 && o < W; o <<= 1) e = max(e, __shfl_xor_sync(mask, e, o));
    if(W > 32) {
        const int c = threadIdx.x & (C - 1), nw = W >> 5, w0 = (threadIdx.x >> 5) & ~(nw - 1);
        if((int) (threadIdx.x & 31) < C) sm_w[(threadIdx.x >> 5) * C + c] = e;
        __syncthreads();
        e = sm_w[w0 * C + c];
        for(int w = 1; w < nw; w++) e = max(e, sm_w[(w0 + w) * C + c]);
    }
    return e;
}

}  // namespace chgb
