"""The Wertheim models' integer square root, reciprocal, power and logarithm
(csrc/wertheim_fx.cuh), compiled for the host and run against extended
precision: the square root correctly rounded, X within 2^-58 of the
reference's expression with the same roundings, rho X^4 within 2^-56, the
logarithm within 2 2^-53 -- with the hardware's single-precision estimates
off by up to two units either way, at the ends of a binade and across 33
decades of t."""
import shutil
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parent.parent
SOURCE = r"""
#include "wertheim_fx.cuh"
#include <cstdio>
#include <cstdlib>
namespace chgb { int fx_est_ulps = 0; }
using namespace chgb;
typedef long double LD;   // 64 bits of mantissa at least
static UnLogEntry T[UNLOG_N];
struct Tab { void operator()(int j, uint32_t &i, int64_t &l) const { i = T[j].inv; l = T[j].ln; } };
static LD val(Un a) { return ldexpl((LD) a.m, a.e - 63); }
static uint64_t bits(double x) { uint64_t b; std::memcpy(&b, &x, 8); return b; }
static double dbl(uint64_t b) { double x; std::memcpy(&x, &b, 8); return x; }
int main(int argc, char **argv) {
    for(int j = 0; j < UNLOG_N; j++) {
        T[j].inv = (uint32_t) llround(2147483648.0 / (1.0 + (j + 0.5) / UNLOG_N));
        T[j].ln = (int64_t) llround(-logl((LD) T[j].inv / 2147483648.0L) * 1152921504606846976.0L);
    }
    fx_est_ulps = atoi(argv[1]);
    srand48(7);
    long wrong = 0;
    LD eX = 0, eP = 0, eL = 0, eB = 0;
    for(int i = 0; i < 300000; i++) {
        double t = ldexp(1.0 + drand48(), (int) (drand48() * 108) - 50), a = 1.0 + t;
        if(i < 500) a = (i & 1 ? 1.0 : 2.0) + ldexp(i, -52), t = a - 1.0;
        else if(i < 1000) a = (i & 1 ? 4.0 : 2.0) - ldexp(i - 499, -51), t = a - 1.0;
        int k;
        if(a < 1.0 + 0x1p-51) continue;
        const double y = (double) un_sqrt(bits(a), k);
        if(ldexp(y, k - 52) != sqrt(a)) wrong++;
        Un X;
        if(!un_X(bits(a), un_from_bits(bits(t)), X)) { wrong++; continue; }
        const LD x = ((LD) sqrt(a) - 1.0L) / ((LD) t / 2);
        eX = fmaxl(eX, fabsl(val(X) / x - 1));
        const double rho = ldexp(1.0 + drand48(), (int) (drand48() * 120) - 100);
        const Un P = un_mul(un_from_bits(bits(rho)), un_pow(X, 4));
        const LD p = (LD) rho * (x * x) * (x * x);
        eP = fmaxl(eP, fabsl(val(P) / p - 1));
        eB = fmaxl(eB, fabsl((LD) dbl(un_to_bits(P)) / val(P) - 1));
        eL = fmaxl(eL, fabsl((LD) un_log(P, Tab()) - ldexpl(logl(val(P)), 53)));
    }
    printf("%ld %.4Lg %.4Lg %.4Lg %.4Lg\n", wrong, eX * 0x1p58L, eP * 0x1p56L, eB * 0x1p53L, eL);
}
"""


@pytest.mark.parametrize("ulps", [-2, -1, 0, 1, 2])
def test_against_extended_precision(tmp_path_factory, ulps):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("wfx")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-x", "c++", "-I", str(REPO / "cahn-hilliard_gb300" / "csrc"),
                    str(d / "t.cpp"), "-o", str(d / "t")], check=True)
    out = subprocess.run([str(d / "t"), str(ulps)], capture_output=True, text=True, check=True).stdout.split()
    wrong, X, P, B, L = int(out[0]), *map(float, out[1:])
    assert wrong == 0
    assert X <= 1.0 and P <= 1.0 and B <= 1.0 and L <= 2.0
