"""The gel mobility's exponential in integers (un_expneg, csrc/wertheim_fx.cuh).

On the CPU: compiled for the host against extended precision.  The polynomial,
its table and floors give 2^-58; the product t = c K has relative error below
4 2^-63 (K's and un_mul's), the reference's argument 2^-64, both times t ln 2
in the result.  On the GPU: the gel mobility against the oracle where each
branch is taken -- c/c0 past the integer range (the library's exp), within it,
and below the last place of 1."""
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
typedef long double LD;
static uint64_t T[UNEXP_N];
int main() {
    for(int j = 0; j < UNEXP_N; j++) T[j] = (uint64_t) (std::exp2(-(LD) j / UNEXP_N) * 9223372036854775808.0L + 0.5L);
    srand48(3);
    LD worst = 0;
    for(int i = 0; i < 400000; i++) {
        const double c0 = ldexp(0.5 + 0.5 * drand48(), (int) (drand48() * 40) - 20);
        const LD K = 1.0L / ((LD) c0 * logl(2.0L));
        int x;
        const LD f = frexpl(K, &x);
        const Un uK{(uint64_t) (f * 18446744073709551616.0L), x - 1};
        double c = c0 * ldexp(1.0 + drand48(), (int) (drand48() * 80) - 72);
        if(i < 2000) c = c0 * 0.6931471805599453 * (i / 8) * (1 + ldexp(i % 8 - 4, -52));   // t at and around whole numbers
        if(c <= 0) continue;
        uint64_t b;
        std::memcpy(&b, &c, 8);
        const Un u = un_from_bits(b);
        if(u.e + uK.e > 7) continue;
        const Un r = un_expneg(u, uK, [](int j) { return T[j]; });
        if(!(r.m >> 63)) { printf("inf\n"); return 0; }
        const LD a = (LD) c / c0, v = ldexpl((LD) r.m, r.e - 63);
        worst = fmaxl(worst, fabsl(v / expl(-a) - 1) / (0x1p-58L + a * 5 * 0x1p-63L));
    }
    printf("%.4Lg\n", worst);
}
"""


def test_against_extended_precision(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    (tmp_path / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-x", "c++", "-I", str(REPO / "cahn-hilliard_gb300" / "csrc"),
                    str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, check=True).stdout
    print(out)
    assert float(out) <= 1.0


@pytest.mark.gpu
@pytest.mark.parametrize("dims,N", [(1, 64), (2, 32)])
@pytest.mark.parametrize("c0", [1e-3, 0.1, 1e22])
def test_mobility_matches_oracle(dims, N, c0):
    import oracle
    from chgb import abi, config
    from chgb.sim import CahnHilliard
    from conftest import rel_maxnorm
    p = config.params(dims, N, "pseudospectral_mobility", "landau", dt=0.02, k=1.0, epsilon=0.9)
    p.mobility_type = abi.MOBILITIES["gel"]
    p.gel_phi_critical, p.gel_c0, p.gel_M_c, p.gel_beta_delta_F = 0.3, c0, 20.0, 90.0
    rho0 = config.init_density(dims, N, [0.4], initial_A=0.3, seed=9)
    sim = CahnHilliard(p, rho0)
    ref = oracle.OracleSim(p, rho0)
    for n in (1, 79):
        sim.evolve(n)
        ref.step(n)
        got, mob = sim.sync(with_mobility=True)
        assert rel_maxnorm(got, ref.rho()) <= 1e-12
        assert rel_maxnorm(mob, ref.mobility()) <= 1e-12
