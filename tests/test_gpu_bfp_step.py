"""The 3D block-fixed-point step in one kernel (taken by rule, kernel_variant
0) against the pair of kernels that kernel_variant 5 asks for: the same bits,
at z chunks that divide the box and chunks that do not, for whole fields and
for fields that take the FP64 sums (NaN, zero, near the small end of the
double range); and the 2D kernel's tiles against the split variant."""
import numpy as np
import pytest

from chgb import config
from chgb.sim import CahnHilliard
from conftest import rel_maxnorm

pytestmark = pytest.mark.gpu


def run(p, rho0, steps, variant):
    q = p.copy()
    q.kernel_variant = variant
    sim = CahnHilliard(q, rho0)
    for n in steps:
        sim.evolve(n)
    out = sim.sync(), sim.launches, sim.kernel_variant
    sim.close()
    return out


@pytest.mark.parametrize("N,field", [(N, f) for N in (64, 128) for f in ("noise", "domains", "nan", "zero", "tiny")]
                         + [(256, "noise"), (256, "nan")])
def test_one_kernel_and_pair_give_the_same_bits(N, field):
    p = config.params(3, N, "euler", "landau", dt=0.005, k=1.0, epsilon=0.9)
    rho0 = config.init_density(3, N, [0.0], initial_A=0.3, seed=N)
    if field == "domains":
        rho0 = np.tanh(40.0 * rho0)
    elif field == "nan":
        rho0[N * N + 5] = np.nan
    elif field == "zero":
        rho0 = rho0 * 0.0
    elif field == "tiny":
        rho0 = rho0 * 2.0 ** -1000
    steps = (1, 6)
    one, n1, v1 = run(p, rho0, steps, 0)
    two, n2, v2 = run(p, rho0, steps, 5)
    assert v1 == v2 == 5 and n1 == 7 + 2 and n2 == 14 + 2
    assert np.array_equal(one, two, equal_nan=True)
    if field in ("noise", "domains"):
        split, _, _ = run(p, rho0, steps, 2)
        assert rel_maxnorm(one, split) <= 1e-14


@pytest.mark.parametrize("N", [32, 64, 512, 1024])
def test_tiles_in_2d(N):
    p = config.params(2, N, "euler", "landau", dt=0.01, k=1.2, epsilon=0.7)
    rho0 = config.init_density(2, N, [0.1], initial_A=0.5, seed=N)
    got, n, v = run(p, rho0, (3, 2), 5)
    assert v == 5 and n == 5 + 2
    split, _, _ = run(p, rho0, (3, 2), 2)
    assert rel_maxnorm(got, split) <= 1e-14
