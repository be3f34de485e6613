"""pseudospectral_mobility modes that one step damps by orders of magnitude: a
single wave of small amplitude without the linear term.  Its amplitude after the
step is the one before times (1 + c S - c (3/4)^d A^2) / (1 + c (S + 2 k q^2)), c =
dt M q^2 (the cubic term's other wave is another mode); compared in extended
precision to 2e-14 relative -- the transforms' own 1e-15 and a few roundings --
which a rounding of the mode before the step would exceed from a denominator of
200 on."""
import numpy as np
import pytest

from chgb import config
from chgb.sim import CahnHilliard

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,N", [(2, 64), (2, 256), (3, 32)])
@pytest.mark.parametrize("dt,S", [(1e-3, 0.0), (0.05, 0.3), (3.0, 0.0), (100.0, 0.0), (100.0, 0.3)])
def test_one_damped_wave(dims, N, dt, S):
    p = config.params(dims, N, "pseudospectral_mobility", "landau", dt=dt, k=1.0, epsilon=0.0, M=0.8, S=S)
    n = 3 * N // 8
    x = np.arange(N)
    wave = np.cos(2.0 * np.pi * ((n * x) % N) / N)
    rho0 = 1e-6 * wave
    for _ in range(dims - 1):
        rho0 = np.multiply.outer(wave, rho0)
    sim = CahnHilliard(p, rho0.reshape(-1))
    sim.evolve(1)
    got = sim.sync()
    sim.close()
    q2 = dims * (np.longdouble(2.0) * np.pi * n / N) ** 2   # the engine's q: pi as a double
    c = np.longdouble(dt) * np.longdouble(p.M) * q2
    want = (1 + c * np.longdouble(S) - c * np.longdouble(0.75) ** dims * np.longdouble(1e-6) ** 2) / (
        1 + c * (np.longdouble(S) + 2 * q2))
    r = rho0.reshape(-1).astype(np.longdouble)
    factor = np.sum(got * r) / np.sum(r * r)
    assert abs(factor - want) <= 2e-14 * abs(want), (float(factor), float(want))
