"""Block fixed point for fields so small that psi^2 drops out of mu beside
the linear term: the shift that places it goes beyond a word.  Fields scaled
by powers of two down to the end of the integer range, and one whose values
span 200 decades, in 2D, as the 3D pair and as the 3D kernel: the split FP64
variant to 1e-14 relative max-norm (a step's own error is a few 2^-56)."""
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
    sim.evolve(steps)
    out = sim.sync()
    sim.close()
    return out


@pytest.mark.parametrize("dims,variant", [(2, 5), (3, 5), (3, 0)])
@pytest.mark.parametrize("power", [-28, -32, -40, -200, -800, "mixed"])
def test_small_fields(dims, variant, power):
    p = config.params(dims, 64, "euler", "landau", dt=0.01 if dims == 2 else 0.005, k=1.0, epsilon=0.9)
    if power == "mixed":
        rng = np.random.default_rng(11)
        rho0 = rng.uniform(-1.0, 1.0, 64 ** dims) * 10.0 ** rng.uniform(-300, -100, 64 ** dims)
    else:
        rho0 = config.init_density(dims, 64, [0.0], initial_A=0.3, seed=dims) * 2.0 ** power
    want = run(p, rho0, 10, 2)
    assert np.any(want)
    assert rel_maxnorm(run(p, rho0, 10, variant), want) <= 1e-14
