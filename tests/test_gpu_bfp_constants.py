"""Block fixed point with a surface term just below a power of two and a large
epsilon: c2's mantissa of all ones, rounded to the step's unit, carries into
the next binade.  Against the split FP64 variant to 1e-14 relative max-norm: a
step's error is below 2 2^-56 of the field's largest value here (3 units of
mu's 2^-58, c1 = 1e-5), which grows by at most 1.2 a step."""
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
@pytest.mark.parametrize("k", [1.0, float(np.nextafter(1.0, 0.0)), 1.0 - 2.0 ** -40])
def test_surface_term_below_a_power_of_two(dims, variant, k):
    p = config.params(dims, 64, "euler", "landau", dt=1e-5, k=k, epsilon=2000.0)
    rho0 = config.init_density(dims, 64, [0.0], initial_A=0.3, seed=dims)
    want = run(p, rho0, 10, 2)
    assert rel_maxnorm(run(p, rho0, 10, variant), want) <= 1e-14
