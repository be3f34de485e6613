"""GPU parity of the line transforms at the sizes where their passes change:
every line length from 2 to 2048 (radix-8, radix-4 and radix-2 passes, one
thread to several warps a line, padded and unpadded buffers), ragged last
column CTAs, and fields whose values lie near the small end of the double
range.  Tolerance 1e-12 relative max-norm, the project's parity bar; a line's
own error is some 2^-(62 - G) sqrt(N), below 1e-13 for these fields."""
import numpy as np
import pytest

import oracle
from chgb import config
from chgb.sim import CahnHilliard
from conftest import rel_maxnorm

pytestmark = pytest.mark.gpu


def check(p, rho0, steps):
    sim = CahnHilliard(p, rho0)
    sim.evolve(steps)
    got = sim.sync()
    sim.close()
    ref = oracle.OracleSim(p, rho0)
    ref.step(steps)
    want = ref.rho()
    ref.close()
    assert np.all(np.isfinite(got))
    assert rel_maxnorm(got, want) <= 1e-12


@pytest.mark.parametrize("dims,N", [(1, 8), (1, 16), (1, 32), (1, 128), (1, 256), (1, 512), (1, 1024), (1, 4096),
                                    (2, 16), (2, 32), (2, 256), (2, 2048), (3, 4), (3, 128)])
def test_every_line_length(dims, N):
    p = config.params(dims, N, "pseudospectral", "landau", dt=0.05, k=1.0, epsilon=0.9)
    check(p, config.init_density(dims, N, [0.0], initial_A=0.3, seed=77 + N), 1 if N ** dims > 1 << 20 else 3)


@pytest.mark.parametrize("N", [4, 32, 64])
def test_three_species_lines(N):
    p = config.params(2, N, "pseudospectral", "saleh", dt=1e-6, dx=10.0, k=[1e6, 2e6, 5e5], B2=2190.0, B3=1e7,
                      delta_AA=4.5e4, delta_BB=6.1e4, saleh_valence=(4, 3, 4))
    check(p, config.init_density(2, N, [9e-5, 7e-5, 3e-5], seed=N), 10)


@pytest.mark.parametrize("power", [-905, -960])
def test_fields_near_the_small_end_of_the_double_range(power):
    p = config.params(2, 64, "pseudospectral", "landau", dt=0.05, k=1.0, epsilon=0.9)
    check(p, config.init_density(2, 64, [0.0], initial_A=0.3, seed=5) * 2.0 ** power, 5)
