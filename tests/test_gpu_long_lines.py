"""GPU parity of the longest line transforms, eight values a thread, for every
model: rows of 1024 and 2048 packed values, columns of 2048 and 4096.  1e-12
relative max-norm, the project's parity bar; a line's own error is some
2^-(62 - G) sqrt(N), below 1e-13 for these fields."""
import numpy as np
import pytest

import oracle
from chgb import config
from chgb.sim import CahnHilliard
from conftest import rel_maxnorm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,N,model", [(1, 2048, "saleh"), (1, 4096, "saleh"), (1, 2048, "simple_wertheim"),
                                          (2, 2048, "saleh"), (2, 2048, "simple_wertheim"), (2, 4096, "landau")])
def test_longest_lines(dims, N, model):
    if model == "landau":
        p = config.params(dims, N, "pseudospectral", "landau", dt=0.05, k=1.0, epsilon=0.9)
        rho0 = config.init_density(dims, N, [0.0], initial_A=0.3, seed=N)
    elif model == "saleh":
        p = config.params(dims, N, "pseudospectral", "saleh", dt=1e-6, dx=10.0, k=[1e6, 2e6, 5e5], B2=2190.0, B3=1e7,
                          delta_AA=4.5e4, delta_BB=6.1e4, saleh_valence=(4, 3, 4))
        rho0 = config.init_density(dims, N, [9e-5, 7e-5, 3e-5], seed=N)
    else:
        p = config.params(dims, N, "pseudospectral", "simple_wertheim", dt=1e-4, dx=10.0, k=1e6, valence=4, B2=2190.0,
                          delta=45168.0)
        rho0 = config.init_density(dims, N, [1.107e-5], seed=N)
    steps = 3 if dims == 1 else 1
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
