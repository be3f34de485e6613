"""Three-species pseudospectral boxes of every size in a batch, up to those
whose row takes more threads than a batch CTA has: the bits of the box alone,
and the CPU oracle's field to 1e-12 relative max-norm, the project's parity
bar."""
import numpy as np
import pytest

import oracle
from chgb import config
from chgb.sim import Batch, CahnHilliard
from conftest import rel_maxnorm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,steps", [((32, 128, 256), 40), ((512, 1024, 64), 3), ((1024, 1024), 34)])
def test_three_species_in_a_batch(sizes, steps):
    reps = [config.params(2, N, "pseudospectral", "saleh", dt=1e-6, dx=10.0, k=[1e6, 2e6, 5e5], B2=2190.0, B3=1e7,
                          delta_AA=4.5e4, delta_BB=6.1e4, saleh_valence=(4, 3, 4)) for N in sizes]
    fields = [config.init_density(2, N, [9e-5, 7e-5, 3e-5], seed=N + i) for i, N in enumerate(sizes)]
    with Batch(reps) as b:
        for i, f in enumerate(fields):
            b.upload(i, f)
        b.step(steps)
        got = [b.download(i) for i in range(len(reps))]
    for i, (p, f) in enumerate(zip(reps, fields)):
        sim = CahnHilliard(p, f)
        sim.evolve(steps)
        assert np.array_equal(got[i], sim.sync()), sizes[i]
        sim.close()
        if steps <= 3 or p.N < 512:
            ref = oracle.OracleSim(p, f)
            ref.step(steps)
            assert rel_maxnorm(got[i], ref.rho()) <= 1e-12, sizes[i]
            ref.close()
