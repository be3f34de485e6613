"""euler_mobility in block fixed point on fields of many decades: a cell's
density after a step is that of the fused FP64 kernel to one unit in its own
last place (the integers' error is held below 2^-56 of it, the two final
roundings half a unit each), however far below the field's largest it lies; and
a Landau field that is quiet away from a large spot keeps its quiet part to
1e-14 of its own largest value."""
import numpy as np
import pytest

from chgb import config
from chgb.sim import CahnHilliard

pytestmark = pytest.mark.gpu


def run(p, rho0, steps, variant):
    q = p.copy()
    q.kernel_variant = variant
    sim = CahnHilliard(q, rho0)
    sim.evolve(steps)
    out = sim.sync()
    assert sim.kernel_variant == (5 if variant == 0 else variant)
    sim.close()
    return out


@pytest.mark.parametrize("dims,N", [(2, 32), (2, 256), (3, 64)])
@pytest.mark.parametrize("mobility,M", [("free_energy", 1.0), ("constant", 1e-9)])
@pytest.mark.parametrize("decades", [0, 2, 6, 10, 14])
def test_every_cell_to_its_own_last_place(dims, N, mobility, M, decades):
    p = config.params(dims, N, "euler_mobility", "simple_wertheim", dt=1e-4, dx=10.0, k=1e6, M=M, mobility=mobility,
                      valence=4, B2=2190.0,
                      delta=config.delta_value({"T": 300, "deltaH": -42200, "deltaS": -119.1, "salt": 0.5,
                                                "sticky_size": 6}, "d"))
    x = np.arange(N ** dims) % N
    rho0 = 1e-5 * 10.0 ** (-decades * (1.0 - np.cos(2.0 * np.pi * x / N)) / 2.0)
    rho0 = rho0 * np.random.default_rng(decades).uniform(0.98, 1.02, N ** dims)
    got, want = run(p, rho0, 1, 0), run(p, rho0, 1, 1)
    assert np.all(np.isfinite(want))
    # a cell that the step changes by more than itself: relative to the change
    assert np.all(np.abs(got - want) <= 2.0 ** -52 * np.maximum(np.abs(want), np.abs(want - rho0) * 8.0))


@pytest.mark.parametrize("dims,N", [(2, 256), (3, 64)])
def test_quiet_landau_field_beside_a_spot(dims, N):
    p = config.params(dims, N, "euler_mobility", "landau", dt=0.005, k=1.0, epsilon=0.9, M=0.7)
    rho0 = np.random.default_rng(3).uniform(-1e-9, 1e-9, (N,) * dims)
    rho0[(slice(4, 12),) * dims] = 0.9
    steps = 3
    got, want = (run(p, rho0.reshape(-1), steps, v).reshape(rho0.shape) for v in (0, 1))
    quiet = (slice(N // 2, 3 * N // 4),) * dims
    assert np.max(np.abs(want[quiet])) < 1e-8
    assert np.max(np.abs(got[quiet] - want[quiet])) <= 1e-14 * np.max(np.abs(want[quiet]))
    assert np.max(np.abs(got - want)) <= 1e-14 * np.max(np.abs(want))
