"""euler_mobility in block fixed point (one species, constant or free-energy
mobility, kernel_variant 0 from N = 32 in 2D and 3D): the fused FP64 kernel
to 1e-12 relative max-norm, the project's parity bar (a step's own error is a
few 2^-57 of the largest flux), mass to 1e-13, the same bits however the steps
are split over calls, and fields outside the integers' range (zeros, a NaN),
which take FP64 as the fused kernel does."""
import numpy as np
import pytest

from chgb import config
from chgb.sim import CahnHilliard
from conftest import rel_maxnorm

pytestmark = pytest.mark.gpu


def box(dims, N, variant=0, mobility="free_energy", M=1.0):
    p = config.params(dims, N, "euler_mobility", "simple_wertheim", dt=1e-4, dx=10.0, k=1e6, M=M,
                      mobility=mobility, valence=4, B2=2190.0,
                      delta=config.delta_value({"T": 300, "deltaH": -42200, "deltaS": -119.1, "salt": 0.5,
                                                "sticky_size": 6}, "d"))
    p.kernel_variant = variant
    return p


def run(p, rho0, *steps):
    sim = CahnHilliard(p, rho0)
    for n in steps:
        sim.evolve(n)
    out, v = sim.sync(), sim.kernel_variant
    sim.close()
    return out, v


def field(dims, N, domains):
    rho0 = config.init_density(dims, N, [1.107e-5], seed=dims + N)
    if domains:   # a dense slab in a dilute background, 300 to 1
        x = np.arange(N ** dims) % N
        rho0 = rho0 * np.where((x > N // 3) & (x < N // 2), 3.0, 0.01)
    return rho0


@pytest.mark.parametrize("dims,N,mobility,M,domains", [
    (2, 32, "free_energy", 1.0, True), (2, 64, "constant", 1.0, False), (2, 512, "free_energy", 1.0, False),
    (2, 512, "free_energy", 1.0, True), (3, 32, "free_energy", 1.0, False),
    (3, 32, "free_energy", 1.0, True), (3, 64, "constant", 0.05, False), (2, 512, "constant", 1.0, False),
    (3, 256, "free_energy", 1.0, False), (3, 256, "free_energy", 1.0, True)])
def test_matches_fp64_kernel(dims, N, mobility, M, domains):
    rho0 = field(dims, N, domains)
    steps = 20 if N < 256 else 4
    got, v = run(box(dims, N, 0, mobility, M), rho0, steps)
    split, _ = run(box(dims, N, 0, mobility, M), rho0, 1, steps - 1)
    want, _ = run(box(dims, N, 1, mobility, M), rho0, steps)
    assert v == 5
    assert np.array_equal(got, split)
    assert rel_maxnorm(got, want) <= 1e-12
    assert abs(got.mean() - rho0.mean()) <= 1e-13 * np.abs(rho0).max()


@pytest.mark.parametrize("dims,M,domains", [(3, 1.0, False), (3, 0.05, True)])
def test_diverging_box(dims, M, domains):
    """Constant mobility beyond the explicit step's stability limit, and a slab
    whose edge drives dilute cells below zero (a NaN logarithm): the integers'
    range ends on the way, and the fused kernel's NaNs stand in the same cells."""
    rho0 = field(dims, 64, domains)
    got, v = run(box(dims, 64, 0, "constant", M), rho0, 20)
    split, _ = run(box(dims, 64, 0, "constant", M), rho0, 1, 19)
    want, _ = run(box(dims, 64, 1, "constant", M), rho0, 20)
    assert v == 5
    assert np.array_equal(got, split, equal_nan=True)
    assert np.isnan(want).any() and np.array_equal(np.isnan(got), np.isnan(want))


def test_zero_and_nan_fields():
    zero = np.zeros(64 ** 3)
    got, _ = run(box(3, 64), zero, 3)
    want, _ = run(box(3, 64, 1), zero, 3)
    assert np.array_equal(got, want, equal_nan=True)
    rho0 = config.init_density(3, 64, [1.107e-5], seed=1)
    rho0[12345] = np.nan
    got, _ = run(box(3, 64), rho0, 2)
    want, _ = run(box(3, 64, 1), rho0, 2)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.max(np.abs(got[ok] - want[ok])) <= 1e-12 * np.max(np.abs(want[ok]))


@pytest.mark.parametrize("steps", [1, 2])
def test_a_new_field_starts_afresh(steps):
    """A field uploaded after an odd or even number of steps runs as in a fresh
    box, whatever the magnitudes of the one before."""
    p = box(2, 64)
    rho0 = config.init_density(2, 64, [1.107e-5], seed=4)
    sim = CahnHilliard(p, rho0 * 16)
    sim.evolve(steps)
    sim.upload(rho0)
    sim.evolve(3)
    got = sim.sync()
    sim.close()
    want, _ = run(p, rho0, 3)
    assert np.array_equal(got, want)
