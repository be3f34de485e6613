"""The pseudospectral adjoint of boxes with eight values a thread (N = 2048 and
4096): the trajectory and the gradients of a field that repeats a smaller box
and a loss seed that repeats with it are the smaller box's, repeated, and the
parameters' gradients the smaller box's times the number of copies.  1e-12
relative, the project's parity bar: a step's error is below 1e-14."""
import numpy as np
import pytest

from chgb import config
from chgb.sim import Adjoint
from conftest import rel_maxnorm

pytestmark = pytest.mark.gpu


def gradients(N, rho0, seed, steps, K):
    p = config.params(2, N, "pseudospectral", "landau", dt=0.05, k=1.1, M=0.9, epsilon=0.8, S=0.3)
    with Adjoint(p, steps, K) as adj:
        _, rho_t = adj.forward(rho0)
        return rho_t, *adj.backward(dl_drho_t=seed)


@pytest.mark.parametrize("N", [1024, 2048, 4096])
def test_repeated_box(N):
    n, steps, K = 256, 7, 3
    copies = N // n
    rho0 = config.init_density(2, n, [0.1], initial_A=0.4, seed=N)
    seed = np.random.default_rng(N).standard_normal(n * n)
    want_t, want_g0, want_g3 = gradients(n, rho0, seed, steps, K)
    tile = lambda x: np.tile(x.reshape(n, n), (copies, copies)).reshape(-1)
    got_t, got_g0, got_g3 = gradients(N, tile(rho0), tile(seed), steps, K)
    assert rel_maxnorm(got_t, tile(want_t)) <= 1e-12
    assert rel_maxnorm(got_g0, tile(want_g0)) <= 1e-12
    # sums over the box of terms of either sign
    scale = copies ** 2 * np.abs(want_g3)
    assert np.all(np.abs(got_g3 - copies ** 2 * want_g3) <= 1e-10 * scale), (got_g3, want_g3)
