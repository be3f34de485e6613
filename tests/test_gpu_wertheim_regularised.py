"""simple_wertheim's f' and mobility for densities on either side of the
regularisation, elementwise against the oracle: 1e-13 relative, as for the
other densities of the device hooks (f' is of order 10 or more here, its
logarithm's error 2 2^-53 times the valence; the mobility a few last places),
and steps of a box with cells on either side to 1e-12 relative max-norm, the
project's parity bar."""
import ctypes

import numpy as np
import pytest

import oracle
from chgb import abi, config
from chgb.sim import CahnHilliard
from conftest import rel_maxnorm

pytestmark = pytest.mark.gpu
DELTA = {"T": 300, "deltaH": -42200, "deltaS": -119.1, "salt": 0.5, "sticky_size": 6}


def wertheim(dims, N, integrator, reg, valence=4, mobility="constant", dt=1e-5):
    p = config.params(dims, N, integrator, "simple_wertheim", dt=dt, dx=10.0, k=1e6,
                      M=1.0 if mobility == "free_energy" else 0.02, mobility=mobility, valence=valence, B2=2190.0,
                      delta=config.delta_value(DELTA, "delta"))
    p.model.regularisation_delta = reg
    return p


@pytest.mark.parametrize("valence", [1, 4, 7])
@pytest.mark.parametrize("reg", [0.0, 1e-12, 1e-6, 1.1e-5, 1.0])
def test_hooks(reg, valence):
    import torch
    lib = abi.load_library()
    p = wertheim(2, 32, "euler", reg, valence)
    rng = np.random.default_rng(valence)
    near = reg * (1.0 + np.concatenate([rng.uniform(-1e-3, 1e-3, 60), [0.0, -2.0 ** -53, 2.0 ** -52]])) if reg else np.empty(0)
    rho = np.concatenate([rng.uniform(1e-7, 1e-4, 512), 10.0 ** rng.uniform(-13, -1, 512), near])
    d_rho = torch.tensor(rho, device="cuda", dtype=torch.float64)
    d_out = torch.zeros_like(d_rho)
    torch.cuda.synchronize()
    for want, call in ((oracle.der_bulk_free_energy(p.model, rho, rho.size),
                        lambda: lib.chgb_der_bulk_free_energy(ctypes.byref(p.model), ctypes.c_void_p(d_rho.data_ptr()),
                                                              ctypes.c_void_p(d_out.data_ptr()), rho.size, None)),
                       (oracle.set_mobility(p.model, rho, 2.5),
                        lambda: lib.chgb_set_mobility(ctypes.byref(p.model), ctypes.c_void_p(d_rho.data_ptr()), 2.5,
                                                      ctypes.c_void_p(d_out.data_ptr()), rho.size, None))):
        abi.check(lib, call())
        torch.cuda.synchronize()
        got = d_out.cpu().numpy()
        scale = np.maximum(np.abs(want), 1.0) if want.min() < -1.0 or want.max() > 1.0 else np.abs(want)
        assert np.max(np.abs(got - want) / scale) <= 1e-13


@pytest.mark.parametrize("integrator,mobility", [("euler", "constant"), ("euler_mobility", "free_energy"),
                                                 ("pseudospectral", "constant")])
@pytest.mark.parametrize("dims,N", [(2, 32), (2, 128), (3, 32)])
@pytest.mark.parametrize("reg", [1.107e-5, 1e-3])
def test_steps(integrator, mobility, dims, N, reg):
    p = wertheim(dims, N, integrator, reg, 4, mobility)
    rho0 = config.init_density(dims, N, [1.107e-5], seed=N)
    sim = CahnHilliard(p, rho0)
    sim.evolve(20)
    ref = oracle.OracleSim(p, rho0)
    ref.step(20)
    assert rel_maxnorm(sim.sync(), ref.rho()) <= 1e-12
    sim.close()
    ref.close()
