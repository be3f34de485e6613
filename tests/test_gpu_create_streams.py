"""chgb_create sets up a box's step state on the box's own stream: work that a
program has pending on the legacy default stream (a framework's default) neither
delays it nor is joined by it, so nothing of the set-up can land after the
first steps.  Shown by a capture under way on a blocking stream, during which
the runtime refuses every operation on the legacy stream."""
import ctypes

import numpy as np
import pytest

from chgb import abi, config
from chgb.sim import CahnHilliard

pytestmark = pytest.mark.gpu


def runtime():
    for name in ("libcudart.so.13", "libcudart.so.12", "libcudart.so"):
        try:
            return ctypes.CDLL(name)
        except OSError:
            pass
    pytest.skip("no shared CUDA runtime")


@pytest.mark.parametrize("integrator,dims,N", [("euler_mobility", 2, 64), ("euler", 2, 512), ("euler", 3, 64)])
def test_no_set_up_on_the_legacy_stream(integrator, dims, N):
    rt = runtime()
    p = config.params(dims, N, integrator, "landau", dt=0.005, k=1.0, epsilon=0.9)
    rho0 = config.init_density(dims, N, [0.0], initial_A=0.3, seed=N)
    CahnHilliard(p, rho0).close()        # whatever a process does once
    stream, graph = ctypes.c_void_p(), ctypes.c_void_p()
    assert rt.cudaStreamCreate(ctypes.byref(stream)) == 0
    assert rt.cudaStreamBeginCapture(stream, 2) == 0        # cudaStreamCaptureModeRelaxed
    try:
        sim = CahnHilliard(p, rho0)
        sim.evolve(3)
        got, variant = sim.sync(), sim.kernel_variant
    finally:
        ended = rt.cudaStreamEndCapture(stream, ctypes.byref(graph))
        if graph.value:
            rt.cudaGraphDestroy(graph)
        rt.cudaStreamDestroy(stream)
    assert variant == 5 and ended == 0
    sim.close()
    other = CahnHilliard(p, rho0)
    other.evolve(3)
    assert other.kernel_variant == 5 and np.array_equal(other.sync(), got)
    other.close()
