"""The work a user of the engine has it do, as cases that can be timed and checked.

A case is one output interval of a program that steps Cahn-Hilliard boxes: the
time steps between two looks at the state, and the look itself.  Every case
goes through the package's public entry points (``CahnHilliard``, ``Adjoint``,
``Batch``), keeps its handle from one interval to the next as such a program
does, and hands back the whole field (a zero-copy view of device memory where
the program reads it there) and whatever else the program reads at that point.

``N`` is a power of two, as the engine demands; step counts are any number.
``exact`` restates each integrator in plain torch, FP64, from its definition.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "cahn-hilliard_gb300"))

from chgb import abi, config  # noqa: E402
from chgb.sim import Adjoint, Batch, CahnHilliard  # noqa: E402

GEL = {"phi_critical": 0.3, "c0": 0.1, "M_c": 20.0}
WERTHEIM = {"valence": 4, "B2": 2190.0}
WERTHEIM_DELTA = {"T": 300, "deltaH": -42200, "deltaS": -119.1, "salt": 0.5, "sticky_size": 6}
SALEH = {"B2": 2190.0, "B3": 1e7, "delta_AA": 4.5e4, "delta_BB": 6.1e4}
SALEH_VALENCE = (4, 3, 4)
SALEH_K = (1e6, 2e6, 5e5)
SALEH_RHO = (9e-5, 7e-5, 3e-5)


def listed():
    return [
        # the smallest run: 10,000 steps of a 64 x 64 quench with the energy every 1000 steps
        _box("euler_2d_64_output_interval", "euler", "landau", 2, 64, 1000, dt=0.01, observe=True),
        # a host program that asks for one step at a time (the reference's evolve() loop over a drop-in integrator)
        _box("euler_3d_64_step_by_step", "euler", "landau", 3, 64, 1, dt=0.005),
        # an ordinary 2D coarsening run, restarted from a state that has already separated into domains
        _box("euler_2d_1024_restart", "euler", "landau", 2, 1024, 100, dt=0.01, init="domains"),
        # the large 3D coarsening run
        _box("euler_3d_256_quench", "euler", "landau", 3, 256, 100, dt=0.005),
        # 3D DNA-nanostar condensation with the density-dependent mobility M0 rho X^4
        _box("wertheim_3d_128_mobility", "euler_mobility", "simple_wertheim", 3, 128, 25, dt=1e-4,
             mobility="free_energy"),
        # two associating species and their linker, semi-implicit
        _box("saleh_2d_256_spectral", "pseudospectral", "saleh", 2, 256, 50, dt=1e-6),
        # the critical quench whose structure factor is followed
        _box("spectral_2d_1024_quench_sq", "pseudospectral", "landau", 2, 1024, 100, dt=0.05, sq=True, observe=True),
        # droplets in 3D, an odd interval
        _box("spectral_3d_128_droplets", "pseudospectral", "landau", 3, 128, 27, dt=0.05, mean=-0.3),
        # a gelling mixture: the mobility follows its own order parameter
        _box("gel_2d_1024_m0_splitting", "pseudospectral_mobility", "landau", 2, 1024, 10, dt=0.02, mobility="gel",
             mean=-0.1, amp=0.3, S=0.3),
        # the same on a small box through the implicit solve
        _box("gel_2d_256_gmres", "pseudospectral_mobility", "landau", 2, 256, 2, dt=0.02, mobility="gel", mean=-0.1,
             amp=0.3, S=0.3, gmres=True),
        # parameter inference: the loss gradient through a trajectory, checkpointed
        _adjoint("adjoint_2d_256_spectral", "pseudospectral", 256, 200),
        # a parameter sweep: boxes of uneven sizes, both integrators, stepped together
        _batch("batch_sweep_mixed", 33, 64, 512, 32, 0.5),
    ]


def draw(rng):
    """A case of the same kinds, anywhere in their ranges."""
    kind = rng.choice(["euler", "euler", "wertheim", "spectral", "spectral", "saleh", "gel", "gmres", "adjoint", "batch"])
    dims = rng.choice([2, 3])
    if kind == "euler":
        N = 2 ** (rng.randint(5, 11) if dims == 2 else rng.randint(5, 8))
        c = _box(None, "euler", "landau", dims, N, _steps(rng, N ** dims, 1000, 1.0),
                 dt=rng.choice([0.0025, 0.005] if dims == 3 else [0.005, 0.01]),
                 init=rng.choice(["noise", "domains"]), observe=rng.random() < 0.5,
                 k=round(rng.uniform(0.5, 1.3), 3), epsilon=round(rng.uniform(0.5, 1.0), 3))
    elif kind == "wertheim":
        N = 2 ** (rng.randint(5, 10) if dims == 2 else rng.randint(5, 7))
        c = _box(None, "euler_mobility", "simple_wertheim", dims, N, _steps(rng, N ** dims, 200, 25.0), dt=1e-4,
                 mobility=rng.choice(["free_energy", "constant"]), observe=rng.random() < 0.5)
    elif kind == "spectral":
        N = 2 ** (rng.randint(6, 11) if dims == 2 else rng.randint(5, 7))
        c = _box(None, "pseudospectral", "landau", dims, N, _steps(rng, N ** dims, 200, 8.0),
                 dt=rng.choice([0.02, 0.05]), mean=rng.choice([0.0, -0.3]), sq=dims == 2 and rng.random() < 0.5,
                 S=rng.choice([0.0, 0.5]), dealias=rng.random() < 0.3, k=round(rng.uniform(0.5, 2.0), 3),
                 epsilon=round(rng.uniform(0.5, 1.0), 3))
    elif kind == "saleh":
        N = 2 ** (rng.randint(6, 9) if dims == 2 else 5)
        c = _box(None, "pseudospectral", "saleh", dims, N, _steps(rng, 3 * N ** dims, 100, 10.0), dt=1e-6)
    elif kind == "gel":
        N = 2 ** (rng.randint(6, 10) if dims == 2 else rng.randint(5, 7))
        c = _box(None, "pseudospectral_mobility", "landau", dims, N, _steps(rng, N ** dims, 50, 40.0), dt=0.02,
                 mobility="gel", mean=-0.1, amp=0.3, S=rng.choice([0.0, 0.3]), dealias=rng.random() < 0.5)
    elif kind == "gmres":
        c = _box(None, "pseudospectral_mobility", "landau", 2, 2 ** rng.randint(6, 8), rng.randint(1, 4), dt=0.02,
                 mobility="gel", mean=-0.1, amp=round(rng.uniform(0.2, 0.4), 3), S=0.3, gmres=True)
    elif kind == "adjoint":
        c = _adjoint(None, rng.choice(["euler", "pseudospectral"]), 2 ** rng.randint(6, 8), _steps(rng, 1, 300, 1.0))
    else:
        hi = rng.choice([256, 512])
        c = _batch(None, rng.randint(5, 48 if hi == 256 else 33), 64, hi, rng.randint(7, 40),
                   rng.choice([0.0, 0.5, 1.0]))
    c.pop("name")
    return c


def _steps(rng, cells, most, weight):
    """Steps of an interval, spread over their logarithm, no dearer than the largest listed case."""
    most = max(1, min(most, int(1.2e9 / (cells * weight))))
    return min(most, int(math.exp(rng.uniform(0.0, math.log(most + 1.0)))) or 1)


def _box(name, integrator, model, dims, N, steps, dt, mobility="constant", init="noise", mean=0.0, amp=1e-2, S=0.0,
         dealias=False, gmres=False, observe=False, sq=False, k=1.0, epsilon=0.9):
    return {"name": name, "kind": "box", "integrator": integrator, "model": model, "dims": dims, "N": N,
            "steps": steps, "dt": dt, "mobility": mobility, "init": init, "mean": mean, "amp": amp, "S": S,
            "dealias": dealias, "gmres": gmres, "observe": observe, "sq": sq, "k": k, "epsilon": epsilon}


def _adjoint(name, integrator, N, steps):
    return {"name": name, "kind": "adjoint", "integrator": integrator, "N": N, "steps": steps,
            "dt": 0.01 if integrator == "euler" else 0.05}


def _batch(name, boxes, N_min, N_max, steps, spectral):
    return {"name": name, "kind": "batch", "boxes": boxes, "N_min": N_min, "N_max": N_max, "steps": steps,
            "spectral": spectral}


# ---------------------------------------------------------------------------
# parameters and initial fields
# ---------------------------------------------------------------------------
def _params(c):
    if c["model"] == "landau":
        p = config.params(c["dims"], c["N"], c["integrator"], "landau", dt=c["dt"], k=c["k"], epsilon=c["epsilon"],
                          mobility=c["mobility"], S=c["S"], use_dealias=c["dealias"])
    elif c["model"] == "simple_wertheim":
        p = config.params(c["dims"], c["N"], c["integrator"], "simple_wertheim", dt=c["dt"], dx=10.0, k=1e6,
                          M=1.0 if c["mobility"] == "free_energy" else 0.05, mobility=c["mobility"],
                          delta=config.delta_value(WERTHEIM_DELTA, "delta"), **WERTHEIM)
    else:
        p = config.params(c["dims"], c["N"], c["integrator"], "saleh", dt=c["dt"], dx=10.0, k=list(SALEH_K),
                          saleh_valence=SALEH_VALENCE, **SALEH)
    if c["mobility"] == "gel":
        p.gel_phi_critical, p.gel_c0, p.gel_M_c = GEL["phi_critical"], GEL["c0"], GEL["M_c"]
        p.gel_beta_delta_F = 10.0 / (1.0 - c["epsilon"]) - math.log(24000.0)
    if c["gmres"]:
        p.use_gmres, p.gmres_restart, p.gmres_max_iter, p.gmres_tol = 1, 10, 200, 1e-11
    return p


def _field(c, seed):
    """Initial density: the seeded noise of a quench, or (a restart) separated domains with smooth interfaces."""
    dims, N = c["dims"], c["N"]
    if c["model"] == "simple_wertheim":
        return config.init_density(dims, N, [1.107e-5], seed=seed)
    if c["model"] == "saleh":
        return config.init_density(dims, N, list(SALEH_RHO), seed=seed)
    if c["init"] == "noise":
        return config.init_density(dims, N, [0.0], initial_A=c["amp"], seed=seed) + c["mean"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((N,) * dims, generator=g, device="cuda", dtype=torch.float64)
    q = _wave_numbers(dims, N, 1.0)[0]
    x = torch.fft.irfftn(torch.fft.rfftn(x) * torch.exp(-q * (0.5 * min(8.0, N / 8)) ** 2), s=(N,) * dims)
    return torch.tanh(1.5 * x / x.std()).mul_(math.sqrt(c["epsilon"])).cpu().numpy().reshape(-1)


def _sweep(c, seed):
    """The boxes of a parameter sweep: uneven sizes, their own constants and seeds."""
    rng = np.random.default_rng(seed)
    sizes = [n for n in (64, 128, 256, 512, 1024) if c["N_min"] <= n <= c["N_max"]]
    out = []
    for i in range(c["boxes"]):
        spectral = (i + 0.5) / c["boxes"] < c["spectral"]
        b = _box(None, "pseudospectral" if spectral else "euler", "landau", 2, sizes[i % len(sizes)], c["steps"],
                 dt=0.05 if spectral else 0.01, mean=float(rng.uniform(-0.4, 0.4)),
                 k=float(rng.uniform(0.5, 2.0 if spectral else 1.4)), epsilon=float(rng.uniform(0.5, 1.0)))
        out.append((b, int(rng.integers(1, 1 << 31))))
    return out


class _View:
    """Device memory of a handle as torch sees it, without a copy; the tensor keeps `owner`, which frees it, alive."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3}


def _view(state, owner, key, ptr, n):
    """The tensor over `ptr` (a handle has two density buffers that it swaps)."""
    views = state["views"]
    if (key, ptr) not in views:
        views[key, ptr] = torch.as_tensor(_View(owner, ptr, n), device="cuda")
    return views[key, ptr]


def prepare(case, seed):
    if case["kind"] == "adjoint":
        p = config.params(2, case["N"], case["integrator"], "landau", dt=case["dt"], epsilon=0.9)
        rho0, target = _adjoint_inputs(case, seed)
        return {"case": case, "adj": Adjoint(p, case["steps"]), "rho0": rho0, "target": target}
    if case["kind"] == "batch":
        boxes = _sweep(case, seed)
        params = [_params(b) for b, _ in boxes]
        batch = Batch(params)
        for i, (b, s) in enumerate(boxes):
            batch.upload(i, _field(b, s))
        # chgb_device_rho of a replica, through the handle that the batch lends
        handles = [batch.lib.chgb_batch_replica(batch._b, i) for i in range(len(boxes))]
        return {"case": case, "batch": batch, "params": params, "handles": handles, "views": {}}
    sim = CahnHilliard(_params(case), _field(case, seed))
    return {"case": case, "sim": sim, "views": {}}


def run(state):
    case = state["case"]
    if case["kind"] == "adjoint":
        # gradient of sum_q (S(q) - S*(q))^2 with respect to the initial field and (epsilon, k, M)
        sq, rho_t = state["adj"].forward(state["rho0"])
        grad_rho0, grad_params = state["adj"].backward(dl_dsq=2.0 * (sq - state["target"]))
        return {"sq": sq, "rho_t": rho_t, "grad_rho0": grad_rho0, "grad_params": grad_params}
    if case["kind"] == "batch":
        batch = state["batch"]
        batch.step(case["steps"])
        batch.synchronize()
        out = []
        for i, (p, h) in enumerate(zip(state["params"], state["handles"])):
            ptr = abi._D()
            abi.check(batch.lib, batch.lib.chgb_device_rho(h, ptr), h)
            out.append(_view(state, batch, i, abi.ctypes.cast(ptr, abi.ctypes.c_void_p).value, p.bins))
        return out
    sim = state["sim"]
    sim.evolve(case["steps"])
    out = {"rho": _view(state, sim, "rho", sim.device_rho(), sim.n)}
    if case["sq"]:
        out["sq"] = sim.structure_factor()[1]
    if case["observe"]:
        out["mass"], out["free_energy"], _ = sim.observables()
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without: the state read and written once (a checkpointed
# gradient also its inputs and outputs), and the arithmetic of its time steps
# ---------------------------------------------------------------------------
def _step_flops(integrator, model, dims, N, gmres=False):
    """Operations of one cell (all species) and time step, from the integrators' definitions."""
    species = 3 if model == "saleh" else 1
    fprime = {"landau": 4.0, "simple_wertheim": 40.0, "saleh": 160.0}[model]
    if integrator == "euler":
        return fprime + species * (2 * (2 * dims + 2) + 4.0)
    if integrator == "euler_mobility":
        return fprime + species * (2 * dims + 4 + 6 * dims + 4.0) + 10.0
    fft = species * 2.5 * dims * math.log2(N)            # one real transform
    if integrator == "pseudospectral":
        return 2 * fft + fprime + species * 4.0
    step = (2 + 2 * dims) * fft + fprime + 30.0 + 10 * dims
    return 12 * step if gmres else step                  # about twelve operator applications to a solve


def work(case):
    if case["kind"] == "adjoint":
        n = case["N"] ** 2
        step = _step_flops(case["integrator"], "landau", 2, case["N"])
        return {"bytes": 8.0 * 3 * n, "flops": 4.0 * step * n * case["steps"]}
    if case["kind"] == "batch":
        boxes = [b for b, _ in _sweep(case, 0)]
        return {"bytes": sum(16.0 * b["N"] ** 2 for b in boxes),
                "flops": sum(_step_flops(b["integrator"], "landau", 2, b["N"]) * b["N"] ** 2 * b["steps"] for b in boxes)}
    cells = case["N"] ** case["dims"]
    species = 3 if case["model"] == "saleh" else 1
    return {"bytes": 16.0 * species * cells,
            "flops": _step_flops(case["integrator"], case["model"], case["dims"], case["N"], case["gmres"]) * cells
            * case["steps"]}


# ---------------------------------------------------------------------------
# the same in plain torch, FP64
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed)
    if case["kind"] == "batch":
        return [_exact_box(b, s)["rho"] for b, s in _sweep(case, seed)]
    return _exact_box(case, seed)


def _exact_box(case, seed):
    p = _params(case)
    dims, N, S = case["dims"], case["N"], p.n_species
    # [species][z][y][x]: x is the fastest axis of the engine's layout
    rho = torch.from_numpy(_field(case, seed)).cuda().reshape((S,) + (N,) * dims)
    if case["integrator"] in ("euler", "euler_mobility"):
        for _ in range(case["steps"]):
            rho = _explicit_step(p, case, rho)
    elif case["integrator"] == "pseudospectral":
        rho = _spectral_steps(p, case, rho)
    else:
        rho = _spectral_mobility_steps(p, case, rho)
    out = {"rho": rho.reshape(-1)}
    if case["sq"]:
        out["sq"] = _structure_factor(rho[0])
    if case["observe"]:
        out["mass"], out["free_energy"] = _observables(p, rho)
    return out


def _column(values, dims):
    return torch.tensor(list(values), dtype=torch.float64, device="cuda").reshape((-1,) + (1,) * dims)


def _laplacian(x, dims):
    out = -2.0 * dims * x
    for a in range(1, dims + 1):
        out = out + torch.roll(x, 1, a) + torch.roll(x, -1, a)
    return out


def _wertheim_X(p, rho):
    a = 2.0 * p.model.valence * p.model.delta * rho
    return 2.0 / (1.0 + torch.sqrt(1.0 + 2.0 * a))


def _bulk(p, rho):
    """f'(rho)."""
    m = p.model
    if m.kind == abi.MODELS["landau"]:
        return rho * (rho * rho - m.epsilon)
    if m.kind == abi.MODELS["simple_wertheim"]:
        return 2.0 * m.B2 * rho + torch.log(rho) + m.valence * torch.log(_wertheim_X(p, rho))
    total = rho.sum(0)
    half = m.saleh_valence[2] // 2
    X = [2.0 / (1.0 + torch.sqrt(1.0 + 4.0 * d * (m.saleh_valence[s] * rho[s] + half * rho[2])))
         for s, d in ((0, m.delta_AA), (1, m.delta_BB))]
    bond = torch.stack([m.saleh_valence[0] * X[0].log(), m.saleh_valence[1] * X[1].log(),
                        half * (X[0].log() + X[1].log())])
    return torch.log(rho) + 2.0 * m.B2 * total + 3.0 * m.B3 * total * total + bond


def _explicit_step(p, case, rho):
    dims = case["dims"]
    mu = _bulk(p, rho) - _column(p.k[:p.n_species], dims) * (2.0 / p.dx ** 2) * _laplacian(rho, dims)
    if case["mobility"] == "constant":
        return rho + p.dt * p.M / p.dx ** 2 * _laplacian(mu, dims)
    M = p.M * rho * _wertheim_X(p, rho) ** p.model.valence
    out = rho
    for a in range(1, dims + 1):
        flux = 0.5 * (M + torch.roll(M, -1, a)) * (torch.roll(mu, -1, a) - mu)
        out = out + p.dt / p.dx ** 2 * (flux - torch.roll(flux, 1, a))
    return out


def _wave_numbers(dims, N, dx):
    """|q|^2 and the components along each stored axis of the half spectrum."""
    full = 2.0 * math.pi * torch.fft.fftfreq(N, dx, dtype=torch.float64, device="cuda")
    full[N // 2] = -math.pi / dx
    half = 2.0 * math.pi / (N * dx) * torch.arange(N // 2 + 1, dtype=torch.float64, device="cuda")
    axes = [full] * (dims - 1) + [half]
    comps = [a.reshape((1,) * i + (-1,) + (1,) * (dims - 1 - i)) for i, a in enumerate(axes)]
    shape = (N,) * (dims - 1) + (N // 2 + 1,)
    return sum(c * c for c in comps).expand(shape), comps


def _c2r(hat, dims, N):
    """Unnormalised inverse of a half spectrum; the last axis drops the imaginary parts a real row cannot hold."""
    for a in range(-dims, -1):
        hat = torch.fft.ifft(hat, dim=a, norm="forward")
    hat = hat.clone()
    hat[..., 0].imag.zero_()
    hat[..., N // 2].imag.zero_()
    return torch.fft.irfft(hat, n=N, dim=-1, norm="forward")


def _r2c(x, dims):
    return torch.fft.rfftn(x, dim=tuple(range(-dims, 0)))


def _dealias_mask(p, case, q2):
    cut = math.pi / p.dx * 2.0 / 3.0
    q = torch.sqrt(q2)
    # the 2D `pseudospectral` dealiaser leaves the cut itself out
    strict = case["integrator"] == "pseudospectral" and case["dims"] == 2
    return ((q < cut) if strict else (q <= cut)).to(torch.float64) if case["dealias"] else 1.0


def _spectral_coefficients(p, q2, dims, mask, k=None, M=None):
    k = _column(p.k[:p.n_species], dims) if k is None else k
    M = p.M if M is None else M
    denom = 1.0 + p.dt * M * (p.splitting_S * q2 + 2.0 * k * q2 * q2)
    return (1.0 + p.dt * M * q2 * p.splitting_S) / denom, p.dt * M * q2 * mask / denom


def _spectral_steps(p, case, rho):
    dims, N = case["dims"], case["N"]
    q2, _ = _wave_numbers(dims, N, p.dx)
    alpha, beta = _spectral_coefficients(p, q2, dims, _dealias_mask(p, case, q2))
    hat = _r2c(rho, dims)
    for _ in range(case["steps"]):
        hat = alpha * hat - beta * _r2c(_bulk(p, rho), dims)
        rho = torch.fft.irfftn(hat, s=(N,) * dims)
    return rho


def _spectral_mobility_steps(p, case, rho):
    dims, N = case["dims"], case["N"]
    bins, dt, S, k = float(N ** dims), p.dt, p.splitting_S, p.k[0]
    q2, comps = _wave_numbers(dims, N, p.dx)
    mask = _dealias_mask(p, case, q2)
    hat = _r2c(rho, dims)
    raw = np.random.RandomState(5489)._bit_generator.random_raw(2 * N ** dims).astype(np.float64)
    gel = torch.from_numpy((raw[0::2] + raw[1::2] * 2.0 ** 32) / 2.0 ** 64 * 1e-4).cuda().reshape(rho.shape)
    e = math.exp(p.gel_beta_delta_F)

    def divergence(h, M):
        """The spectrum of div(M grad x) for the spectrum h of x."""
        out = 0.0
        for kd in comps:
            flux = M * _c2r(1j * kd * h * mask, dims, N) / bins
            out = out + 1j * kd * mask * _r2c(flux, dims)
        return out

    for _ in range(case["steps"]):
        g = (e / (1.0 + e) * (rho + 1.0) / 2.0 - p.gel_phi_critical) / (1.0 - p.gel_phi_critical)
        gel = gel + p.gel_M_c * (g * gel - gel * gel) * dt
        M = torch.exp(-gel / p.gel_c0)
        M0 = float(M.max())
        f = _bulk(p, rho)
        denom = 1.0 + dt * M0 * (S * q2 + 2.0 * k * q2 * q2)
        if not case["gmres"]:
            fh = _r2c(f, dims)
            div = divergence((fh + 2.0 * k * q2 * hat) * mask, M - M0)
            hat = (hat + dt * div - dt * M0 * q2 * (fh - S * hat)) / denom
            rho = _c2r(hat / bins, dims, N)
            continue
        b = rho + dt * _c2r(divergence(_r2c(f - S * rho, dims), M), dims, N) / bins

        def A(x):
            h = (S + 2.0 * k * q2) * _r2c(x, dims) * mask
            return x - dt * _c2r(divergence(h, M), dims, N) / bins

        def P(x):
            return _c2r(_r2c(x, dims) / denom, dims, N) / bins

        rho = _solve(A, P, b, rho)
        hat = _r2c(rho, dims)
    return rho


def _solve(A, P, b, x, cycles=6, m=25):
    """Preconditioned GMRES, far below the engine's own tolerance."""
    scale = float(P(b).norm())
    for _ in range(cycles):
        r = P(b - A(x))
        beta = float(r.norm())
        if beta <= 1e-15 * scale:
            break
        V, H = [r / beta], np.zeros((m + 1, m))
        for j in range(m):
            w = P(A(V[j]))
            for _twice in range(2):
                for i in range(j + 1):
                    h = float((w * V[i]).sum())
                    H[i, j] += h
                    w = w - h * V[i]
            H[j + 1, j] = float(w.norm())
            V.append(w / H[j + 1, j])
            y, res = np.linalg.lstsq(H[:j + 2, :j + 1], beta * np.eye(j + 2)[0], rcond=None)[:2]
            if len(res) and math.sqrt(float(res[0])) <= 1e-15 * scale:
                break
        for i, yi in enumerate(y):
            x = x + float(yi) * V[i]
    return x


def _shells(N):
    i = torch.fft.fftfreq(N, 1.0 / N, dtype=torch.float64, device="cuda")
    return torch.round(torch.sqrt(i[:, None] ** 2 + i[None, :] ** 2)).to(torch.int64).reshape(-1)


def _structure_factor(rho):
    N = rho.shape[-1]
    sk = torch.fft.fft2(rho - rho.mean()).abs().square().reshape(-1) / N ** 2
    shell = _shells(N)
    count = torch.bincount(shell).to(torch.float64)
    return torch.zeros_like(count).index_add(0, shell, sk) / count


def _observables(p, rho):
    """(average mass, average free energy) of Landau and simple_wertheim boxes."""
    dims, m = p.dims, p.model
    if m.kind == abi.MODELS["landau"]:
        f = -0.5 * m.epsilon * rho ** 2 + 0.25 * rho ** 4
    else:
        X = _wertheim_X(p, rho)
        f = m.B2 * rho ** 2 + rho * (torch.log(rho * m.density_conversion_factor) - 1.0)
        f = f + m.valence * rho * (torch.log(X) + 0.5 * (1.0 - X))
    for a in range(1, dims + 1):
        f = f + p.k[0] * ((torch.roll(rho, -1, a) - rho) / p.dx) ** 2
    V = p.dx ** 3 / p.bins
    return float(rho.sum()) * V, float(f.sum()) * V


def _adjoint_inputs(case, seed):
    N = case["N"]
    rho0 = config.init_density(2, N, [0.0], initial_A=1e-2, seed=seed)
    n = int(_shells(N).max()) + 1
    q = 2.0 * math.pi * np.arange(n) / N
    # a target spectrum with the peak a quench of this length grows
    return rho0, 1e-3 * np.exp(-((q - 0.65) / 0.3) ** 2) * (1.0 + 0.1 * np.cos(seed + np.arange(n)))


def _exact_adjoint(case, seed):
    N = case["N"]
    p = config.params(2, N, case["integrator"], "landau", dt=case["dt"], epsilon=0.9)
    rho0, target = _adjoint_inputs(case, seed)
    x0 = torch.from_numpy(rho0).cuda().reshape(1, N, N).requires_grad_()
    eps, k, M = (torch.tensor(v, dtype=torch.float64, device="cuda", requires_grad=True)
                 for v in (p.model.epsilon, p.k[0], p.M))
    rho = x0
    if case["integrator"] == "euler":
        for _ in range(case["steps"]):
            mu = rho * (rho * rho - eps) - 2.0 * k / p.dx ** 2 * _laplacian(rho, 2)
            rho = rho + p.dt * M / p.dx ** 2 * _laplacian(mu, 2)
    else:
        q2, _ = _wave_numbers(2, N, p.dx)
        alpha, beta = _spectral_coefficients(p, q2, 2, 1.0, k, M)
        hat = _r2c(rho, 2)
        for _ in range(case["steps"]):
            hat = alpha * hat - beta * _r2c(rho * (rho * rho - eps), 2)
            rho = torch.fft.irfftn(hat, s=(N, N))
    sq = _structure_factor(rho[0])
    loss = (sq - torch.from_numpy(target).cuda()).square().sum()
    g = torch.autograd.grad(loss, [x0, eps, k, M])
    return {"sq": sq.detach(), "rho_t": rho.detach().reshape(-1), "grad_rho0": g[0].reshape(-1),
            "grad_params": torch.stack(g[1:])}
