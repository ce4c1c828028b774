"""The measured workloads: what users of the fiber solver have it do, from one short fiber to the full batch.

Every fiber case makes the round trip of the reference's fast solver: the fiber data goes in (``set_states``), one
time span is advanced from the start of the simulation, the fiber data comes back (``states``).  Inputs follow from
the seed: travelling action potentials of random position and width on every fiber, gates near their steady
states, uneven element lengths, per-fiber conductivities and channel conductances, motor units of which some fire
at the start of the span.  ``exact`` restates the same equations in 64-bit torch.
"""
import ctypes
import math

import numpy as np
import torch
import torch.utils.checkpoint

from opendihu_b200 import _native, adjoint, emg, solver, workloads

STIMULUS_MS = 0.1       # setSpecificStatesRepeatAfterFirstCall: junction nodes are held at 20 mV that long


def listed():
    return [
        # the hodgkin_huxley_fast example: one short fiber, the smallest call (launches and latency)
        dict(name="hh_one_fiber", kind="hh", fibers=1, min_nodes=101, max_nodes=101, scheme="ImplicitEuler",
             method="split", precision="fp64", rule="vc", approximate=False, dt0=2e-4, dt=2e-3, steps=50),
        # plain configuration in the default method and precision: 16 fibers of 14.8 cm
        dict(name="hh_plain_fp64", kind="hh", fibers=16, min_nodes=1481, max_nodes=1481, scheme="ImplicitEuler",
             method="split", precision="fp64", rule="vc", approximate=False, dt0=1e-4, dt=1e-3, steps=400),
        # the same fibers with useSinglePrecision and the fused method (one fiber over a thread-block cluster)
        dict(name="hh_plain_fp32", kind="hh", fibers=16, min_nodes=1481, max_nodes=1481, scheme="ImplicitEuler",
             method="fused", precision="fp32", rule="vc", approximate=False, dt0=1e-4, dt=1e-3, steps=400),
        # the reference's default settings: approximate exponential, onlyComputeIfHasBeenStimulated and
        # disableComputationWhenStatesAreCloseToEquilibrium on, the 7 x 7 fibers of its examples
        dict(name="hh_default_options", kind="hh", fibers=49, min_nodes=1481, max_nodes=1481, scheme="ImplicitEuler",
             method="split", precision="fp64", rule="vc", approximate=True, dt0=1e-4, dt=1e-3, steps=50, skip=True),
        # the batching configuration at full size: 4096 uneven fibers, FP32 reaction, fused (the headline workload)
        dict(name="hh_batch_fp32", kind="hh", fibers=4096, min_nodes=500, max_nodes=2500, scheme="CrankNicolson",
             method="fused", precision="fp32", rule="center", approximate=False, dt0=1e-4, dt=1e-3, steps=150),
        # a quarter of that batch in the default method and precision
        dict(name="hh_batch_fp64", kind="hh", fibers=1024, min_nodes=500, max_nodes=2500, scheme="CrankNicolson",
             method="split", precision="fp64", rule="center", approximate=False, dt0=1e-4, dt=1e-3, steps=50),
        # Shorten muscle model (56 states), FP32 reaction: a 13 x 13 grid of fibers
        dict(name="shorten_fp32", kind="shorten", fibers=169, min_nodes=1481, max_nodes=1481, method="split",
             precision="fp32", dt0=1e-5, dt=5e-4, steps=8),
        # the same model in FP64 on a 6 x 6 grid
        dict(name="shorten_fp64", kind="shorten", fibers=36, min_nodes=1481, max_nodes=1481, method="split",
             precision="fp64", dt0=1e-5, dt=5e-4, steps=4),
        # gradients of a sensor trace with respect to conductivities and channel parameters (forward and backward)
        dict(name="hh_adjoint", kind="adjoint", fibers=64, min_nodes=1481, max_nodes=1481, sensors=32, checkpoint=50,
             dt0=1e-4, dt=1e-3, steps=100),
        # EMG: one static bidomain solve on the mesh of the coupled example (Jacobi-preconditioned)
        dict(name="emg_jacobi", kind="emg", nx=25, ny=25, nz=149, rtol=1e-8, preconditioner="jacobi"),
        # EMG on the large mesh (multigrid, the default from 300,000 nodes)
        dict(name="emg_multigrid", kind="emg", nx=97, ny=97, nz=297, rtol=1e-8, preconditioner="multigrid"),
        # the diffusion solve as a standalone operator on device arrays (codes with their own reaction step)
        dict(name="diffusion_operator", kind="diffusion", fibers=4096, min_nodes=500, max_nodes=2500,
             scheme="CrankNicolson", dt=1e-3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hh", "hh", "hh", "hh", "hh", "shorten", "adjoint", "emg", "diffusion"])
    if kind == "emg":
        return dict(kind=kind, nx=rng.randint(9, 49), ny=rng.randint(9, 49), nz=rng.randint(21, 160), rtol=1e-8,
                    preconditioner=rng.choice(["jacobi", "multigrid"]))
    lo = _log_int(rng, 40, 1500)
    hi = rng.randint(lo, 2500)
    mean = 0.5 * (lo + hi)
    scheme = rng.choice(["ImplicitEuler", "CrankNicolson"])
    if kind == "diffusion":
        return dict(kind=kind, fibers=_log_int(rng, 1, min(4096, 6e6 / mean)), min_nodes=lo, max_nodes=hi,
                    scheme=scheme, dt=1e-3)
    if kind == "shorten":
        n = rng.randint(1, max(1, int(min(100, 1e5 / mean))))
        return dict(kind=kind, fibers=n, min_nodes=lo, max_nodes=hi, method="split",
                    precision=rng.choice(["fp32", "fp64"]), dt0=1e-5, dt=5e-4, steps=rng.randint(1, 4))
    if kind == "adjoint":
        n = _log_int(rng, 1, max(2, min(64, 6e4 / hi)))
        return dict(kind=kind, fibers=n, min_nodes=hi, max_nodes=hi, sensors=rng.randint(4, 32),
                    checkpoint=rng.choice([10, 25, 50]), dt0=1e-4, dt=1e-3, steps=rng.randint(20, 80))
    fibers = _log_int(rng, 1, max(2, min(4096, 2e6 / mean)))
    method, precision = rng.choice([("split", "fp64"), ("split", "fp64"), ("fused", "fp32"), ("fused", "fp32"),
                                    ("split", "fp32"), ("fused", "fp64")])
    rule = rng.choice(["vc", "center"])
    if rule == "vc":   # the vc rule is the one of equally long fibers
        lo = hi
        fibers = max(1, min(fibers, int(2e6 / hi)))
    return dict(kind="hh", fibers=fibers, min_nodes=lo, max_nodes=hi, scheme=scheme, method=method,
                precision=precision, rule=rule, dt0=1e-4, dt=1e-3, steps=rng.randint(20, 120),
                # (1 + x/1024)^1024 in FP32 is exactly 1 for small x: 0/0 at the models' removable singularities
                approximate=precision == "fp64" and rng.random() < 0.4)


# ------------------------------------------------------------------------------------------ inputs

def _lengths(case):
    lo, hi = case["min_nodes"], case["max_nodes"]
    return np.random.default_rng(17).integers(lo, hi + 1, size=case["fibers"])   # the layout belongs to the case


def _gates(v):
    """Steady states of the Hodgkin-Huxley gates at v."""
    am = 0.1 * (v + 50.0) / -np.expm1(-(v + 50.0) / 10.0)
    an = 0.01 * (v + 65.0) / -np.expm1(-(v + 65.0) / 10.0)
    bm, bn = 4.0 * np.exp(-(v + 75.0) / 18.0), 0.125 * np.exp((v + 75.0) / 80.0)
    ah, bh = 0.07 * np.exp(-(v + 75.0) / 20.0), 1.0 / (np.exp(-(v + 45.0) / 10.0) + 1.0)
    return am / (am + bm), ah / (ah + bh), an / (an + bn)


def _waves(lengths, rng):
    """Vm of all nodes: two pulses of random position, width and height per fiber on the resting potential."""
    n = np.asarray(lengths)
    pos = np.arange(int(n.sum())) - np.repeat(np.cumsum(n) - n, n)
    v = np.zeros(len(pos))
    for _ in range(2):
        c, w = rng.uniform(0, 1, len(n)) * n, rng.uniform(8.0, 60.0, len(n))
        a = rng.uniform(20.0, 105.0, len(n))
        v = np.maximum(v, np.repeat(a, n) * np.exp(-((pos - np.repeat(c, n)) / np.repeat(w, n)) ** 2))
    return v - 74.98


def _fibers(case, seed):
    """The fiber system of a case, its initial states in system.states."""
    rng = np.random.default_rng(seed)
    lengths = _lengths(case)
    n_mus = 100
    firing = (rng.uniform(0, 1, (40, n_mus)) < 0.3).astype(np.uint8)
    firing[0, :2] = (1, 0)
    shorten = case["kind"] == "shorten"
    cm = 0.58 if shorten else workloads.CM
    sigma = rng.uniform(2.5, 5.0, len(lengths))
    s = solver.uniform_fibers(
        workloads.SHORTEN if shorten else workloads.HH, lengths, 0.01, sigma / (workloads.AM * cm),
        firing_events=firing, motor_unit_no=rng.integers(0, n_mus, len(lengths)), call_frequency=0.1,
        repeat_after_first_call=STIMULUS_MS, call_enable_begin=0.0, end_time=case["steps"] * case["dt"],
        dt_0d=case["dt0"], dt_1d=case["dt"], dt_splitting=case["dt"], dt_repeated_call=case["dt"],
        diffusion_scheme=case.get("scheme", "ImplicitEuler"), clamp_rule=case.get("rule", "center"),
        approximate_exponential_function=bool(case.get("approximate", False)))
    if case.get("skip"):
        s.only_compute_if_has_been_stimulated = True
        s.skip_close_to_equilibrium = True
    s.element_lengths = s.element_lengths * rng.uniform(0.95, 1.05, len(s.element_lengths))
    v = _waves(lengths, rng)
    if shorten:
        init = solver.model_sizes(s.model)[3]
        s.states = np.repeat(init[:, None], s.n_nodes, axis=1) * rng.uniform(0.99, 1.01, (len(init), s.n_nodes))
        s.states[0] = v
    else:
        s.states = np.stack([v, *(g * rng.uniform(0.9, 1.0, len(v)) for g in _gates(v))])
        s.parameters = workloads.hh_parameters(s, rng.uniform(0.8, 1.2, len(lengths)),
                                               rng.uniform(0.8, 1.2, len(lengths)))
    return s


def _sensors(case, system):
    idx = np.linspace(0, case["min_nodes"] - 1, case["sensors"]).round().astype(np.int64)
    return (np.asarray(system.fiber_offsets[:-1])[:, None] + idx[None, :]).reshape(-1)


def _emg(case, seed):
    """Vm on the 3D mesh: travelling pulses along z, different on every fiber column, and the box's keywords."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rng = np.random.default_rng(seed)
    _, _, kw = workloads.emg_box(n_fibers_x=1, n_fibers_y=1, n_nodes=10 * (nz - 1) + 1, mesh_nodes=(nx, ny, nz))
    c, w, a = rng.uniform(0, nz, (ny, nx)), rng.uniform(2.0, 8.0, (ny, nx)), rng.uniform(20.0, 105.0, (ny, nx))
    z = np.arange(nz)[:, None, None]
    return -74.98 + a * np.exp(-((z - c) / w) ** 2), kw


def _diffusion(case, seed):
    rng = np.random.default_rng(seed)
    n = _lengths(case)
    off = np.concatenate([[0], np.cumsum(n)])
    return dict(off=off, h=0.01 * rng.uniform(0.95, 1.05, int(off[-1]) - len(n)),
                pf=rng.uniform(2.5, 5.0, len(n)) / workloads.AM, u=_waves(n, rng))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "emg":
        vm, kw = _emg(case, seed)
        bid = emg.StaticBidomainSolver(
            emg_solver={"relativeTolerance": case["rtol"], "absoluteTolerance": 1e-30, "maxIterations": 5000},
            potential_flow_solver={"relativeTolerance": 1e-12, "absoluteTolerance": 1e-30, "maxIterations": 5000},
            initial_guess_nonzero=False, preconditioner=case["preconditioner"], **kw)
        bid.initialize()
        return dict(kind=kind, bid=bid, vm=vm.reshape(-1))
    if kind == "diffusion":
        d = _diffusion(case, seed)
        dev = {k: torch.from_numpy(v).cuda() for k, v in d.items()}
        return dict(kind=kind, dt=case["dt"], scheme=solver.SCHEMES[case["scheme"]],
                    x=torch.empty_like(dev["u"]), **dev)
    system = _fibers(case, seed)
    if kind == "adjoint":
        sensors = _sensors(case, system)
        weight = np.random.default_rng(seed + 1).uniform(-1.0, 1.0, (case["steps"], len(sensors)))
        return dict(kind=kind, engine=adjoint.AdjointEngine(system, sensors, checkpoint_every=case["checkpoint"]),
                    prefactor=torch.from_numpy(np.asarray(system.prefactor)),
                    parameters=torch.from_numpy(system.parameters), weight=torch.from_numpy(weight))
    sv = solver.FastMonodomainSolver(system, method=case["method"], precision=case["precision"])
    sv.initialize()
    initial = sv.pinned_states()
    initial[:] = system.states
    return dict(kind=kind, solver=sv, initial=initial, out=sv.pinned_states(), end=system.end_time)


def run(state):
    kind = state["kind"]
    if kind == "emg":
        bid = state["bid"]
        bid.set_vm(state["vm"])
        bid.advanceTimeSpan()
        return bid.phi_e()
    if kind == "diffusion":
        x = state["x"].copy_(state["u"])
        p = [ctypes.c_void_p(state[k].data_ptr()) for k in ("off", "h", "pf")]
        _native.check(_native.lib().fdm_diffusion_solve(
            len(state["pf"]), len(x), *p, state["dt"], state["scheme"], ctypes.c_void_p(x.data_ptr()),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return x
    if kind == "adjoint":
        prefactor = state["prefactor"].detach().requires_grad_(True)
        parameters = state["parameters"].detach().requires_grad_(True)
        trace = adjoint.strang_trace(prefactor, parameters, state["engine"])
        (trace * state["weight"]).sum().backward()
        return {"trace": trace.detach(), "prefactor": prefactor.grad, "parameters": parameters.grad}
    sv = state["solver"]
    sv.set_states(state["initial"])
    sv.rewind()
    sv.setTimeSpan(0.0, state["end"])
    sv.advanceTimeSpan()
    return sv.states(out=state["out"])


def work(case):
    """Arithmetic of the models' equations (an exponential, logarithm or division counted once) and the
    diffusion solve (13 per node and Strang step), inputs read and outputs written once."""
    kind = case["kind"]
    if kind == "emg":
        # K(sigma_i) Vm and one application of K(sigma_i + sigma_e), 27 entries each; Vm in, phi_e out
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 16 * n, "flops": 4 * 27 * n}
    n = int(_lengths(case).sum())
    if kind == "diffusion":
        return {"bytes": 24 * n, "flops": 40 * n}
    states, ops, params = (56, 1251, 2) if kind == "shorten" else (4, 61, 3)
    substeps = 2 * round(0.5 * case["dt"] / case["dt0"]) * case["steps"]
    flops = n * (substeps * (2 * ops + 5 * states) + 13 * case["steps"])
    if kind == "adjoint":
        # the reverse of a step at least twice the step; parameters in, their gradients out
        return {"bytes": 8 * n * (states + 2 * params), "flops": 3 * flops}
    return {"bytes": 16 * n * states + 8 * n * params, "flops": flops}


# ------------------------------------------------------------------------- the same in 64-bit torch

def _pad(lengths, device):
    """Index of every node in a [fiber, longest fiber] array, and the mask of real nodes."""
    n = torch.as_tensor(np.asarray(lengths), device=device)
    mask = torch.arange(int(n.max()), device=device)[None, :] < n[:, None]
    return mask.reshape(-1).nonzero()[:, 0], mask


def _shift(x, k):
    """x[:, i - k] (k > 0) or x[:, i + |k|] (k < 0), zero outside."""
    if abs(k) >= x.shape[1]:
        return torch.zeros_like(x)
    return torch.nn.functional.pad(x[:, :-k], (k, 0)) if k > 0 else torch.nn.functional.pad(x[:, -k:], (0, -k))


class _Diffusion:
    """(K - M/dt) x = -M/dt u (implicit Euler) or its Crank-Nicolson form, by parallel cyclic reduction."""

    def __init__(self, mask, h, pf, dt, scheme):
        right = mask & _shift(mask.double(), -1).bool()
        hr = torch.where(right, h, torch.ones_like(h))
        zero = torch.zeros_like(h)
        k = torch.where(right, pf[:, None] / hr, zero)      # element to the right of a node
        m = torch.where(right, h / dt, zero)
        theta = 1.0 if scheme == "ImplicitEuler" else 0.5
        kl, ml = _shift(k, 1), _shift(m, 1)
        a, c = theta * kl - ml / 6, theta * k - m / 6
        b = torch.where(mask, -theta * (kl + k) - (ml + m) / 3, torch.ones_like(h))
        self.l, self.r = -(1 - theta) * kl - ml / 6, -(1 - theta) * k - m / 6
        self.m = (1 - theta) * (kl + k) - (ml + m) / 3
        self.levels, step = [], 1
        while step < h.shape[1]:
            # beyond the ends of the array the diagonal is taken as 1: the entries there are zero
            bl = _shift(b - 1, step) + 1
            br = _shift(b - 1, -step) + 1
            al, ga = -a / bl, -c / br
            self.levels.append((step, al, ga))
            b, a, c = (b + al * _shift(c, step) + ga * _shift(a, -step), al * _shift(a, step), ga * _shift(c, -step))
            step *= 2
        self.b = b

    def __call__(self, u):
        d = self.l * _shift(u, 1) + self.m * u + self.r * _shift(u, -1)
        for step, al, ga in self.levels:
            d = d + al * _shift(d, step) + ga * _shift(d, -step)
        return d / self.b


def _approximate_exp(x):
    y = 1.0 + x / 1024.0
    for _ in range(10):
        y = y * y
    return y


def _hh(exp, p, v, m, h, n):
    i_stim, g_na, g_k = p
    am = -0.1 * (v + 50.0) / (exp(-(v + 50.0) / 10.0) - 1.0)
    bm = 4.0 * exp(-(v + 75.0) / 18.0)
    ah = 0.07 * exp(-(v + 75.0) / 20.0)
    bh = 1.0 / (exp(-(v + 45.0) / 10.0) + 1.0)
    an = -0.01 * (v + 65.0) / (exp(-(v + 65.0) / 10.0) - 1.0)
    bn = 0.125 * exp((v + 75.0) / 80.0)
    current = g_na * m ** 3 * h * (v - 40.0) + g_k * n ** 4 * (v + 87.0) + 0.3 * (v + 64.387)
    return i_stim - current, am * (1 - m) - bm * m, ah * (1 - h) - bh * h, an * (1 - n) - bn * n


def _strang(case, system, device):
    """Step function of the fiber system over padded arrays, its initial states and parameters."""
    lengths = np.diff(np.asarray(system.fiber_offsets))
    index, mask = _pad(lengths, device)

    def padded(x):
        out = torch.zeros(mask.numel(), dtype=torch.float64, device=device)
        out[index] = torch.as_tensor(np.ascontiguousarray(x), device=device)
        return out.reshape(mask.shape)

    # element i lies to the right of node i: the last node of a fiber has none
    h = np.zeros(system.n_nodes)
    h[np.delete(np.arange(system.n_nodes), np.cumsum(lengths) - 1)] = system.element_lengths
    h = padded(h)
    centre = np.asarray(system.stimulation_point_index)
    if case.get("rule", "center") == "center":
        first = np.maximum(centre - 1, 0)
        junction = [first + k for k in range(3)]
    else:   # the first three lanes of the buffer of four nodes (counted over all fibers) that holds the centre
        start = np.cumsum(lengths) - lengths
        first = (start + centre) // 4 * 4 - start
        junction = [first + k for k in range(3)]
    mu = np.asarray(system.motor_unit_no) % system.firing_events.shape[1]
    fires = np.asarray(system.firing_events)[0, mu] != 0
    clamp = np.zeros(mask.shape, bool)
    for j in junction:
        ok = fires & (j >= 0) & (j < lengths)
        clamp[np.nonzero(ok)[0], j[ok]] = True
    clamp = torch.as_tensor(clamp, device=device) & mask
    exp = _approximate_exp if case.get("approximate") else torch.exp
    n0 = round(0.5 * case["dt"] / case["dt0"])
    dt0 = 0.5 * case["dt"] / n0

    def half(y, p, t0):
        for k in range(n0):
            held = t0 + k * dt0 < STIMULUS_MS - 5e-14
            f = _hh(exp, p, *y)
            ys = [a + dt0 * b for a, b in zip(y, f)]
            if held:
                ys[0] = torch.where(clamp, 20.0, ys[0])
            g = _hh(exp, p, *ys)
            y = [a + 0.5 * dt0 * (b + c) for a, b, c in zip(y, f, g)]
            if held:
                y[0] = torch.where(clamp, 20.0, y[0])
        return y

    def step(solve, p, t, *y):
        y = half(list(y), p, t)
        y[0] = solve(torch.where(mask, y[0], torch.zeros_like(y[0])))
        return tuple(half(y, p, t + 0.5 * case["dt"]))

    return step, [padded(s) for s in system.states], [padded(s) for s in system.parameters], h, mask, index


def _exact_adjoint(case, seed, system, device):
    step, y, p, h, mask, index = _strang(case, system, device)
    pf = torch.as_tensor(np.asarray(system.prefactor), device=device).requires_grad_(True)
    p = [q.requires_grad_(True) for q in p]
    solve = _Diffusion(mask, h, pf, case["dt"], system.diffusion_scheme)
    sensors = index[torch.as_tensor(_sensors(case, system), device=device)]
    weight = np.random.default_rng(seed + 1).uniform(-1.0, 1.0, (case["steps"], len(sensors)))
    trace = []
    for j in range(case["steps"]):
        y = torch.utils.checkpoint.checkpoint(
            lambda t, *z: step(solve, p, t, *z), j * case["dt"], *y, use_reentrant=False)
        trace.append(y[0].reshape(-1)[sensors])
    trace = torch.stack(trace)
    (trace * torch.as_tensor(weight, device=device)).sum().backward()
    return {"trace": trace.detach().cpu(), "prefactor": pf.grad.cpu(),
            "parameters": torch.stack([q.grad.reshape(-1)[index] for q in p]).cpu()}


def _exact_emg(case, seed, device):
    """The box's stiffness matrices are sums of Kronecker products of the one-dimensional ones: solved directly
    in the generalized eigenvectors of (stiffness, mass) of the three directions."""
    vm, kw = _emg(case, seed)
    pos = kw["node_positions"].reshape(case["nz"], case["ny"], case["nx"], 3)
    axes = (pos[:, 0, 0, 2], pos[0, :, 0, 1], pos[0, 0, :, 0])      # z, y, x as the arrays are indexed
    along_i, across_i = kw["sigma_i"][0], kw["sigma_i"][4]
    along_e, across_e = kw["sigma_e"][0], kw["sigma_e"][4]
    mats = []
    for x in axes:
        d = torch.as_tensor(np.diff(x), device=device)
        n = len(x)
        k, m = (torch.zeros(n, n, dtype=torch.float64, device=device) for _ in range(2))
        i = torch.arange(n - 1, device=device)
        for q, off, same in ((k, -1.0 / d, 1.0 / d), (m, d / 6, d / 3)):
            q[i, i + 1] = off
            q[i + 1, i] = off
            q[i, i] += same
            q[i + 1, i + 1] += same
        low = torch.linalg.cholesky(m)
        t = torch.linalg.solve_triangular(low, k, upper=False)
        t = torch.linalg.solve_triangular(low, t.T, upper=False)
        lam, q = torch.linalg.eigh(0.5 * (t + t.T))
        mats.append((k, m, lam, torch.linalg.solve_triangular(low.T, q, upper=True)))

    def apply(a, b, c, x):
        x = (a @ x.reshape(x.shape[0], -1)).reshape(-1, x.shape[1], x.shape[2])
        return b @ (x @ c.T)

    v = torch.as_tensor(vm, device=device)
    (kz, mz, lz, qz), (ky, my, ly, qy), (kx, mx, lx, qx) = mats
    rhs = -(along_i * apply(kz, my, mx, v) + across_i * (apply(mz, ky, mx, v) + apply(mz, my, kx, v)))
    lam = (along_i + along_e) * lz[:, None, None] + (across_i + across_e) * (ly[None, :, None] + lx[None, None, :])
    y = apply(qz.T, qy.T, qx.T, rhs)
    y = torch.where(lam > 1e-9 * lam.max(), y / lam, torch.zeros_like(y))
    phi = apply(qz, qy, qx, y).reshape(-1)
    return (phi - phi.mean()).cpu().numpy()


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind == "shorten" or case.get("skip"):
        return None     # 56 states, and the skipped buffers: no short restatement
    if kind == "emg":
        return _exact_emg(case, seed, device)
    if kind == "diffusion":
        d = _diffusion(case, seed)
        index, mask = _pad(np.diff(d["off"]), device)
        h, u = (torch.zeros(mask.numel(), dtype=torch.float64, device=device) for _ in range(2))
        u[index] = torch.as_tensor(d["u"], device=device)
        h[index[torch.as_tensor(np.delete(np.arange(len(d["u"])), d["off"][1:] - 1), device=device)]] = \
            torch.as_tensor(d["h"], device=device)
        pf = torch.as_tensor(d["pf"], device=device)
        x = _Diffusion(mask, h.reshape(mask.shape), pf, case["dt"], case["scheme"])(u.reshape(mask.shape))
        return x.reshape(-1)[index].cpu()
    system = _fibers(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, seed, system, device)
    step, y, p, h, mask, index = _strang(case, system, device)
    pf = torch.as_tensor(np.asarray(system.prefactor), device=device)
    solve = _Diffusion(mask, h, pf, case["dt"], system.diffusion_scheme)
    with torch.no_grad():
        for j in range(case["steps"]):
            y = step(solve, p, j * case["dt"], *y)
    return torch.stack([q.reshape(-1)[index] for q in y]).cpu().numpy()
