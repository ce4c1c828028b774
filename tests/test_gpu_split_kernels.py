"""The split path's kernels at the sizes where their work partition changes: the stimulation schedule (a warp per
fiber, 32 substeps at a time), the factorization (chunks started speculatively, tiles) and the diffusion solves."""
import ctypes as C

import numpy as np
import pytest
import torch

import helpers as H
from oracle import oracle as O
from opendihu_b200 import _native as N
from opendihu_b200 import solver as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frequency,repeat,dt0,steps", [
    (900.0, 3e-4, 1e-4, 33),      # phases of a few substeps: several begin and end within one word of 32 bits
    (5000.0, 1e-4, 1e-4, 7),      # a phase ends at almost every substep; 70 bits: a last word of 6
    (40.0, 1e-2, 1.6e-5, 5),      # 31 substeps per half step: words that straddle half steps
    (10.0, 0.05, 5e-4, 64),       # one substep per half step, exactly four words
])
def test_schedule_word_edges(frequency, repeat, dt0, steps):
    rng = np.random.default_rng(3)
    s = S.uniform_fibers(H.HH, [40, 64, 33], 0.01, 3.828 / 500, call_frequency=frequency,
                         repeat_after_first_call=repeat, call_enable_begin=0.0, end_time=steps * 1e-3, dt_0d=dt0,
                         dt_1d=1e-3, dt_splitting=1e-3, dt_repeated_call=1e-3, clamp_rule="center")
    s.firing_events = (rng.random((7, 2)) < 0.7).astype(np.uint8)
    s.motor_unit_no = np.array([0, 1, 0], np.int32)
    s.jitter = rng.uniform(-0.3, 0.3, (3, 4))
    s.call_enable_begin = np.array([0.0, 0.002, 0.0])
    s = H.complete(s)
    spec = H.oracle_spec(s.copy(), n_threads=1)
    spec["log_capacity"] = 20000
    run = O.OracleRun(spec)
    ref = np.ascontiguousarray(s.states, np.float64).copy()
    run.run(ref)
    t, f, lost = run.stimulation_log()
    order = np.lexsort((f, t))
    assert lost == 0 and len(t) >= 2
    for per_launch in (1, 3, 100):
        with S.FastMonodomainSolver(s.copy(), method="split", precision="fp64", steps_per_launch=per_launch) as slv:
            slv.enable_stimulation_log()
            slv.advanceTimeSpan()
            log = slv.stimulation_log()
            vm = slv.vm()
        np.testing.assert_array_equal(log["time"], t[order])
        np.testing.assert_array_equal(log["fiber"], f[order])
        # every clamp decision equal: FP64 Vm within rounding of the oracle's
        assert np.max(np.abs(vm - ref[0])) < 1e-8


def _tridiagonal(h, pf, dt, scheme, u):
    """One diffusion solve by dense elimination: (K - M/dt) x = -M/dt u or its Crank-Nicolson form."""
    n = len(h) + 1
    K, M = np.zeros((n, n)), np.zeros((n, n))
    for e, he in enumerate(h):
        K[e:e + 2, e:e + 2] += pf / he * np.array([[-1.0, 1.0], [1.0, -1.0]])
        M[e:e + 2, e:e + 2] += he / 6 * np.array([[2.0, 1.0], [1.0, 2.0]])
    if scheme == "ImplicitEuler":
        return np.linalg.solve(K - M / dt, -M / dt @ u)
    return np.linalg.solve(K / 2 - M / dt, (-K / 2 - M / dt) @ u)


# lengths around the chunks (a warm-up of 12 nodes), the 256 threads and the tile of 2560 nodes; dt = 10 couples the
# nodes so strongly that no chunk's guess is right and the rounds run
@pytest.mark.parametrize("lengths", [[2, 3, 12, 13, 14, 101], [255, 256, 257, 511, 512, 513], [2559, 2560, 2561],
                                     [5120, 5200]])
@pytest.mark.parametrize("scheme", ["ImplicitEuler", "CrankNicolson"])
@pytest.mark.parametrize("dt", [1e-3, 10.0])
def test_diffusion_operator(lengths, scheme, dt):
    rng = np.random.default_rng(5)
    off = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    h = 0.01 * rng.uniform(0.8, 1.2, off[-1] - len(lengths))
    pf = rng.uniform(2.5, 5.0, len(lengths)) / 500
    u = rng.uniform(-80.0, 40.0, off[-1])
    ref = np.concatenate([_tridiagonal(h[off[f] - f:off[f + 1] - f - 1], pf[f], dt, scheme, u[off[f]:off[f + 1]])
                          for f in range(len(lengths))])
    dev = [torch.from_numpy(x).cuda() for x in (off, h, pf)]
    for entry in ("fdm_diffusion_solve", "fdm_diffusion_solve_noalloc"):
        x = torch.from_numpy(u.copy()).cuda()
        N.check(getattr(N.lib(), entry)(len(lengths), len(u), *[C.c_void_p(d.data_ptr()) for d in dev], dt,
                                        S.SCHEMES[scheme], C.c_void_p(x.data_ptr()), None))
        torch.cuda.synchronize()
        # condition number: at most 4 pf/h dt / (h/3) + 3, about 2e4 at dt = 10; 100 roundings of it
        assert np.max(np.abs(x.cpu().numpy() - ref)) < 80 * 2.3e-16 * 100 * max(1.0, 2e3 * dt)


@pytest.mark.parametrize("lengths", [[41] * 600, [40 + k % 89 for k in range(600)], [40 + k % 217 for k in range(600)],
                                     [257 + k % 40 for k in range(595)], [2, 511, 512, 513], [1024, 1025, 1537, 2049], [2560], [2561, 40], [2570] * 592])
def test_split_diffusion_partitions(lengths):
    s = S.uniform_fibers(H.HH, lengths, 0.01, 3.828 / 500, call_frequency=0.1, repeat_after_first_call=0.1,
                         call_enable_begin=0.0, end_time=2e-3, dt_0d=5e-4, dt_1d=1e-3, dt_splitting=1e-3,
                         dt_repeated_call=1e-3, clamp_rule="center", diffusion_scheme="CrankNicolson")
    rng = np.random.default_rng(1)
    s = H.complete(s)
    s.states = s.states.copy()
    s.states[0] += rng.uniform(0.0, 60.0, s.n_nodes)
    ref = H.run_oracle(s.copy())[0]
    with S.FastMonodomainSolver(s.copy(), method="split", precision="fp64") as slv:
        slv.advanceTimeSpan()
        got = slv.states()
    assert np.max(np.abs(got - ref)) < 1e-9


# lane widths that divide the warp (tested and scanned in the reaction kernel) and that do not (kernels of their own);
# 5 fibers of 30 to 61 nodes, and enough nodes for several blocks of the scan
@pytest.mark.parametrize("width,scale", [(1, 1), (2, 1), (3, 1), (5, 1), (16, 1), (4, 12), (3, 12), (8, 12)])
def test_equilibrium_lane_widths(width, scale):
    import test_gpu_equilibrium as EQ
    from opendihu_b200 import workloads as WL
    s = WL.batched_hh(clamp_rule="vc", n_fibers=5, min_nodes=30 * scale, max_nodes=61 * scale, seed=5, end_time=0.3,
                      diffusion_scheme="ImplicitEuler", n_ranks=2, vc_width=width)
    s.firing_events = np.array([[1, 0, 1, 1, 0]], np.uint8)
    s.motor_unit_no = np.arange(5, dtype=np.int32)
    H.complete(s)
    s.states = np.repeat(EQ._rest()[:, None], s.n_nodes, axis=1)
    s.skip_close_to_equilibrium = True
    ref, ref_status, ref_counter, _ = EQ._oracle(s)
    with S.FastMonodomainSolver(s.copy(), method="split", precision="fp64", steps_per_launch=7) as slv:
        slv.advanceTimeSpan()
        st = slv.states()
        status, counter = slv.equilibrium_state()
    assert np.max(np.abs(st - ref)) < 1e-8
    np.testing.assert_array_equal(status, ref_status)
    np.testing.assert_array_equal(counter, ref_counter)


# fused, a fiber over the CTAs of a cluster: with the usual step the halos carry the sweeps across the CTAs, with a step
# of 0.1 ms (0.75 per node and sweep) they cannot and the scan totals are exchanged; fibers that end inside a CTA, at
# its end and inside a neighbour's halo
@pytest.mark.parametrize("dt", [1e-3, 0.1])
@pytest.mark.parametrize("threads,per_thread", [(128, 2), (192, 1)])
def test_cluster_halos(dt, threads, per_thread):
    cap = threads * per_thread
    s = S.uniform_fibers(H.HH, [cap * 3, cap * 2, cap * 2 + 1, cap + 5, cap - 1, 2], 0.01, 3.828 / 500,
                         call_frequency=0.1, repeat_after_first_call=0.1, call_enable_begin=0.0, end_time=4 * dt,
                         dt_0d=dt / 10, dt_1d=dt, dt_splitting=dt, dt_repeated_call=dt, clamp_rule="center",
                         diffusion_scheme="CrankNicolson")
    s = H.complete(s)
    s.states = s.states.copy()
    s.states[0] += np.random.default_rng(2).uniform(0.0, 40.0, s.n_nodes)
    ref = H.run_oracle(s.copy())[0]
    for precision, tol in (("fp64", (1e-8, 1e-8)), ("fp32", (0.1, 1e-3))):   # FP32: the mode's accuracy contract
        with S.FastMonodomainSolver(s.copy(), method="fused", precision=precision, threads_per_block=threads,
                                    nodes_per_thread=per_thread, cluster_size=3, steps_per_launch=3) as slv:
            slv.advanceTimeSpan()
            got = slv.states()
        assert np.max(np.abs(got[0] - ref[0])) < tol[0] and np.max(np.abs(got[1:] - ref[1:])) < tol[1]


# whole windows in one launch (few fibers: at most 2048 nodes, clusters of 1 to 8 CTAs with an SM each): one to eight
# CTAs, nodes per CTA from 2 to 256, fibers shorter than the cluster's first CTA, the last number of fibers that still
# fits 8 and 1 CTAs ("8" and "1") and the first that does not, 2049 nodes (a launch per half step and solve); windows of
# 1, 7, 20 steps.  The forms give the same values, bit for bit, so that a fiber's do not depend on how many others there
# are.
@pytest.mark.parametrize("lengths", [[2], [3, 2], [128], [129], [256, 257], [1481], [2048, 2, 255, 1024, 1025],
                                     ("8", 0, 1024), ("8", 1, 1024), ("8", 1, 2041), ("1", 0, 100), ("1", 1, 100), [2049, 40]])
@pytest.mark.parametrize("approximate", [False, True])
def test_window_partitions(lengths, approximate):
    if isinstance(lengths, tuple):
        csize, beyond, nodes = lengths
        lengths = [nodes] * (N.lib().fdm_resident_clusters(0, int(csize)) + beyond)
    rng = np.random.default_rng(7)
    s = S.uniform_fibers(H.HH, lengths, 0.01, 3.828 / 500, call_frequency=0.5, repeat_after_first_call=0.1,
                         call_enable_begin=0.0, end_time=0.02, dt_0d=2e-4, dt_1d=1e-3, dt_splitting=1e-3,
                         dt_repeated_call=1e-3, clamp_rule="center", approximate_exponential_function=approximate,
                         algebraics_for_transfer=[0, 4, 8])
    s = H.complete(s)
    s.states = s.states.copy()
    s.states[0] += rng.uniform(0.0, 40.0, s.n_nodes)
    ref = H.run_oracle(s.copy())[0]
    nodes = sorted({0, s.n_nodes // 2, s.n_nodes - 1})
    first = None
    # with profiling the same steps run as a launch per half step and solve
    for profile, per_launch in ((True, 0), (False, 0), (False, 1), (False, 7)):
        with S.FastMonodomainSolver(s.copy(), method="split", precision="fp64", profile=profile,
                                    steps_per_launch=per_launch, trace_nodes=nodes, trace_capacity=20) as slv:
            slv.advanceTimeSpan()
            values = slv.states(), slv.algebraics(), slv.trace()
        # 400 right-hand sides: roundings of 1e-14 of Vm and, with the approximate exponential, its 1024th power's 1e-13
        assert np.max(np.abs(values[0] - ref)) < 1e-8
        first = first or values
        for v, v0 in zip(values, first):
            np.testing.assert_array_equal(v, v0)


# the reverse diffusion with a fiber per CTA: 128 x 4, 256 x 4, 256 x 6, 256 x 8, 512 x 8 nodes and one node more; against
# central differences in each fiber's conductivity
@pytest.mark.parametrize("n_nodes", [512, 513, 1024, 1025, 1536, 1537, 2048, 2049])
@pytest.mark.parametrize("scheme", ["ImplicitEuler", "CrankNicolson"])
def test_adjoint_diffusion_shapes(n_nodes, scheme):
    from opendihu_b200 import adjoint as ADJ
    from opendihu_b200 import workloads as WL
    s = H.complete(H.c1_system(n_fibers=2, n_nodes=n_nodes, end_time=0.02, diffusion_scheme=scheme))
    s.states = s.states.copy()
    s.states[0] += np.random.default_rng(6).uniform(0.0, 40.0, s.n_nodes)
    sensors = np.array([0, n_nodes // 2, n_nodes - 1, n_nodes, 2 * n_nodes - 1])
    pf = np.array([3.0, 4.5]) / 500
    s.prefactor = pf.copy()
    s.parameters = WL.hh_parameters(s, np.ones(2), np.ones(2))
    eng = ADJ.AdjointEngine(s, sensors, checkpoint_every=7)
    try:
        trace = eng.forward(pf, s.parameters)
        w = np.random.default_rng(8).standard_normal(np.shape(trace))
        g = eng.backward(w)["prefactor"]
        for f in range(2):
            e = np.zeros(2)
            e[f] = 1e-5 * pf[f]
            d = (np.sum(w * eng.forward(pf + e, s.parameters)) - np.sum(w * eng.forward(pf - e, s.parameters))) / 2e-5
            # the loss is rounded at 1e-13 of some 1e3, the difference quotient at 1e-10 / 1e-5
            assert abs(g[f] * pf[f] - d) < 1e-4 + 1e-5 * abs(d)
    finally:
        eng.close()
