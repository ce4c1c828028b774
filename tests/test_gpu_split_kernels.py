"""The split path's kernels at the sizes where their work partition changes: the stimulation schedule (a warp per
fiber, 32 substeps at a time)."""
import numpy as np
import pytest

import helpers as H
from oracle import oracle as O
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
