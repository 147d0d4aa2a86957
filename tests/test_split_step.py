"""Read-outs of the slot fields, inside a step opened with aprl_run_step_begin
too: the trials issued ahead are in flight, and those after the converged one do
nothing.  In the bit-reproducible mode the same step through the seams gives the
same bits."""
import numpy as np
import pytest

import checkers
from aprl_b200 import native, workloads

pytestmark = pytest.mark.gpu


def converged(cfg, trial, residual):
    force, defect, scale, calls = residual
    work = 0.0 if calls == 0 else (defect / scale if scale > 0 else defect)
    return (trial >= (2 if calls else 1) and force < cfg.force_tolerance
            and work < cfg.work_tolerance)


@pytest.mark.parametrize("trials", [2, 3])
def test_slot_fields_inside_an_open_step(trials):
    """trials 2: one of the three trials issued ahead does not run."""
    w = workloads.small_case(steps=4)
    cfg = w.config = workloads.with_determinism(w.config)
    if trials == 2:
        cfg.force_tolerance = cfg.work_tolerance = 0.5
    split = native.Run(native.load(), cfg).load_workload(w)
    seams = native.Run(native.load(), cfg).load_workload(w)
    for _ in range(4):
        split.step_begin()
        seams.advance_magnetic()
        seams.preview_electric()
        trial = 1
        while not converged(cfg, trial, seams.coupling_trial()):
            trial += 1
        assert trial == trials
        expected = seams.slot_fields()
        inside = split.slot_fields()
        split.step_end()
        after = split.slot_fields()
        for k in expected:
            np.testing.assert_array_equal(inside[k], expected[k], err_msg=k)
            np.testing.assert_array_equal(after[k], expected[k], err_msg=k)
        assert np.any(expected["used_e"] != expected["next_e"])
        seams.commit_electric()
        seams.shift()
        assert split.stats()["iterations"] == trials


@pytest.mark.parametrize("shape", ["linear-binomial3", "quintic-compensated"])
def test_slots_without_a_push_read_zero(shape):
    """beginStep resets every slot, and a held particle's is not pushed.  The
    memory is first given to a run whose slots all hold fields."""
    full = native.Run(native.load(), (w := workloads.small_case(particles=2000)).config)
    full.load_workload(w).step(1)
    full.close()
    w = workloads.streaming_case(steps=4, particles=900, shape=shape)
    g = native.Run(native.load(), w.config).load_workload(w)
    o = checkers.run(checkers.oracle(), w)
    for r in (g, o):
        r.advance_magnetic()
        r.preview_electric()
    for _ in range(3):
        g.coupling_trial()
        o.coupling_trial()
        got, expected = g.slot_fields(), o.slot_fields()
        idle = ~np.any(expected["used_b"] != 0.0, axis=1)
        assert idle.any() and not idle.all()
        for k in expected:
            assert not np.any(got[k][idle]), k
            assert checkers.max_relative(got[k], expected[k]) <= 1e-12, k
