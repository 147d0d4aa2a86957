"""Read-outs inside a step opened with aprl_run_step_begin: the trials issued
ahead are in flight, and those after the converged one do nothing.  In the
bit-reproducible mode the same step through the seams gives the same bits."""
import numpy as np
import pytest

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
