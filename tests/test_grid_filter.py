"""The grid-side filter of the particle shapes against the oracle.

Particles deposit narrow weights into a raw current and gather from filtered
arrays; the filter passes work in x tiles of 28 and 30 nodes, z chunks of 8 to
32 planes and columns marked by the deposits, and a sparse linear-binomial3 run
(under one particle per 24 cells) reads the wide stencils directly in its first
trial.  The extents below put the last tile, the last chunk and the ring's wrap
at their edges, on either side of the sparse rule, and the read-out of J
applies the filter on its own.  Bound: the terms are the oracle's in another
order, so each array agrees to 1e-12 of its largest magnitude, as in the other
step tests.
"""
import numpy as np
import pytest

import checkers
from aprl_b200 import native, workloads

pytestmark = pytest.mark.gpu
RTOL = 1e-12

EXTENTS = [  # nx, ny, nz, particles
    (27, 17, 16, 60),    # sparse; nx + 3 = 30
    (28, 18, 31, 900),   # dense; Jy rows one past a 28-node tile
    (29, 20, 33, 1200),
    (30, 19, 63, 2500),
    (61, 16, 25, 400),   # sparse; three tiles
]


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("shape", ["linear-binomial3", "quintic-compensated"])
@pytest.mark.parametrize("nx,ny,nz,particles", EXTENTS)
def test_steps_match_oracle(nx, ny, nz, particles, shape, deterministic):
    w = workloads.small_case(nx=nx, ny=ny, nz=nz, particles=particles, steps=3, shape=shape)
    w.config = workloads.with_determinism(w.config, deterministic)
    g = native.Run(native.load(), w.config).load_workload(w)
    o = checkers.run(checkers.oracle(), w)
    for _ in range(3):
        g.step(1)
        o.step(1)
        for a in range(6):
            assert checkers.max_relative(g.get_field(a), o.get_field(a)) <= RTOL, a
    assert g.stats()["iterations"] == o.stats()["iterations"]


def test_current_read_out_between_trials():
    """J read after each trial of the seams, then the trials go on."""
    w = workloads.small_case(nx=30, ny=18, nz=33, particles=1500, steps=2)
    g = native.Run(native.load(), w.config).load_workload(w)
    o = checkers.run(checkers.oracle(), w)
    for r in (g, o):
        r.advance_magnetic()
        r.preview_electric()
    for _ in range(3):
        g.coupling_trial()
        o.coupling_trial()
        for a in range(6, 9):
            assert checkers.max_relative(g.get_field(a), o.get_field(a)) <= RTOL, a
    for r in (g, o):
        r.commit_electric()
        r.shift()
    for a in range(6):
        assert checkers.max_relative(g.get_field(a), o.get_field(a)) <= RTOL, a


def test_set_current_is_read_back_until_the_next_step():
    w = workloads.small_case(steps=2)
    g = native.Run(native.load(), w.config).load_workload(w)
    value = np.random.default_rng(3).standard_normal(g.get_field(8).shape)
    g.set_field(8, value)
    np.testing.assert_array_equal(g.get_field(8), value)
    g.advance_magnetic()
    assert not np.any(g.get_field(8))


@pytest.mark.parametrize("shape", ["linear-binomial3", "quintic-compensated"])
def test_whole_steps_equal_the_seams(shape):
    """Whole steps crop the carriers inside the trial and swap arrays instead
    of copying them; the seams leave the crop to the shift.  In the
    bit-reproducible mode both give the same bits and counters."""
    w = workloads.small_case(nx=32, ny=24, nz=60, particles=3000, steps=8, shape=shape,
                             z_fraction=(0.02, 0.99), margin_cells=1)
    cfg = w.config = workloads.with_determinism(w.config)
    whole = native.Run(native.load(), cfg).load_workload(w)
    seams = native.Run(native.load(), cfg).load_workload(w)
    for _ in range(8):
        whole.step(1)
        seams.advance_magnetic()
        seams.preview_electric()
        for trial in range(1, cfg.max_trials + 1):
            force, defect, scale, calls = seams.coupling_trial()
            work = 0.0 if calls == 0 else (defect / scale if scale > 0 else defect)
            if trial >= (2 if calls else 1) and force < cfg.force_tolerance and \
                    work < cfg.work_tolerance:
                break
        seams.commit_electric()
        seams.shift()
    a, b = checkers.state(whole), checkers.state(seams)
    for x, y in zip(a["fields"] + a["histories"], b["fields"] + b["histories"]):
        np.testing.assert_array_equal(x, y)
    for group in ("particles", "carriers"):
        for k in a[group]:
            np.testing.assert_array_equal(a[group][k], b[group][k])
    for k in ("particles", "carriers", "exits", "cpml_entries", "cropped_carriers"):
        assert a["stats"][k] == b["stats"][k], k
    assert a["stats"]["cropped_carriers"] > 0
