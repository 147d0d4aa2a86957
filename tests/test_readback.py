"""Uploads and read-outs: ring-ordered fields and histories in two runs of
planes, particles ordered on the device, and large copies driven by several
threads over page-locked lanes.  Everything is a copy, so equality is exact."""
import subprocess
import sys
import threading

import numpy as np
import pytest

import checkers
from aprl_b200 import native, workloads

pytestmark = pytest.mark.gpu


def large_case():
    # 96 x 80 x 96 cells: 6 MB a component, above the size that is staged
    return workloads.small_case(nx=96, ny=80, nz=96, particles=120_000, steps=6, fields=False)


def test_fields_histories_and_particles_round_trip():
    w = large_case()
    r = native.Run(native.load(), w.config)
    r.set_reference(w.reference)
    r.set_particles(w.particles)
    got = r.get_particles()
    for k in ("x", "y", "z", "ux", "uy", "uz", "charge", "mass", "id"):
        np.testing.assert_array_equal(got[k], w.particles[k])
    rng = np.random.default_rng(1)
    for steps in (0, 3):  # the ring's base at zero, then moved
        if steps:
            r.step(steps)
            ids = r.get_particles()["id"]
            rank = {v: n for n, v in enumerate(w.particles["id"].tolist())}
            order = np.array([rank[v] for v in ids.tolist()])
            assert np.all(np.diff(order) > 0)
        for a in range(6):
            value = rng.standard_normal(r.get_field(a).shape)
            r.set_field(a, value)
            np.testing.assert_array_equal(r.get_field(a), value)
        for h in (0, 3, 9, 11):
            value = rng.standard_normal(r.history_length(h))
            r.set_history(h, value)
            np.testing.assert_array_equal(r.get_history(h), value)


def test_non_finite_reference_is_refused_and_the_table_kept():
    w = large_case()
    w.config.reference_nz = 120
    table = workloads.synthetic_reference(w.config)
    r = native.Run(native.load(), w.config)
    r.set_reference(table)
    bad = table[2].copy()
    bad[-1, -1, -1] = np.inf
    with pytest.raises(native.AprlError, match="Non-finite moving-window inlet"):
        r.set_reference(table[:2] + [bad] + table[3:])
    np.testing.assert_array_equal(r.get_reference(2), table[2])


def test_concurrent_callers_share_the_lanes():
    w = large_case()
    runs = []
    for _ in range(3):
        r = native.Run(native.load(), w.config)
        r.set_reference(w.reference)
        runs.append(r)
    failed = []

    def work(r, seed):
        try:
            rng = np.random.default_rng(seed)
            for _ in range(3):
                r.set_particles(w.particles)
                value = rng.standard_normal(r.get_field(1).shape)
                r.set_field(1, value)
                if not np.array_equal(r.get_field(1), value):
                    failed.append("field")
                if not np.array_equal(r.get_particles()["z"], w.particles["z"]):
                    failed.append("particles")
        except Exception as e:  # noqa: BLE001
            failed.append(repr(e))

    threads = [threading.Thread(target=work, args=(r, n)) for n, r in enumerate(runs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


def test_page_locked_memory_round_trip():
    """Memory the driver knows is left to it, at any size."""
    torch = pytest.importorskip("torch")
    w = large_case()
    r = native.Run(native.load(), w.config)
    r.set_reference(w.reference)
    value = np.random.default_rng(5).standard_normal(r.get_field(0).shape)
    locked = torch.from_numpy(value).pin_memory().numpy()
    r.set_field(0, locked)
    out = torch.empty(value.shape, dtype=torch.float64).pin_memory().numpy()
    r.b("run_get_field", r.handle, 0, native._ptr(out), out.size)
    np.testing.assert_array_equal(out, value)
    np.testing.assert_array_equal(r.get_field(0), value)


def test_a_device_pointer_does_not_end_the_process():
    """A read-out into a device pointer is the driver's to refuse (or to copy,
    where it takes the pointer's own word for its place)."""
    code = f"""
import ctypes, sys
sys.path[:0] = [{checkers.REPO!r}, {checkers.REPO + "/tests"!r}]
import torch
import test_readback
from aprl_b200 import native
w = test_readback.large_case()
r = native.Run(native.load(), w.config)
r.set_reference(w.reference)
t = torch.zeros(r.get_field(0).shape, dtype=torch.float64, device="cuda")
p = ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))
try:
    r.b("run_get_field", r.handle, 0, p, t.numel())
    print("copied")
except native.AprlError as e:
    print("refused")
torch.cuda.synchronize()
"""
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    assert out.stdout.split() in (["refused"], ["copied"])


def test_copies_from_a_thread_on_another_device():
    torch = pytest.importorskip("torch")
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    w = large_case()
    with torch.cuda.device(1):
        r = native.Run(native.load(), w.config)
        r.set_reference(w.reference)
        r.set_particles(w.particles)
    with torch.cuda.device(0):
        value = np.random.default_rng(5).standard_normal(r.get_field(0).shape)
        r.set_field(0, value)
        np.testing.assert_array_equal(r.get_field(0), value)
        np.testing.assert_array_equal(r.get_particles()["z"], w.particles["z"])
        assert not np.any(r.get_field(8))
