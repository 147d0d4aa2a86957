"""Device memory of a run: what its steps need is reserved with its particles,
so that no step depends on the memory free when it comes, and the scan server's
estimate covers what the run holds.  Measured in a fresh
process, as the growth of the device's memory in use (the runs' pool keeps
what it was given, so the growth is its high-water mark)."""
import subprocess
import sys

import pytest

import checkers

pytestmark = pytest.mark.gpu

PROLOGUE = """
import sys
sys.path.insert(0, {repo!r})
import torch
from aprl_b200 import native, workloads
torch.zeros(1, device="cuda")
def used():
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free
def case(nx, ny, nz, particles, precision, shape):
    cfg = workloads.with_precision(workloads.make_config(
        nx, ny, nz, 5e-6, 5e-6, 2e-6, 8, 10.0, shape, 8), precision)
    bunch = workloads.gaussian_bunch(cfg, particles, 20e-12, 1e9, 50e-6, 20e-6, 1e-6, 1e-4, seed=1)
    return cfg, bunch
def loaded(cfg, bunch):
    r = native.Run(native.load(), cfg)
    r.allocate_reference()
    r.set_particles(bunch)
    return r
# Every kernel of the step loaded, on a grid too small to matter.
def warm(precision, shape):
    for particles in (400, 40000):
        cfg, bunch = case(40, 40, 40, particles, precision, shape)
        r = loaded(cfg, bunch)
        r.step(2)
        r.close()
"""


def child(body):
    code = PROLOGUE.format(repo=checkers.REPO) + body
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    return [int(v) for v in out.stdout.split()]


@pytest.mark.parametrize("precision", ["fp64", "fp32-mixed"])
def test_a_dense_runs_first_step_allocates_no_grid_array(precision):
    loaded, stepped = child(f"""
warm({precision!r}, "linear-binomial3")
cfg, bunch = case(128, 128, 256, 600000, {precision!r}, "linear-binomial3")
r = loaded(cfg, bunch)
a = used()
r.step(2)
print(a, used())
""")
    component = 129 * 128 * 257 * (8 if precision == "fp64" else 4)
    assert stepped - loaded < component, (stepped - loaded) / component


@pytest.mark.parametrize("precision", ["fp64", "fp32-mixed"])
@pytest.mark.parametrize("shape,particles", [("linear-binomial3", 60000),
                                             ("linear-binomial3", 600000),
                                             ("quintic-compensated", 600000)])
def test_the_scan_estimate_covers_a_run(precision, shape, particles):
    estimate, held = child(f"""
warm({precision!r}, {shape!r})
cfg, bunch = case(128, 128, 256, {particles}, {precision!r}, {shape!r})
a = used()
r = loaded(cfg, bunch)
r.step(2)
b = used()
scan = native.Scan(native.load(), slots=1)
print(scan.footprint(cfg, {particles}), b - a)
""")
    # Neither short nor, beyond the margins for carriers and pool rounding, wasteful.
    assert held <= estimate <= 1.25 * held, (estimate / 2**20, held / 2**20)


def test_reading_one_component_of_j_allocates_one_array():
    before, after = child("""
warm("fp64", "linear-binomial3")
cfg, bunch = case(128, 128, 256, 60000, "fp64", "linear-binomial3")
r = loaded(cfg, bunch)
r.step(1)
a = used()
r.get_field(6)
print(a, used())
""")
    assert after - before <= 2 * 128 * 129 * 257 * 8
