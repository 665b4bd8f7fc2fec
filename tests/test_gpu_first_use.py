"""Kernels are set up when a handle first uses their shape: every way in works as
the first one of a process (its shared-memory limits are set, its occupancy is
not taken before that) and gives what it gives later."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

WAYS = {
    "split": "one(precision='fp64', nx=64, ny=64)",
    "full": "one(precision='fp64', nx=300, ny=300)",
    "tuner": "one(precision='fp64', nx=64, ny=64, autotune=True)",
    "tuner_fp32": "one(precision='fp32', nx=200, ny=200, autotune=True)",
    "exact": "one(precision='mixed', nx=64, ny=64, exact=True, solver='hll')",
    "hancock": "one(precision='fp64', nx=64, ny=64, order='hancock')",
    "hancock_mixed": "one(precision='mixed', nx=64, ny=64, order='hancock', exact=True)",
    "ensemble": "many(precision='mixed')",
    "ensemble_tuner": "many(precision='fp64', autotune=True)",
}
CODE = """
import sys
sys.path.insert(0, %r)
import numpy as np
import pmhd

def one(steps=40, **kw):
    with pmhd.Solver(**kw) as s:
        s.init_problem(pmhd.PROBLEM_ORSZAG_TANG)
        st = s.advance(max_steps=steps)
        assert st.steps == steps and st.ctas >= 1
        return s.get_state()

def many(**kw):
    ms = [pmhd.member(n, n, pmhd.PROBLEM_ORSZAG_TANG, (1.0,), t_end=1e9) for n in (32, 100)]
    with pmhd.Ensemble(ms, **kw) as e:
        e.advance(max_steps=40)
        return e.get_state(1)

first, later = %s, %s
scale = np.abs(later).max(axis=(0, 1))
assert np.isfinite(first).all()
assert np.all(np.abs(first - later)[..., :8] <= 1e-4 * scale[:8])
print("FIRST_USE_OK")
"""


@pytest.mark.parametrize("way", sorted(WAYS))
def test_each_way_in_works_as_the_first_of_a_process(pmhd_lib, way):
    import os

    pkg = os.path.dirname(os.path.dirname(os.path.abspath(pmhd_lib.__file__)))
    r = subprocess.run([sys.executable, "-c", CODE % (pkg, WAYS[way], WAYS[way])], capture_output=True, text=True,
                       timeout=120)
    assert "FIRST_USE_OK" in r.stdout, r.stdout + r.stderr


TIMED = """
import sys
sys.path.insert(0, %r)
import pmhd
best = 1e9
for solver in %r:
    with pmhd.Solver(nx=1024, ny=512, precision=%r, order="hancock", solver=solver) as s:
        s.init_problem(pmhd.PROBLEM_ORSZAG_TANG)
        s.advance(max_steps=8)
        best = min(s.advance(max_steps=32).device_ms for _ in range(5))
print("MS", best)
"""


@pytest.mark.parametrize("precision", ["fp32", "mixed"])
def test_the_first_handle_does_not_set_the_next_ones_occupancy(pmhd_lib, precision):
    """An HLLD handle after an HLL one runs as many CTAs per SM as one that is the first
    of its process (half as many took 1.5 times as long)."""
    import os

    pkg = os.path.dirname(os.path.dirname(os.path.abspath(pmhd_lib.__file__)))
    ms = {}
    for solvers in (["hlld"], ["hll", "hlld"]):
        r = subprocess.run([sys.executable, "-c", TIMED % (pkg, solvers, precision)], capture_output=True, text=True,
                           timeout=120)
        assert "MS " in r.stdout, r.stdout + r.stderr
        ms[len(solvers)] = float(r.stdout.split("MS ")[1])
    assert ms[2] < 1.2 * ms[1], ms
