"""The opt-in trace (PB_GPU_TRACE=1): a line per factorisation and per CG launch on stderr, each with the
precision, the iteration limit and the grid of its launch."""
import os
import re
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
from plabundle_gb300 import synth
from plabundle_gb300.device import Gb300Context
from plabundle_gb300.problem import SolveOptions
for mixed in (True, False):
    o = SolveOptions()
    o.backend.enablePlaMatrixMixedPrecision = mixed
    ctx = Gb300Context(0)
    assert ctx.upload(synth.ring_problem(seed=2, n_cameras=8, n_points=200), o) == 0
    ctx.solve()
"""


def test_trace_lines_name_precision_limit_and_grid():
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, env=dict(os.environ, PB_GPU_TRACE="1"),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    cg = re.findall(r"^PB_GPU_CG precision=(\d) iterations=(\d+) relres=(\S+) converged=([01]) max_it=(\d+) grid=(\d+)$",
                    r.stderr, re.M)
    assert len(cg) == len(re.findall(r"^PB_GPU_CG ", r.stderr, re.M)) > 2
    assert {c[0] for c in cg} == {"0", "1"}
    for _, it, rel, _, most, grid in cg:
        assert int(it) <= int(most) and float(rel) >= 0 and int(grid) >= 1
    assert re.search(r"^PB_GPU_FACTOR precision=1 n=\d+ shift=\S+ status=0$", r.stderr, re.M)
