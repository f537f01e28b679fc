"""Aggregation of graphs whose nodes are queued many times.

On random graphs a node is a neighbour of many rounder nodes and is listed by
each, so that the list of good seeds outgrows the number of nodes.  The setup
ran over the end of an array there, which ended the process; in one of its
own it now ends by itself.
"""
import os
import subprocess
import sys

import pytest

SCRIPT = """
import sys
import numpy as np
import doug_gb300 as D
n = int(sys.argv[1])
rng = np.random.default_rng(5)
i, j = rng.integers(0, n, (2, 2 * n))
i, j = i[i != j], j[i != j]
w = rng.uniform(0.5, 1.5, len(i))
r, c, v = np.concatenate([i, j]), np.concatenate([j, i]), -np.concatenate([w, w])
d = np.bincount(r, -v, minlength=n) + 0.05
k = np.arange(n)
s = D.DougSolver(dict(solver=2, method=1, fine_method=1, levels=1, smoothers=1, strong1="0.08", overlap=1, radius1=2,
                      maxasize1=100000, solve_tolerance="1.0e-8", solve_maxiters=3000))
s.set_matrix_coo(n, np.concatenate([r, k]) + 1, np.concatenate([c, k]) + 1, np.concatenate([v, d]))
s.set_partition((1 + k * 8 // n).astype(np.int32))
try:
    s.setup()
except D.DougError as e:
    assert e.status == D.DG_NO_DEVICE, e
"""


@pytest.mark.parametrize("n", [200, 1000, 6000])
def test_setup_of_a_random_graph(n):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    run = subprocess.run([sys.executable, "-c", SCRIPT, str(n)], cwd=root, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
