"""The tiled many-column sweeps, asked for when the solver is made and no longer
when its matrix changes."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import os, sys
import numpy as np
sys.path[:0] = sys.argv[1:]
from blood_network_b200 import amg
from test_gpu_solve_paths import _random_spd, _vascular
n, ia, ja, val = _vascular(3_000, False)
other = _random_spd(n, 6, 5)[1:]
B = np.random.default_rng(1).standard_normal((n, 5))
s = amg.AMGSolver(n, ia, ja, val, min_size=200, stop=amg.STOP_RELRES)
X, its, rel, rc = s.solve_block(B, tol=1e-9)
assert rc == 0
del os.environ["BN_BLOCK_IC_TILES"]
s.set_matrix(*other)
got = s.solve_block(B, tol=1e-9, maxiter=20)
s.close()
s = amg.AMGSolver(n, ia, ja, val, min_size=200, stop=amg.STOP_RELRES)  # never had tiles
s.set_matrix(*other)
want = s.solve_block(B, tol=1e-9, maxiter=20)
s.close()
assert got[3] == want[3] and (got[1] == want[1]).all()
assert got[0].tobytes() == want[0].tobytes() and np.isfinite(got[0]).all()
"""


def test_another_matrix_without_the_tiles():
    here = os.path.dirname(os.path.abspath(__file__))
    # a process of its own: the block solve reads the switch once
    r = subprocess.run([sys.executable, "-c", CODE, here, os.path.dirname(here)],
                       env=dict(os.environ, BN_BLOCK_IC_TILES="1"), capture_output=True, text=True,
                       timeout=200)
    assert r.returncode == 0, r.stderr[-2000:]
