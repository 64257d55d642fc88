"""dposv above the order where the substitutions get a launch of their own."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FRESH = """
import numpy as np, chameleon_b200 as cb
n, nb, nrhs = %d, %d, %d
cb.init()
g = np.random.default_rng(n)
A0 = g.uniform(-0.5, 0.5, (n, n)); A0 = A0 + A0.T + n * np.eye(n)
B0 = g.uniform(-0.5, 0.5, (n, nrhs))
dA, dB = cb.Desc.create(n, n, nb), cb.Desc.create(n, nrhs, nb)
dA.from_numpy(A0); dB.from_numpy(B0)
assert cb.dposv_Tile(cb.ChamLower, dA, dB) == 0
X = dB.to_numpy()
r = np.linalg.norm(B0 - A0 @ X) / (np.linalg.norm(A0) * np.linalg.norm(X))
assert r <= 8 * n * np.finfo(float).eps, r
"""


@pytest.mark.parametrize("n,nb,nrhs", [(3144, 262, 64), (3200, 200, 900)])
def test_first_call_of_a_process(n, nb, nrhs):
    """The substitutions need more counters than the factorization, and no
    earlier call has grown the workspace."""
    subprocess.run([sys.executable, "-c", FRESH % (n, nb, nrhs)], cwd=ROOT, check=True, timeout=300)
