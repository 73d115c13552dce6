"""The tensor-core rotation of the projection at its own sizes: 1296 blocks (more than its 304 CTAs
take at once), widths around its tile widths, against NumPy.  A copy of the library whose bounded
waits run out at once shows that this call takes that route."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from tests.projection_helpers import mesh, overlaps, project, projections, rotated
from wannier90_gb300 import build as B_

pytestmark = pytest.mark.gpu

MP = (6, 6, 6)
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


# two products of W terms, entries of M up to 4: 2 x 2 W 2^-53 x 4, twice that for the tails
@pytest.mark.parametrize("W", [9, 16, 17, 32, 33, 64, 65, 100])
@pytest.mark.parametrize("cond", [1.2, 30.0])
def test_rotation_of_many_blocks(W, cond):
    lattice, kp, nnlist = mesh(MP)
    K, B = nnlist.shape
    M = overlaps(K, B, W, 1)
    A, U = projections(K, W, cond, 2)
    ierr, err, got, m = project(lattice, kp, M, A)
    assert ierr == 0, err
    np.testing.assert_allclose(got, U, atol=8 * W * 2.0 ** -53 * cond)
    np.testing.assert_allclose(m, rotated(M, got, nnlist), atol=8 * W * 2.0 ** -53 * 4)


CHILD = r"""
import json, sys
sys.path.insert(0, %(root)r)
from tests.projection_helpers import mesh, overlaps, project, projections
lattice, kp, nnlist = mesh(%(mp)r)
K, B = nnlist.shape
out = []
for W in (9, 17, 33, 65):
    ierr, err, _, _ = project(lattice, kp, overlaps(K, B, W, 1), projections(K, W, 2.0, 2)[0])
    out.append((W, ierr, err))
print(json.dumps(out))
"""


def test_that_route_is_taken_and_reports_a_timed_out_wait(tmp_path):
    lib = B_.build(extra_nvcc=["-DW90G_SPIN_LIMIT=0"], libdir=str(tmp_path / "spin0"))
    r = subprocess.run([sys.executable, "-c", CHILD % dict(root=ROOT, mp=MP)], capture_output=True, text=True,
                       env=dict(os.environ, W90G_LIBRARY=lib), timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    for W, ierr, err in json.loads(r.stdout.strip().splitlines()[-1]):
        assert ierr == 1 and "bounded wait of the tensor-core rotation ran out" in err, (W, ierr, err)
