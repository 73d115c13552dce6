"""The products outside the iteration on values that digits cannot carry: NaN, infinities and
magnitudes near the ends of FP64.  Everything else in the call keeps its results."""
import numpy as np
import pytest

from tests.engine_helpers import run_engine
from tests.projection_helpers import mesh, overlaps, project, projections, rotated
from oracle import w90_oracle as O
from wannier90_gb300 import synth

pytestmark = pytest.mark.gpu

# 216 k-points, 1296 blocks: the tensor-core rotation; one width per tile width
WIDTHS = [12, 20, 40, 100]
MP = (6, 6, 6)


@pytest.mark.parametrize("W", WIDTHS)
def test_non_finite_overlaps_stay_non_finite(W):
    lattice, kp, nnlist = mesh(MP)
    K, B = nnlist.shape
    M = overlaps(K, B, W, 1)
    A, U = projections(K, W, 2.0, 2)
    bad = {(0, 0): np.nan, (5, 1): np.inf, (7, 2): -np.inf, (K - 1, B - 1): complex(0.0, np.nan)}
    for (k, b), v in bad.items():
        M[k, b, W // 3, W - 1] = v
    ierr, err, got, m = project(lattice, kp, M, A)
    assert ierr == 0, err
    # an element of M reaches every element of its block
    for k, b in bad:
        assert not np.isfinite(m[k, b]).any(), (k, b, np.nanmax(np.abs(m[k, b])))
    clean = np.ones((K, B), dtype=bool)
    for k, b in bad:
        clean[k, b] = False
        M[k, b] = 0.0
    np.testing.assert_allclose(m[clean], rotated(M, got, nnlist)[clean], atol=8 * W * 2.0 ** -53 * 4)


@pytest.mark.parametrize("W", WIDTHS)
@pytest.mark.parametrize("scale", [2.0 ** -1000, 2.0 ** -300, 2.0 ** 300, 2.0 ** 1000])
def test_overlaps_of_extreme_magnitude(W, scale):
    lattice, kp, nnlist = mesh(MP)
    K, B = nnlist.shape
    M = overlaps(K, B, W, 3)
    A, _ = projections(K, W, 2.0, 4)
    ierr, err, got, m = project(lattice, kp, M * scale, A)
    assert ierr == 0, err
    np.testing.assert_allclose(m / scale, rotated(M, got, nnlist), atol=8 * W * 2.0 ** -53 * 4)


# a lone entry in its row and column meets no finite partner in A^H A
@pytest.mark.parametrize("W", [5, 12, 20, 40])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("diagonal", [True, False])
def test_non_finite_projections_do_not_come_out_finite(W, value, diagonal):
    lattice, kp, nnlist = mesh((2, 2, 2))
    K, B = nnlist.shape
    M = overlaps(K, B, W, 5)
    A, _ = projections(K, W, 2.0, 6)
    if diagonal:
        A[3] = np.eye(W)
    A[3, W - 1, W - 1] = value
    ierr, err, got, _ = project(lattice, kp, M, A)
    if ierr == 0:
        assert not np.isfinite(got[3]).all()
    else:
        assert ierr == 1 and "k-point 4" in err, err


@pytest.mark.parametrize("W", [8, 20, 40, 100])
def test_a_nan_in_the_entry_u_stays_in_its_rows(W):
    """U = U0 R at the end of a tensor-path solve: the iteration does not read U0."""
    p = synth.make_problem(kind="sc", a=5.0, mp=(2, 2, 2), num_wann=W, rmax=1, eps=0.05 / np.sqrt(W), seed=5)
    km = O.kmesh_get(p.real_lattice, p.kpoints, 36)
    U0, M0 = O.overlap_project(synth.to_math_m(p.m), synth.to_math_u(p.a), km["nnlist"])
    ctl = O.WannControl(num_iter=2)
    want = run_engine(p.real_lattice, p.kpoints, M0, U0, ctl, W, project=False, extra={"gpu_tensor": 1})
    assert want["ierr"] == 0, want["err"]
    U1 = U0.copy()
    U1[2, W // 2, 1] = np.nan
    out = run_engine(p.real_lattice, p.kpoints, M0, U1, ctl, W, project=False, extra={"gpu_tensor": 1})
    hit = np.zeros(U0.shape[:2], dtype=bool)
    hit[2, W // 2] = True
    assert not np.isfinite(out["U"][hit]).any()
    np.testing.assert_allclose(out["U"][~hit], want["U"][~hit], atol=8 * W * 2.0 ** -53)
    assert np.array_equal(out["M"], want["M"])
