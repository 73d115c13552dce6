"""The FP64 projection (num_wann <= 8, and what the tensor-core polar factor leaves) against a polar
factor in extended precision, over the widths and condition numbers of its routes: few steps from A,
more of them, and past its first 32 steps; magnitudes that are scaled first; rank-deficient A."""
import numpy as np
import pytest

from tests.projection_helpers import mesh, overlaps, project, projections

pytestmark = pytest.mark.gpu


def _polar(A):
    """Newton-Schulz in the widest floats NumPy has (at least as wide as FP64's 53 bits)."""
    X = A.astype(np.clongdouble)
    X = X / np.sqrt((np.abs(X) ** 2).sum((1, 2)))[:, None, None]
    eye = np.eye(A.shape[1])
    for _ in range(120):
        G = np.conj(np.swapaxes(X, 1, 2)) @ X
        X = X @ (1.5 * eye - 0.5 * G)
        if np.abs(G - eye).max() < 1e-15:
            break
    return X


# the steps' roundings add up like W + 4 of them at the size of the result, times what A's own rounding
# is worth: (4 + 0.1 cond) (W + 4) 2^-53
@pytest.mark.parametrize("W", [1, 2, 3, 5, 6, 8])
@pytest.mark.parametrize("cond", [1.02, 3.0, 100.0, 5e3, 1e5])
def test_small_projection(W, cond):
    if W == 1 and cond > 2.0:
        pytest.skip("one singular value")
    lattice, kp, nnlist = mesh((3, 3, 2))
    K, B = nnlist.shape
    A, _ = projections(K, W, cond, seed=7 * W)
    ierr, err, got, _ = project(lattice, kp, overlaps(K, B, W, 1), A)
    assert ierr == 0, err
    assert np.abs(got - _polar(A)).max() <= (4 + 0.1 * cond) * (W + 4) * 2.0 ** -53


@pytest.mark.parametrize("W", [1, 4, 8])
@pytest.mark.parametrize("scale", [2.0 ** -500, 2.0 ** -120, 2.0 ** 120, 2.0 ** 500])
def test_magnitude_of_the_projections_does_not_matter(W, scale):
    lattice, kp, nnlist = mesh((3, 3, 2))
    K, B = nnlist.shape
    M = overlaps(K, B, W, 1)
    A, _ = projections(K, W, 3.0, seed=W)
    want = project(lattice, kp, M, A)
    got = project(lattice, kp, M, A * scale)
    assert want[0] == got[0] == 0, got[1]
    np.testing.assert_allclose(got[2], want[2], atol=5 * (W + 4) * 2.0 ** -53)


@pytest.mark.parametrize("W", [1, 2, 5, 8])
@pytest.mark.parametrize("kind", ["zero column", "equal columns", "zero"])
def test_small_rank_deficient_projection_is_refused(W, kind):
    if W == 1 and kind == "equal columns":
        pytest.skip("one column")
    lattice, kp, nnlist = mesh((2, 2, 2))
    K, B = nnlist.shape
    A, _ = projections(K, W, 2.0, seed=W)
    if kind == "zero column":
        A[4, :, 0] = 0.0
    elif kind == "zero":
        A[4] = 0.0
    else:
        # small integers: the Gram matrix is exact and so is its singularity
        A[4] = np.round(4 * A[4].real) + 1j * np.round(4 * A[4].imag)
        A[4, :, 1] = A[4, :, 0]
    ierr, err, _, _ = project(lattice, kp, overlaps(K, B, W, 1), A)
    if kind == "equal columns" and ierr == 0:
        pytest.skip("the computed eigenvalue of A^H A came out positive")
    assert ierr == 1 and "k-point 5" in err, err
