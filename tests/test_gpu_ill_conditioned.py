"""The FP64 form of the projection's polar factor (num_wann <= 8, several problems in one engine, and
what the tensor-core iteration leaves) over its range of condition numbers.

Tolerances.  U is unitary to a Newton-Schulz step's own rounding, W + 2 terms of at most 2 per
element and their square: 16 W 2^-53.  A perturbation of eps |A| -- the input's own rounding here,
the products' W eps in the iteration -- moves the polar factor by its ratio to the two smallest
singular values: 8 W 2^-53 cond."""
import numpy as np
import pytest

from tests.projection_helpers import mesh, overlaps, project, projections

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [2, 5, 8, 9, 16, 17, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("cond", [1e2, 1e4, 3e4, 1e5, 1e6, 1e7])
def test_polar_factor_of_an_ill_conditioned_projection(W, cond):
    lattice, kp, nnlist = mesh((3, 3, 2))
    K, B = nnlist.shape
    A, U = projections(K, W, cond, seed=W)
    ierr, err, got, _ = project(lattice, kp, overlaps(K, B, W, 1), A)
    assert ierr == 0, err
    eye = np.broadcast_to(np.eye(W), U.shape)
    np.testing.assert_allclose(np.conj(np.swapaxes(got, 1, 2)) @ got, eye, atol=16 * W * 2.0 ** -53)
    np.testing.assert_allclose(got, U, atol=8 * W * 2.0 ** -53 * cond)
