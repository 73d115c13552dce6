"""The FP64 form of the projection's polar factor (num_wann <= 8, several problems in one engine, and
what the tensor-core iteration leaves) over its range of condition numbers.

Tolerances.  U is unitary to a Newton-Schulz step's own rounding, W + 2 terms of at most 2 per
element and their square: 16 W 2^-53.  A perturbation of eps |A| -- the input's own rounding here,
the products' W eps in the iteration -- moves the polar factor by its ratio to the two smallest
singular values: 8 W 2^-53 cond."""
import numpy as np
import pytest

from oracle import w90_oracle as O
from tests.engine_dis import run_dis
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


@pytest.mark.parametrize("nb,W", [(3, 2), (7, 4), (12, 8), (18, 12), (40, 24), (64, 40)])
@pytest.mark.parametrize("cond", [1e2, 1e3, 1e5, 1e7])
def test_polar_factors_of_an_ill_conditioned_disentanglement(nb, W, cond):
    """U_opt^H A carries the projections' condition number into U."""
    lattice, kp, nnlist = mesh((2, 2, 2))
    K, B = nnlist.shape
    A = projections(K, nb, cond, seed=nb)[0][:, :, nb - W:]
    s = np.linalg.svd(A, compute_uv=False)
    assert s[:, 0].max() < 3.1 and s[:, -1].min() > 2.9 / cond
    eig = np.sort(np.random.default_rng(1).random((K, nb)), axis=1)
    out = run_dis(lattice, kp, overlaps(K, B, nb, 1), A, eig, W, O.DisControl(num_iter=1))
    assert out["ierr"] == 0, out["err"]
    U, V = out["U0"], out["Uopt"]
    eye = np.broadcast_to(np.eye(W), U.shape)
    np.testing.assert_allclose(np.conj(np.swapaxes(V, 1, 2)) @ V, eye, atol=16 * nb * 2.0 ** -53)
    np.testing.assert_allclose(np.conj(np.swapaxes(U, 1, 2)) @ U, eye, atol=16 * W * 2.0 ** -53)
    X = np.conj(np.swapaxes(V, 1, 2)) @ A
    u, t, v = np.linalg.svd(X)
    ok = t[:, -1] > 1e-7 * t[:, 0]
    got, want = U[ok], (u @ v)[ok]
    tol = (8 * nb * 2.0 ** -53 * t[:, 0] / t[:, -1])[ok]
    assert (np.abs(got - want).max((1, 2)) <= tol).all(), (np.abs(got - want).max((1, 2)), tol)
