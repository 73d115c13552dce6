"""Trial steps down to zero on the tensor path: the optimal step's exp may not lean on powers of a
trial matrix whose norm its FP32 estimate cannot see."""
import numpy as np
import pytest

from oracle import w90_oracle as O
from tests.engine_helpers import run_engine
from wannier90_gb300 import synth

pytestmark = pytest.mark.gpu


def _problem(W):
    p = synth.make_problem(kind="sc", a=5.0, mp=(3, 3, 3), num_wann=W, rmax=1, eps=0.3 / np.sqrt(W), seed=5)
    km = O.kmesh_get(p.real_lattice, p.kpoints, 36)
    U0, M0 = O.overlap_project(synth.to_math_m(p.m), synth.to_math_u(p.a), km["nnlist"])
    return p, km, M0, U0


# one width per tile width; the trial changes the spread by less than it is computed to, so the
# parabola's minimum is arbitrary, but the step to it is a rotation whatever its length
@pytest.mark.parametrize("W", [6, 13, 24, 40, 100])
@pytest.mark.parametrize("trial", [1e-5, 1e-7, 1e-9, 1e-11, 1e-14, 1e-100, 1e-170, -1e-10])
def test_the_step_after_a_tiny_trial_is_a_rotation(W, trial):
    p, km, M0, U0 = _problem(W)
    out = run_engine(p.real_lattice, p.kpoints, M0, U0, O.WannControl(num_iter=2, trial_step=trial), W, project=False,
                     extra={"gpu_tensor": 1})
    assert out["ierr"] == 0, out["err"]
    U = out["U"]
    assert np.isfinite(U).all()
    # a solve of two exps of degree 12 with up to some thirty squarings: 56-bit products, whose
    # rounding a squaring doubles at most
    np.testing.assert_allclose(np.conj(np.swapaxes(U, 1, 2)) @ U, np.broadcast_to(np.eye(W), U.shape), atol=1e-9)
    R = np.conj(np.swapaxes(U0, 1, 2)) @ U
    want = np.conj(np.swapaxes(R, 1, 2))[:, None] @ M0 @ R[km["nnlist"]]
    np.testing.assert_allclose(out["M"], want, atol=1e-9)


@pytest.mark.parametrize("W", [6, 13, 24, 40, 100])
def test_a_zero_trial_step_moves_nothing(W):
    p, _, M0, U0 = _problem(W)
    out = run_engine(p.real_lattice, p.kpoints, M0, U0, O.WannControl(num_iter=2, trial_step=0.0), W, project=False,
                     extra={"gpu_tensor": 1})
    assert out["ierr"] == 0, out["err"]
    np.testing.assert_allclose(out["U"], U0, atol=8 * W * 2.0 ** -53)
    np.testing.assert_allclose(out["M"], M0, atol=W * 2.0 ** -44)
