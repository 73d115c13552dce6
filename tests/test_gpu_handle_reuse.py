"""A handle whose options change between calls, at shapes that let its engine keep its arrays:
every result is that of a fresh handle."""
import numpy as np
import pytest

from tests.projection_helpers import mesh
from oracle import w90_oracle as O
from wannier90_gb300 import library as w90
from wannier90_gb300 import synth

pytestmark = pytest.mark.gpu


def _again(c, **options):
    """The options of another problem on a handle that has solved one."""
    for k, v in options.items():
        w90.w90_set_option(c, k, v)
    w90.check(c, w90.w90_input_setopt(c, "again"), "w90_input_setopt")


def _solve(c, m0, u0):
    m = np.array(m0, order="F", copy=True)
    u = np.array(u0, order="F", copy=True)
    K, W = u.shape[2], u.shape[0]
    w90.w90_set_m_local(c, m)
    w90.w90_set_u_matrix(c, u)
    w90.w90_set_u_opt(c, np.asfortranarray(np.broadcast_to(np.eye(W, dtype=np.complex128)[:, :, None], (W, W, K)).copy()))
    assert w90.w90_wannierise(c) == 0, c.last_error()
    return m, u, w90.w90_get_log(c, 6)[:, :8].copy()


def _problem(kp, lattice, W, seed):
    """Smooth overlaps over the k-points in the order given, from random orbitals."""
    rng = np.random.default_rng(seed)
    _, nnlist, _, bk = synth.kmesh_tables(lattice, kp)
    H = rng.standard_normal((W, W)) + 1j * rng.standard_normal((W, W))
    tau = rng.random((W, 3)) @ lattice
    gen = [0.1 / np.sqrt(W) * (X - np.conj(X.T)) for X in (H, 1j * H, H @ H / W)]
    U = []
    for k in kp:
        w, v = np.linalg.eigh(1j * sum(np.sin(2 * np.pi * k[i]) * gen[i] for i in range(3)))
        U.append((v * np.exp(-1j * w)) @ np.conj(v.T))
    U = np.array(U)
    ph = np.exp(-1j * np.einsum("kbi,ai->kba", bk, tau))
    M = np.conj(np.swapaxes(U, 1, 2))[:, None] @ (ph[..., None] * U[nnlist])
    return synth.from_math_m(M), synth.from_math_u(np.broadcast_to(np.eye(W), U.shape).astype(complex))


@pytest.mark.parametrize("W,tensor", [(8, 0), (8, 1), (20, 1), (40, 1), (70, 1)])
def test_other_k_order_on_the_same_handle(W, tensor):
    lattice, kp, _ = mesh((3, 3, 3))
    perm = np.random.default_rng(1).permutation(len(kp))
    o = dict(num_wann=W, num_iter=5, iprint=0, gpu_tensor=tensor, conv_window=-1)
    c = w90.setup(kpoints=kp, unit_cell_cart=lattice, **o)
    _solve(c, *_problem(kp, lattice, W, 3))
    _again(c, kpoints=kp[perm], unit_cell_cart=lattice, **o)
    args = _problem(kp[perm], lattice, W, 3)
    got = _solve(c, *args)
    want = _solve(w90.setup(kpoints=kp[perm], unit_cell_cart=lattice, **o), *args)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_other_kernel_options_on_the_same_handle():
    """gpu_mupdate_pipe and gpu_exp_smem choose among kernels of the same results."""
    lattice, kp, _ = mesh((3, 3, 3))
    W = 20
    args = _problem(kp, lattice, W, 4)
    o = dict(num_wann=W, num_iter=5, iprint=0, gpu_tensor=1, conv_window=-1)
    want = _solve(w90.setup(kpoints=kp, unit_cell_cart=lattice, **o), *args)
    c = w90.setup(kpoints=kp, unit_cell_cart=lattice, **o)
    for pipe, smem in ((1, 0), (0, 0), (0, 1), (1, 1), (1, 0)):
        _again(c, kpoints=kp, unit_cell_cart=lattice, gpu_mupdate_pipe=pipe, gpu_exp_smem=smem, **o)
        for a, b in zip(_solve(c, *args), want):
            assert np.array_equal(a, b), (pipe, smem)


def test_other_guiding_schedule_on_the_same_handle():
    p = synth.make_problem(kind="sc", a=4.0, mp=(3, 3, 3), num_wann=4, rmax=1, eps=0.3, seed=11)
    km = O.kmesh_get(p.real_lattice, p.kpoints, 36)
    U0, M0 = O.overlap_project(synth.to_math_m(p.m), synth.to_math_u(p.a), km["nnlist"])
    args = synth.from_math_m(M0), synth.from_math_u(U0)
    frac = np.random.default_rng(3).random((4, 3))
    o = dict(num_wann=4, num_iter=5, iprint=0, conv_window=-1, guiding_centres=1, guiding_centres_frac=frac)
    new = dict(num_no_guide_iter=2, num_guide_cycles=2)
    c = w90.setup(kpoints=p.kpoints, unit_cell_cart=p.real_lattice, num_no_guide_iter=0, num_guide_cycles=1, **o)
    first = _solve(c, *args)
    _again(c, kpoints=p.kpoints, unit_cell_cart=p.real_lattice, **new, **o)
    got = _solve(c, *args)
    want = _solve(w90.setup(kpoints=p.kpoints, unit_cell_cart=p.real_lattice, **new, **o), *args)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    assert not np.array_equal(first[2], want[2])
