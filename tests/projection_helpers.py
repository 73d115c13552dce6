"""Random projection problems and the calls on them (math layout: M[k, b, m, n], A[k, m, n])."""
import numpy as np

from wannier90_gb300 import library as w90
from wannier90_gb300 import synth


def mesh(mp):
    lattice, kp = synth.lattice("sc", 5.0), synth.mp_kpoints(*mp)
    return lattice, kp, synth.kmesh_tables(lattice, kp)[1]


def overlaps(K, B, W, seed):
    rng = np.random.default_rng(seed)
    z = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    return z(K, B, W, W) / np.sqrt(2.0 * W)


def projections(K, W, cond, seed):
    """A = U S V with singular values from 3 / cond to 3, and the polar factor U V."""
    rng = np.random.default_rng(seed)
    u, _, v = np.linalg.svd(rng.standard_normal((K, W, W)) + 1j * rng.standard_normal((K, W, W)))
    s = np.exp(rng.uniform(-np.log(cond), 0.0, (K, W))) * 3.0
    if W > 1:
        s[:, 0], s[:, -1] = 3.0, 3.0 / cond
    return (u * s[:, None, :]) @ v, u @ v


def rotated(M, U, nnlist):
    return np.conj(np.swapaxes(U, 1, 2))[:, None] @ M @ U[nnlist]


def project(lattice, kpoints, M, A):
    """w90_project_overlap on host arrays: ierr, message, U, M."""
    c = w90.setup(kpoints=kpoints, unit_cell_cart=lattice, num_wann=A.shape[1], iprint=0)
    m = np.array(synth.from_math_m(M), order="F", copy=True)
    u = np.array(synth.from_math_u(A), order="F", copy=True)
    w90.w90_set_m_local(c, m)
    w90.w90_set_u_matrix(c, u)
    ierr = w90.w90_project_overlap(c)
    return ierr, c.last_error(), synth.to_math_u(u), synth.to_math_m(m)
