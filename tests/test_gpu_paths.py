"""The tensor-core steps around the iteration and the wide M update against plain 64-bit NumPy,
at the sizes where a tile, a column chunk, a K-step or a dispatch rule ends.

Tolerances.  A product with 7-bit digits leaves out the digit pairs of the diagonals above the
seventh: at most 6 * 2W * 2^12 * 2^-7 units of 2^-56 (row scale x column scale), i.e. W 2^-47.4 times
scales of at most 4 for entries up to 1; two products per block, hence W 2^-44 on M.  56-bit products
and FP64 sums stay below 4 W 2^-53 per element; a polar factor's error carries its condition number."""
import numpy as np
import pytest

from oracle import w90_oracle as O
from tests.engine_helpers import run_engine
from wannier90_gb300 import library as w90
from wannier90_gb300 import synth

pytestmark = pytest.mark.gpu


def _projected(kind, mp, W, seed, eps=0.05):
    p = synth.make_problem(kind=kind, a=5.0, mp=mp, num_wann=W, rmax=1, eps=eps / np.sqrt(W), seed=seed)
    km = O.kmesh_get(p.real_lattice, p.kpoints, 36)
    U0, M0 = O.overlap_project(synth.to_math_m(p.m), synth.to_math_u(p.a), km["nnlist"])
    return p, km, M0, U0


def _rotated(M0, U, nnlist):
    return np.conj(np.swapaxes(U, 1, 2))[:, None] @ M0 @ U[nnlist]


# tile rows B W (not) a multiple of 128, chunk widths 24 and 32, 2 to 4 chunks, ragged K-steps
@pytest.mark.parametrize("kind,W,mp", [("sc", 33, (3, 3, 3)), ("fcc", 40, (2, 2, 2)), ("sc", 48, (3, 3, 3)),
                                       ("fcc", 64, (2, 2, 2)), ("sc", 65, (3, 3, 3)), ("fcc", 96, (2, 2, 2)),
                                       ("sc", 100, (3, 3, 3)), ("sc", 128, (3, 3, 3))])
def test_wide_update_is_the_rotation_of_the_entry_overlaps(kind, W, mp):
    p, km, M0, U0 = _projected(kind, mp, W, seed=5)
    ctl = O.WannControl(num_iter=3, lfixstep=True, fixed_step=0.5)
    out = run_engine(p.real_lattice, p.kpoints, M0, U0, ctl, W, project=False, extra={"gpu_tensor": 1})
    assert out["ierr"] == 0, out["err"]
    R = np.conj(np.swapaxes(U0, 1, 2)) @ out["U"]           # the accumulated rotation
    np.testing.assert_allclose(np.conj(np.swapaxes(R, 1, 2)) @ R, np.broadcast_to(np.eye(W), R.shape), atol=1e-13)
    np.testing.assert_allclose(out["M"], _rotated(M0, R, km["nnlist"]), atol=W * 2.0 ** -44)
    # the spread record (diagonal statistics and the direct off-diagonal sum) from that M
    ref = O.wann_main(M0, U0, km, ctl)
    for row, it in zip(out["log"][1:], ref.iters):
        assert abs(row[3] - it.spread.om_tot) <= 1e-9 * abs(it.spread.om_tot) + 2e-10


def _project(A, M, nnlist, kpoints, lattice):
    """w90_project_overlap on host arrays (math layout)."""
    K, W = A.shape[:2]
    c = w90.setup(kpoints=kpoints, unit_cell_cart=lattice, num_wann=W, iprint=0)
    m = np.array(synth.from_math_m(M), order="F", copy=True)
    u = np.array(synth.from_math_u(A), order="F", copy=True)
    w90.w90_set_m_local(c, m)
    w90.w90_set_u_matrix(c, u)
    ierr = w90.w90_project_overlap(c)
    return ierr, c.last_error(), synth.to_math_u(u), synth.to_math_m(m)


def _random_problem(W, cond, seed):
    lattice, kp = synth.lattice("sc", 5.0), synth.mp_kpoints(3, 3, 2)
    _, nnlist, _, _ = synth.kmesh_tables(lattice, kp)
    rng = np.random.default_rng(seed)
    K, B = nnlist.shape
    z = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    u, _, v = np.linalg.svd(z(K, W, W))
    s = np.exp(rng.uniform(-np.log(cond), 0.0, (K, W))) * 3.0
    s[:, 0], s[:, -1] = 3.0, 3.0 / cond
    M = z(K, B, W, W) / np.sqrt(2.0 * W)
    return lattice, kp, nnlist, (u * s[:, None, :]) @ v, u @ v, M


# below and above the width from which the projection runs on the tensor cores (9), its tile
# widths, and the condition numbers it leaves to the FP64 kernel (1e7)
@pytest.mark.parametrize("W", [1, 5, 8, 9, 16, 17, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("cond", [1.2, 30.0, 1e7])
def test_projection_against_the_svd(W, cond):
    if W == 1 and cond > 1.2:
        pytest.skip("one singular value")
    lattice, kp, nnlist, A, U, M = _random_problem(W, cond, seed=W)
    ierr, err, got, m = _project(A, M, nnlist, kp, lattice)
    assert ierr == 0, err
    # the FP64 form behind the iteration starts from A^H A: its eigenvalues carry cond^2, which the
    # correction takes back to first order
    tol = 8 * W * 2.0 ** -53 * cond if cond < 1e5 else 1e-3
    np.testing.assert_allclose(got, U, atol=tol)
    np.testing.assert_allclose(m, _rotated(M, got, nnlist), atol=8 * W * 2.0 ** -53 * 4)


@pytest.mark.parametrize("W", [4, 12, 40])
def test_rank_deficient_projection_is_refused(W):
    lattice, kp, nnlist, A, _, M = _random_problem(W, 2.0, seed=W)
    A[3, :, W // 2] = 0.0
    ierr, err, _, _ = _project(A, M, nnlist, kp, lattice)
    assert ierr == 1
    assert "rank deficient at k-point 4" in err, err


# an FP32 maximum up to 5e-6 passes on its own; above it FP64 decides at 1e-5
@pytest.mark.parametrize("W", [5, 40])
@pytest.mark.parametrize("scale,ok", [(1.0, True), (1.0 + 3.0e-6, True), (1.0 + 4.9e-6, True), (1.0 + 5.1e-6, False)])
def test_unitarity_verdict_near_the_bound(W, scale, ok):
    p, _, M0, U0 = _projected("sc", (2, 2, 2), W, seed=9)
    out = run_engine(p.real_lattice, p.kpoints, M0, U0 * scale, O.WannControl(num_iter=1), W, project=False)
    assert (out["ierr"] == 0) == ok, out["err"]


# spread chunks of 16 blocks from 512 blocks (k,b) on, one-CTA spreads up to 3072 statistics
@pytest.mark.parametrize("W,mp", [(3, (4, 4, 4)), (8, (4, 4, 4)), (9, (4, 4, 4)), (7, (5, 5, 5)), (6, (5, 5, 4))])
@pytest.mark.parametrize("tensor", [0, 1])
def test_spread_passes_over_their_chunk_rules(W, mp, tensor):
    p, km, M0, U0 = _projected("sc", mp, W, seed=2)
    ctl = O.WannControl(num_iter=3)
    out = run_engine(p.real_lattice, p.kpoints, M0, U0, ctl, W, project=False, extra={"gpu_tensor": tensor})
    assert out["ierr"] == 0, out["err"]
    ref = O.wann_main(M0, U0, km, ctl)
    for row, it in zip(out["log"], [ref.initial] + ref.iters):
        assert abs(row[3] - it.spread.om_tot) <= 1e-9 * abs(it.spread.om_tot) + 2e-10
        assert int(row[6]) == int(it.lquad)
    np.testing.assert_allclose(out["centres"].T, ref.centres.T, atol=1e-7)


# slabs of several groups and of one, a last slab that is shorter; both digit forms
@pytest.mark.parametrize("kind,W,mp", [("sc", 33, (3, 3, 3)), ("fcc", 48, (2, 2, 2)), ("sc", 64, (1, 1, 3)),
                                       ("sc", 40, (1, 1, 2)), ("sc", 100, (2, 2, 2)), ("sc", 128, (2, 2, 2))])
def test_wide_update_in_slabs_equals_the_whole(kind, W, mp):
    """A served job that fits its budget only with the image of Z in slabs gives the same bits."""
    torch = pytest.importorskip("torch")
    p, km, M0, U0 = _projected(kind, mp, W, seed=9)
    res = []
    budget = 1e12
    for _ in range(2):
        h = w90.setup(kpoints=p.kpoints, unit_cell_cart=p.real_lattice, num_wann=W, num_iter=4, iprint=0, gpu_tensor=1,
                      conv_window=-1)
        m = torch.from_numpy(synth.from_math_m(M0).reshape(-1, order="F").view(np.float64).copy()).cuda()
        u = torch.from_numpy(synth.from_math_u(U0).reshape(-1, order="F").view(np.float64).copy()).cuda()
        torch.cuda.synchronize()
        srv = w90.Server(budget, max_active=1, chunk_iters=2)
        assert srv.submit(h, m.data_ptr(), u.data_ptr(), 0) == 0, h.last_error()
        srv.drain()
        done = srv.poll()
        peak = srv.stats()["peak_bytes"]
        srv.close()
        assert len(done) == 1 and done[0][1] == 0, h.last_error()
        assert peak <= budget
        res.append((m.cpu().numpy(), u.cpu().numpy(), w90.w90_get_log(h, 5).copy()))
        budget = peak - 1
    (m1, u1, l1), (m2, u2, l2) = res
    assert np.array_equal(m1, m2) and np.array_equal(u1, u2)
    assert np.array_equal(l1[:, :8], l2[:, :8])
