"""The remaining tensor-core routes with their bounded waits driven to run out (W90G_SPIN_LIMIT=0, see
test_gpu_bounded_wait.py): the one-CTA-per-group M update, the wide M update behind an FP64 exp, U = U0 R
after no iteration, the disentanglement's rotation -- an error each -- and the polar factors, which the
FP64 kernel then forms.  The normal build does the same calls afterwards."""
import json
import os
import subprocess
import sys

import pytest

from wannier90_gb300 import build as B

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import json, sys
import numpy as np
sys.path.insert(0, %(root)r)
from oracle import w90_oracle as O
from tests.engine_dis import run_dis
from tests.projection_helpers import mesh, overlaps, project, projections
from wannier90_gb300 import library as w90, synth
out = {}
def solve(W, num_iter, **extra):
    p = synth.make_problem(kind="sc", a=4.0, mp=(2, 2, 2), num_wann=W, rmax=1, eps=0.3, seed=2)
    h = w90.setup(kpoints=p.kpoints, unit_cell_cart=p.real_lattice, num_wann=W, num_iter=num_iter, iprint=0,
                  gpu_tensor=1, **extra)
    m, u = np.array(p.m, order="F", copy=True), np.array(p.a, order="F", copy=True)
    w90.w90_set_m_local(h, m)
    w90.w90_set_u_matrix(h, u)
    w90.w90_set_u_opt(h, np.asfortranarray(np.broadcast_to(np.eye(W, dtype=np.complex128)[:, :, None],
                                                           (W, W, len(p.kpoints))).copy()))
    assert w90.w90_project_overlap(h) == 0, h.last_error()
    return [w90.w90_wannierise(h), h.last_error()]
for W in (6, 13, 24):
    out["one CTA per group, %%d" %% W] = solve(W, 3, gpu_tensor_exp=0, gpu_mupdate_pipe=0)
for W in (40, 100):
    out["wide, %%d" %% W] = solve(W, 3, gpu_tensor_exp=0)
for W in (6, 13, 24, 40, 100):
    out["U0 R, %%d" %% W] = solve(W, 0)
lattice, kp, nnlist = mesh((2, 2, 2))
K, nB = nnlist.shape
for nb, W in ((14, 9), (24, 16), (48, 32)):
    A, _ = projections(K, nb, 2.0, 1)
    r = run_dis(lattice, kp, overlaps(K, nB, nb, 1), A[:, :, :W], np.sort(np.random.default_rng(1).random((K, nb)), axis=1),
                W, O.DisControl(num_iter=1))
    out["disentanglement, %%d" %% W] = [r["ierr"], r["err"]]
polar = []
for W in (9, 24, 40, 100):
    A, U = projections(K, W, 2.0, 1)
    ierr, err, got, _ = project(lattice, kp, overlaps(K, nB, W, 1), A)
    polar.append([ierr, float(np.abs(got - U).max()), 8 * W * 2.0 ** -53 * 2.0])
print(json.dumps([out, polar]))
"""


def _run(env):
    r = subprocess.run([sys.executable, "-c", CHILD % dict(root=ROOT)], capture_output=True, text=True, env=env,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_every_route_reports_and_the_gpu_stays_usable(tmp_path):
    lib = B.build(extra_nvcc=["-DW90G_SPIN_LIMIT=0"], libdir=str(tmp_path / "spin0"))
    res, polar = _run(dict(os.environ, W90G_LIBRARY=lib))
    for name, (ierr, msg) in res.items():
        assert ierr == 1 and "bounded wait" in msg, (name, ierr, msg)
    for ierr, err, tol in polar:
        assert ierr == 0 and err <= tol
    res, polar = _run(dict(os.environ))
    for name, (ierr, msg) in res.items():
        assert ierr == 0, (name, ierr, msg)
    for ierr, err, tol in polar:
        assert ierr == 0 and err <= tol
