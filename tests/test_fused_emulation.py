"""The fused hand-overs of the iteration -- the search in the gradient's last CTA, the control steps
in the spread passes' last CTAs, one spread launch or two -- on the CPU emulation of k_fp64.cu
(tests/emu/emu_fused.cpp): several problems in one launch, each with its own form, against the
same iteration one kernel at a time, and against the oracle."""
import ctypes as C
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

from oracle import w90_oracle as O
from wannier90_gb300 import synth

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "wannier90_gb300", "csrc")


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    tmp = tmp_path_factory.mktemp("emu_fused")
    src = open(os.path.join(CSRC, "k_fp64.cu")).read()
    src = re.sub(r"extern __shared__ double2 smem\[\];", "double2* smem = emu_dyn_smem<double2>();", src)
    src = re.sub(r'asm volatile\("mov\.u64 %0, %%globaltimer;" : "=l"\((\w+)\)\);', r"\1 = 0;", src)
    (tmp / "k_fp64_emu.cu").write_text(src)
    out = str(tmp / "emu_fused.so")
    subprocess.run([gxx, "-std=c++20", "-O1", "-shared", "-fPIC", "-D__CUDACC__", "-DEMU_FIBERS", "-I" + str(tmp),
                    "-I" + os.path.join(HERE, "emu"), "-I" + CSRC, os.path.join(HERE, "emu", "emu_fused.cpp"), "-o", out],
                   check=True)
    return C.CDLL(out)


def _problem(W, mp, seed):
    p = synth.make_problem(kind="sc", a=5.0, mp=mp, num_wann=W, rmax=1, eps=0.05 / np.sqrt(W), seed=seed)
    km = O.kmesh_get(p.real_lattice, p.kpoints, 36)
    U0, M0 = O.overlap_project(synth.to_math_m(p.m), synth.to_math_u(p.a), km["nnlist"])
    return km, M0, U0


def _solve(lib, problems, num_iter, window, tol, per, fused):
    n = len(problems)
    col = lambda X: np.ascontiguousarray(np.swapaxes(X, -1, -2)).view(np.float64)
    keep = [(np.ascontiguousarray(km["nnlist"], dtype=np.int32), np.ascontiguousarray(km["bk"], dtype=np.float64),
             np.ascontiguousarray(km["wb"], dtype=np.float64), col(M0), col(U0)) for km, M0, U0 in problems]
    logs = [np.zeros((num_iter + 1, 10)) for _ in problems]
    Us = [np.zeros_like(k[4]) for k in keep]
    rows = np.zeros(n, dtype=np.int32)
    ints = lambda v: np.array(v, dtype=np.int32)
    W, K, B = (ints([U0.shape[1] for _, _, U0 in problems]), ints([len(U0) for _, _, U0 in problems]),
               ints([M0.shape[1] for _, M0, _ in problems]))
    wbtot = np.array([km["wbtot"] for km, _, _ in problems])
    ptr = lambda arrays: (C.c_void_p * n)(*[a.ctypes.data for a in arrays])
    vp = lambda a: C.c_void_p(a.ctypes.data)
    lib.emu_solve.argtypes = ([C.c_int] + [C.c_void_p] * 9 + [C.c_int, C.c_int, C.c_double, C.c_int, C.c_int] +
                              [C.c_void_p] * 3)
    rc = lib.emu_solve(n, vp(W), vp(K), vp(B), ptr([k[0] for k in keep]), ptr([k[1] for k in keep]),
                       ptr([k[2] for k in keep]), vp(wbtot), ptr([k[3] for k in keep]), ptr([k[4] for k in keep]),
                       num_iter, window, tol, per, fused, ptr(logs), ptr(Us), vp(rows))
    assert rc == 0, rc
    return [log[:r] for log, r in zip(logs, rows)], Us


# 648 statistics in a chunk of 64 blocks or several; 3072 and 3456 around the one-launch rule; a
# convergence window that ends one problem before the other
@pytest.mark.parametrize("shapes,num_iter,window,tol,per", [
    ([(4, (3, 3, 3)), (9, (4, 4, 4))], 2, -1, 0.0, 64),
    ([(8, (4, 4, 4))], 1, -1, 0.0, 64),
    ([(3, (2, 2, 2)), (5, (3, 3, 3)), (2, (2, 2, 2))], 6, 2, 1e-2, 16),
])
def test_fused_iteration_equals_the_kernels_one_by_one(emu, shapes, num_iter, window, tol, per):
    problems = [_problem(W, mp, seed=3 + i) for i, (W, mp) in enumerate(shapes)]
    logs, Us = _solve(emu, problems, num_iter, window, tol, per, 1)
    plain, Up = _solve(emu, problems, num_iter, window, tol, per, 0)
    for (km, M0, U0), a, b, ua, ub in zip(problems, logs, plain, Us, Up):
        assert len(a) == len(b)
        assert np.array_equal(a[:, 6], b[:, 6])
        # one CTA sums Omega_D over all blocks at once, two passes by chunk: rounding
        np.testing.assert_allclose(a[:, 1:6], b[:, 1:6], rtol=0, atol=1e-12 * np.abs(b[:, 3]).max())
        np.testing.assert_allclose(ua, ub, rtol=0, atol=1e-11)
        r = O.wann_main(M0, U0, km, O.WannControl(num_iter=num_iter, conv_window=window, conv_tol=tol))
        assert len(a) == 1 + len(r.iters)
        for row, it in zip(a, [r.initial] + r.iters):
            assert abs(row[3] - it.spread.om_tot) <= 1e-10 * abs(it.spread.om_tot) + 1e-11


@pytest.fixture(scope="module")
def emu_dis(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    tmp = tmp_path_factory.mktemp("emu_dis_split")
    src = open(os.path.join(CSRC, "dis.cu")).read()
    src = src[:src.index("int dis_run(")] + "}  // namespace w90g\n"
    src = re.sub(r"extern __shared__ double2 (\w+)\[\];", r"double2* \1 = emu_dyn_smem<double2>();", src)
    (tmp / "dis_emu.cu").write_text(src)
    out = str(tmp / "emu_dis_split.so")
    subprocess.run([gxx, "-std=c++20", "-O1", "-shared", "-fPIC", "-D__CUDACC__", "-DEMU_FIBERS", "-I" + str(tmp),
                    "-I" + os.path.join(HERE, "emu"), "-I" + CSRC, os.path.join(HERE, "emu", "emu_dis_split.cpp"),
                    os.path.join(CSRC, "sym_tables.cpp"), "-o", out], check=True)
    return C.CDLL(out)


# frozen windows of several states per k, of none, and the silicon case's; 16, 64 and 32 threads a step
@pytest.mark.parametrize("name,step_threads", [("silicon_dis", 64), ("copper_dis", 16), ("basic2_dis", 32)])
def test_split_disentanglement_against_the_oracle(emu_dis, name, step_threads):
    """The engine's forms of the disentanglement kernels -- frozen states split off Z, one rotation by
    U_opt U0 -- on the reference's cases: Omega_I lines 1e-10, U_opt U and M0 1e-9."""
    from tests import golden_cases as G
    d = G.load(name)
    kn = d["knobs"]
    km = O.kmesh_get(d["real_lattice"], d["kpt_latt"], int(kn["search_shells"]))
    M = G.assemble_m(d, km["nnlist"], km["nncell"])
    nb, W, K, B = int(d["num_bands"]), int(kn["num_wann"]), len(d["kpt_latt"]), km["nntot"]
    dc = G.dis_control(d)
    dc.num_iter, dc.conv_tol = 4, 0.0
    f = lambda X: np.ascontiguousarray(np.swapaxes(X, -1, -2)).astype(np.complex128)
    Mf, Af, eig = f(M), f(d["amn"]), np.ascontiguousarray(d["eig"])
    nn, wb = np.ascontiguousarray(km["nnlist"], dtype=np.int32), np.ascontiguousarray(km["wb"])
    log, status = np.zeros((dc.num_iter, 3)), np.zeros(1, dtype=np.int32)
    U0, M0, Uo = (np.zeros(s, dtype=np.complex128) for s in ((K, W, W), (K, B, W, W), (K, W, nb)))
    vp = lambda a: C.c_void_p(a.ctypes.data)
    lib = emu_dis
    lib.emu_dis_engine.argtypes = ([C.c_int] * 4 + [C.c_void_p, C.c_void_p, C.c_double] + [C.c_void_p] * 3 +
                                   [C.c_int] + [C.c_double] * 3 + [C.c_int] + [C.c_double] * 2 + [C.c_int] * 2 +
                                   [C.c_void_p] * 5)
    rc = lib.emu_dis_engine(nb, W, K, B, vp(nn), vp(wb), km["wbtot"], vp(eig), vp(Mf), vp(Af), dc.num_iter,
                            dc.mix_ratio, dc.win_min, dc.win_max, int(dc.frozen_states), dc.froz_min, dc.froz_max, 32,
                            step_threads, vp(log), vp(U0), vp(M0), vp(Uo), vp(status))
    assert rc == 0 and status[0] == 0
    U0o, M0o, Uoo, _, recs = O.dis_main(M, d["amn"], d["eig"], km, W, dc)
    assert len(recs) == dc.num_iter
    for row, r in zip(log, recs):
        assert abs(row[1] - r.omega_i_prev) < 1e-10 and abs(row[2] - r.omega_i) < 1e-10
    g = lambda X: np.swapaxes(X, -1, -2)
    np.testing.assert_allclose(g(Uo) @ g(U0), Uoo @ U0o, atol=1e-9)
    np.testing.assert_allclose(g(M0), M0o, atol=1e-9)
