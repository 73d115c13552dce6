"""w90g_profile_device times the kernels that a solve launches."""
import ctypes as C

import numpy as np
import pytest

from wannier90_gb300 import library as w90
from wannier90_gb300 import synth
from wannier90_gb300._native import lib

pytestmark = pytest.mark.gpu


# the search in the gradient's last CTA up to 512 of them (27 k, 648 k); one spread launch or two
@pytest.mark.parametrize("mp,W,tensor", [((3, 3, 3), 4, 0), ((3, 3, 3), 10, 1), ((9, 9, 8), 2, 0), ((4, 4, 4), 40, 1)])
def test_profile_launches_what_a_solve_does(mp, W, tensor):
    torch = pytest.importorskip("torch")
    iters = 3
    p = synth.make_problem(kind="sc", a=5.0, mp=mp, num_wann=W, rmax=1, eps=0.05 / np.sqrt(W), seed=1)
    m = torch.from_numpy(p.m.reshape(-1, order="F").view(np.float64).copy()).cuda()
    u = torch.from_numpy(p.a.reshape(-1, order="F").view(np.float64).copy()).cuda()
    h = w90.setup(kpoints=p.kpoints, unit_cell_cart=p.real_lattice, num_wann=W, num_iter=iters, iprint=0,
                  gpu_tensor=tensor, conv_window=-1)
    assert w90.w90_project_overlap_device(h, m.data_ptr(), u.data_ptr()) == 0, h.last_error()
    torch.cuda.synchronize()
    names = [lib().w90g_profile_kernel_name(i).decode() for i in range(9)]
    ms, cnt = (C.c_double * 9)(), (C.c_int * 9)()
    assert lib().w90g_profile_device(h._h, C.c_void_p(m.data_ptr()), C.c_void_p(u.data_ptr()), iters, ms, cnt) == 0
    count = dict(zip(names, cnt))
    assert lib().w90g_profile_kernel_name(9) == b""
    fused = len(p.kpoints) * ((W + 31) // 32) ** 2 <= 512
    assert count["k_ctrl_search"] == (0 if fused else iters), count
    assert count["k_ctrl_step"] == count["k_ctrl_end"] == count["k_precond"] == 0, count
    assert count["k_grad"] == iters and count["init"] == 1, count
    assert iters <= count["k_exp_u"] == count["k_m_update"] == count["k_omega"] <= 2 * iters, count
