"""Device memory of a disentanglement: the arrays of the problem and nothing beside them."""
import ctypes as C

import numpy as np
import pytest

from oracle import w90_oracle as O
from tests.engine_dis import run_dis
from tests.projection_helpers import mesh, overlaps, projections

pytestmark = pytest.mark.gpu

USED_MEM_HIGH = 8   # CU_MEMPOOL_ATTR_USED_MEM_HIGH


def _pool():
    torch = pytest.importorskip("torch")
    torch.zeros(1, device="cuda")
    cu = C.CDLL("libcuda.so.1")
    pool = C.c_void_p()
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), torch.cuda.current_device()) == 0
    return cu, pool


# num_wann below and above the width of the tensor-core steps; fewer and more blocks than its CTAs
@pytest.mark.parametrize("nb,W,mp", [(12, 8, (4, 4, 4)), (16, 10, (4, 4, 4)), (24, 16, (3, 3, 3)), (48, 32, (3, 3, 4)),
                                     (20, 12, (6, 6, 6)), (64, 40, (2, 2, 2))])
@pytest.mark.parametrize("frozen", [False, True])
def test_peak_device_memory(nb, W, mp, frozen):
    cu, pool = _pool()
    lattice, kp, nnlist = mesh(mp)
    K, B = nnlist.shape
    A = projections(K, nb, 2.0, seed=1)[0][:, :, :W]
    eig = np.sort(np.random.default_rng(1).random((K, nb)), axis=1)
    dc = O.DisControl(num_iter=3, conv_tol=0.0, frozen_states=frozen, froz_max=0.2)
    zero = C.c_uint64(0)
    assert cu.cuMemPoolSetAttribute(pool, USED_MEM_HIGH, C.byref(zero)) == 0
    out = run_dis(lattice, kp, overlaps(K, B, nb, 1), A, eig, W, dc)
    assert out["ierr"] == 0, out["err"]
    high = C.c_uint64(0)
    assert cu.cuMemPoolGetAttribute(pool, USED_MEM_HIGH, C.byref(high)) == 0
    # M as given, windowed and rotated; A and U_opt twice; Z twice and its eigenvectors; U; 8 work matrices
    entries = K * (B * (2 * nb * nb + W * W) + 3 * nb * W + 3 * nb * nb + W * W + 8 * nb * nb)
    small = K * (12 * nb + 4 * B + 64) + 32 * 1024
    assert high.value <= 16 * entries + small, (high.value, 16 * entries)
