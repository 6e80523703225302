"""The device's persisting-L2 limit over the life of a handle: set aside while a kernel that wants it can run, and handed
back when the handle returns to a kernel that does without."""
import ctypes as C
import gc

import numpy as np
import pytest

import project_xplus_b200 as xp

pytestmark = pytest.mark.gpu
CU_LIMIT_PERSISTING_L2_CACHE_SIZE = 6


def _limit():
    v = C.c_size_t()
    assert C.CDLL("libcuda.so.1").cuCtxGetLimit(C.byref(v), CU_LIMIT_PERSISTING_L2_CACHE_SIZE) == 0
    return v.value


def _chain(n):
    """Tridiagonal, too many rows for the SM-resident kernels."""
    rp = np.concatenate([[0], np.cumsum(np.concatenate([[2], np.full(n - 2, 3), [2]]))]).astype(np.int32)
    ci = (np.arange(n)[:, None] + [-1, 0, 1]).reshape(-1)[1:-1].astype(np.int32)
    return rp, ci, np.tile([-1.0, 2.1, -1.0], n)[1:-1]


def test_back_to_jacobi_hands_the_set_aside_back():
    m = _chain(1_600_000)
    g = np.tile([0.0, 1.0], len(m[0]) - 1)[1:]  # G = I
    s = xp.PcgSolver(*m)
    gc.collect()
    before = _limit()
    s.set_gtg(g)
    assert _limit() > before  # the global-memory G^T G kernel
    s.set_gtg(None)
    assert _limit() == before
    other = xp.PcgSolver(*m, resident=False)  # a handle that keeps its own
    held = _limit()
    assert held > before
    s.set_gtg(g)
    s.set_gtg(None)
    assert _limit() == held
    b = np.cos(np.arange(s.n))
    r = s.solve(b, tau=1e-8, tau_mode=xp.XPLUS_TAU_REL_TRUE)
    assert r.status == "converged"
    other.close()
    s.close()
    assert _limit() == before
