"""A breakdown at p'.Ap' = 0, in every solve kernel: the solution is that of the iterations before it.

A is a chain of blocks [[1, -1], [-1, 1]] and b = (1, 0, 1, 0, ...).  Every number of the first iteration is a small
whole one in any of the precisions: p = b, alpha = 1, x = b, r = (0, 1, ...), beta = 1, and then p = (1, 1, ...), which
A takes to zero.  So the solve ends in its second iteration with x = b and one iteration done."""
import numpy as np
import pytest

import project_xplus_b200 as xp
from project_xplus_b200.batch import BatchSolver

pytestmark = pytest.mark.gpu


def _chain(blocks):
    n = 2 * blocks
    rp = np.arange(0, 2 * n + 1, 2, dtype=np.int32)
    ci = np.repeat(np.arange(n, dtype=np.int32).reshape(-1, 2), 2, axis=0).reshape(-1)
    return rp, ci, np.tile([1.0, -1.0, -1.0, 1.0], blocks), np.tile([1.0, 0.0], blocks)


F64 = dict(values_dtype="f64", vector_dtype="f64")


@pytest.mark.parametrize("blocks,kw", [
    (1, dict()), (1, dict(chunk=1)), (1, dict(index16=False)), (1, dict(values_dtype="bf16")), (700, dict()),
    (50_000, dict()), (50_000, dict(chunk=2, values_dtype="f16")),                   # one barrier, SM-resident
    (1, dict(barriers_per_iter=2)), (50_000, dict(barriers_per_iter=2)),             # two barriers
    (1, dict(resident=False)), (50_000, dict(resident=False)),                       # global memory
    (800_000, dict()),                                                               # windowed
    (1, F64), (500, F64), (50_000, F64)], ids=str)
@pytest.mark.parametrize("tau_mode", [xp.XPLUS_TAU_ABS_RR, xp.XPLUS_TAU_REL_TRUE])
def test_jacobi(blocks, kw, tau_mode):
    rp, ci, v, b = _chain(blocks)
    s = xp.PcgSolver(rp, ci, v, **kw)
    r = s.solve(b, tau=1e-12, tau_mode=tau_mode)
    s.close()
    assert (r.status, r.iterations) == ("breakdown", 1)
    np.testing.assert_array_equal(r.solution, b)
    assert r.residual_rel == 1.0


@pytest.mark.parametrize("resident", [True, False])
@pytest.mark.parametrize("blocks", [1, 700, 50_000])
def test_gtg(blocks, resident):
    rp, ci, v, b = _chain(blocks)
    s = xp.PcgSolver(rp, ci, v, resident=resident)
    s.set_gtg(np.tile([1.0, 0.0, 1.0], blocks))  # G = I: rows {a_00} and {a_10, a_11} of the lower pattern
    r = s.solve(b, tau=1e-12)
    s.close()
    assert (r.status, r.iterations) == ("breakdown", 1)
    np.testing.assert_array_equal(r.solution, b)


@pytest.mark.parametrize("resident", [True, False])
def test_batch(resident):
    chains = [_chain(k) for k in (1, 40, 3000)]
    s = BatchSolver([c[:3] for c in chains])
    s.set_resident(resident)
    b = np.concatenate([c[3] for c in chains])
    r = s.solve(b, tau=1e-12)
    s.close()
    assert r["status_names"] == ["breakdown"] * 3 and r["iterations"].tolist() == [1] * 3
    np.testing.assert_array_equal(r["x"], b)
