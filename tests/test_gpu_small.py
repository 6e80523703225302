"""The one-CTA FP64 kernel at the edges of what it takes: fewer rows than a warp, one to four slices per warp, slices
without off-diagonal slots, every value type and chunk, against a direct solve and the golden's residual history."""
import numpy as np
import pytest

import project_xplus_b200 as xp
from oracle import oracle as O
from project_xplus_b200 import generators as gen

pytestmark = pytest.mark.gpu


def _dense(d):
    a = np.zeros((d.n, d.n))
    np.add.at(a, (np.repeat(np.arange(d.n), np.diff(d.row_ptr)), d.col_idx), d.values)
    return a


@pytest.mark.parametrize("side", [1, 2, 5, 6, 22, 23, 32, 33, 45])
@pytest.mark.parametrize("kw", [dict(values_dtype="f64"), dict(values_dtype="f64", chunk=1, index16=False),
                                dict(values_dtype="f32"), dict(values_dtype="f32", row_sum_form=False, chunk=2),
                                dict(values_dtype="bf16"), dict(values_dtype="f64", block_threads=512, sigma=1)],
                         ids=lambda k: "-".join(f"{a}={b}" for a, b in k.items()))
def test_matches_a_direct_solve(side, kw):
    d, _ = gen.fem2d(side, sigma=1.0, seed=side, x_seed=side)
    s = xp.PcgSolver.from_dataset(d, vector_dtype="f64", **kw)
    r = s.solve(d.b, np.linspace(-1, 1, d.n), tau=1e-12, tau_mode=xp.XPLUS_TAU_REL_TRUE)
    s.close()
    a = _dense(d)
    assert r.status == "converged"
    # ||A dx|| <= 1e-12 ||b|| and ||dx|| <= ||A^-1|| ||A dx||, plus the direct solve's own rounding
    bound = (1e-12 + 1e-14 * np.linalg.cond(a)) * np.linalg.norm(d.b) * np.linalg.norm(np.linalg.inv(a), 2)
    assert np.linalg.norm(r.solution - np.linalg.solve(a, d.b)) <= bound


@pytest.mark.parametrize("side", [6, 22, 32, 45])
def test_residual_history_starts_as_the_golden(side):
    d, _ = gen.fem2d(side, sigma=0.5, seed=side, x_seed=side)
    s = xp.PcgSolver.from_dataset(d, values_dtype="f64", vector_dtype="f64")
    r = s.solve(d.b, d.x0, tau=1e-10, trace=True)
    s.close()
    ref = O.golden(d, 1e-10)
    assert abs(r.iterations - ref["iterations"]) <= 1
    k = min(15, r.iterations)  # within the horizon where two FP64 runs stay together
    np.testing.assert_allclose([t.residual for t in r.iteration_trace[:k]], ref["trace"][:k, 4], rtol=1e-9)


def test_slices_without_slots():
    n = 300  # a diagonal matrix but for a chain among its last rows
    rows = [[(i, 1.0 + 0.01 * i)] for i in range(n)]
    for i in range(250, n - 1):
        rows[i].append((i + 1, -0.2))
        rows[i + 1].insert(0, (i, -0.2))
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    ci = np.array([c for r in rows for c, _ in r], np.int32)
    v = np.array([a for r in rows for _, a in r])
    b = np.cos(np.arange(n))
    a = np.zeros((n, n))
    a[np.repeat(np.arange(n), np.diff(rp)), ci] = v
    for kw in (dict(values_dtype="f32", sigma=1), dict(values_dtype="f64", sigma=1)):
        s = xp.PcgSolver(rp, ci, v, vector_dtype="f64", **kw)
        r = s.solve(b, tau=1e-12, tau_mode=xp.XPLUS_TAU_REL_TRUE)
        s.close()
        np.testing.assert_allclose(r.solution, np.linalg.solve(a, b), atol=1e-10)
