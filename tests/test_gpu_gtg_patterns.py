"""G^T G where the patterns of A, G and G^T differ: entries that A stores on one side of the diagonal only, and a G whose
pattern is not A's.  Every form of the kernel takes them, with the same bits."""
import numpy as np
import pytest

import project_xplus_b200 as xp
from project_xplus_b200 import generators as gen
from project_xplus_b200._lib import check, lib, ptr
from project_xplus_b200.learned import fsai_lower

pytestmark = pytest.mark.gpu


def _with_zeros(d, rows, cols):
    """d's matrix with explicit zeros at (rows, cols)."""
    i = np.concatenate([np.repeat(np.arange(d.n), np.diff(d.row_ptr)), rows])
    j = np.concatenate([d.col_idx, cols])
    v = np.concatenate([d.values, np.zeros(len(rows))])
    o = np.lexsort((j, i))
    rp = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=d.n))]).astype(np.int32)
    return rp, j[o].astype(np.int32), v[o]


def _g(rp, ci, seed=0):
    """Lower-triangular G of any pattern: a diagonal near 1, small entries elsewhere."""
    i = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    low = ci <= i
    g = np.random.default_rng(seed).uniform(-0.05, 0.05, low.sum())
    return np.where(ci[low] == i[low], 1.0 + g, g)


def _same(matrix, b, pattern, g, tau=1e-8, tau_mode=xp.XPLUS_TAU_REL_TRUE, max_iters=400, **kw):
    """Both forms of the kernel solve alike."""
    out = []
    for resident in (True, False):
        s = xp.PcgSolver(*matrix, resident=resident, **kw)
        check(lib.xplus_pcg_set_gtg(s.handle, ptr(pattern[0]), ptr(pattern[1]), ptr(g), 0))
        out.append(s.solve(b, np.linspace(-1, 1, len(b)), tau=tau, tau_mode=tau_mode, max_iters=max_iters, trace=True))
        s.close()
    a, c = out
    assert c.metrics["kernel_form"] == "pcg_gtg_kernel"
    assert (a.status, a.iterations, a.replacements) == (c.status, c.iterations, c.replacements)
    np.testing.assert_array_equal(a.solution, c.solution)
    np.testing.assert_array_equal([t.rr for t in a.iteration_trace], [t.rr for t in c.iteration_trace])
    return a


@pytest.mark.parametrize("side,reach", [(23, 100), (91, 300), (91, 3000), (274, 9000), (274, 30000)])
@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("kw", [dict(), dict(chunk=2, sigma=1), dict(values_dtype="bf16", build_on_gpu=False)], ids=str)
def test_one_sided_zeros(side, reach, lower, kw):
    d = gen.fem2d(side, sigma=1.5, seed=side)[0]
    far = np.arange(reach, d.n, max(1, (d.n - reach) // 9))
    m = _with_zeros(d, *((far, far - reach) if lower else (far - reach, far)))
    exact = fsai_lower(*m)
    r = _same(m, d.b, m, exact, max_iters=2000, **kw)
    assert r.status == "converged" or kw.get("values_dtype") == "bf16"
    # 12 bytes of shared memory per row of a window: all 91^2 rows fit, 30000 do not
    if side < 274 or reach == 30000:
        assert r.metrics["kernel_form"] == ("pcg_gtg_res_kernel" if side < 274 else "pcg_gtg_kernel")
    # and with values at the one-sided entries too
    _same(m, d.b, m, np.where(exact == 0.0, 0.01, exact), **kw)


def test_an_offset_that_fits_int16_on_one_side_only():
    d = gen.fem2d(190, sigma=1.0, seed=2)[0]
    m = _with_zeros(d, np.array([32768, 33000]), np.array([0, 232]))  # -32768 in G, +32768 in G^T
    r = _same(m, d.b, m, np.where(fsai_lower(*m) == 0.0, 0.01, fsai_lower(*m)), sigma=1)
    assert r.metrics["kernel_form"] == "pcg_gtg_kernel"


@pytest.mark.parametrize("side", [23, 91, 274])
def test_a_pattern_that_is_not_the_matrix_s(side):
    d = gen.fem2d(side, sigma=1.0, seed=side)[0]
    rng = np.random.default_rng(side)
    rows = np.repeat(np.arange(d.n), np.diff(d.row_ptr))
    ci = np.where(d.col_idx == rows, rows, np.minimum((rng.random(d.nnz) * rows).astype(np.int32), rows)).astype(np.int32)
    _same((d.row_ptr, d.col_idx, d.values), d.b, (d.row_ptr, ci), _g(d.row_ptr, ci), tau=1e-20,
          tau_mode=xp.XPLUS_TAU_ABS_RR, max_iters=40)


@pytest.mark.parametrize("first", [0, 64, 8192])
def test_a_slice_of_g_without_entries(first):
    """Rows first .. first + 31 have entries right of the diagonal only."""
    d = gen.fem2d(91, sigma=1.0, seed=1)[0]
    rows = np.repeat(np.arange(d.n), np.diff(d.row_ptr))
    k = np.arange(d.nnz) - d.row_ptr[rows]
    above = (rows >= first) & (rows < first + 32) & (rows < d.n - 10)
    ci = np.where(above, rows + 1 + k, d.col_idx).astype(np.int32)
    r = _same((d.row_ptr, d.col_idx, d.values), d.b, (d.row_ptr, ci), _g(d.row_ptr, ci), tau=1e-20,
              tau_mode=xp.XPLUS_TAU_ABS_RR, max_iters=30, sigma=1)
    assert r.metrics["kernel_form"] == "pcg_gtg_kernel"
