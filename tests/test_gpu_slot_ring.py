"""The slot ring of the one-barrier SM-resident kernel against the two-barrier kernel, which reads its slots
group by group: sizes at the edges of its units (one slice, an odd number of slices per warp, bands without a slice,
rows wider than a unit, slices without slots) and the layouts that go through it or past it."""
import numpy as np
import pytest

import project_xplus_b200 as xp
from project_xplus_b200 import generators as gen

pytestmark = pytest.mark.gpu


def _solve(d, **kw):
    s = xp.PcgSolver.from_dataset(d, **kw)
    r = s.solve(d.b, tau=1e-9, tau_mode=xp.XPLUS_TAU_REL_TRUE)
    s.close()
    return r


@pytest.mark.parametrize("dim,side", [(2, 3), (2, 6), (2, 69), (2, 97), (2, 151), (2, 390), (3, 5), (3, 31), (3, 45)])
@pytest.mark.parametrize("kw", [dict(chunk=4), dict(chunk=2), dict(chunk=1), dict(index16=False),
                                dict(values_dtype="bf16"), dict(values_dtype="f16", chunk=2), dict(sigma=1)],
                         ids=lambda k: "-".join(f"{a}={b}" for a, b in k.items()))
def test_ring_matches_the_two_barrier_kernel(dim, side, kw):
    d, x = (gen.fem2d(side, sigma=1.0, seed=side, perm_seed=1, rcm=True) if dim == 2 else gen.fem3d(side, sigma=1.0, seed=side))
    one, two = _solve(d, **kw), _solve(d, barriers_per_iter=2, **kw)
    assert one.status == two.status == "converged"
    # both end with ||b - A x|| <= 1e-9 ||b|| in FP64: within twice that of each other in the residual
    a = np.repeat(np.arange(d.n), np.diff(d.row_ptr))
    dx = one.solution - two.solution
    gap = np.bincount(a, weights=d.values * dx[d.col_idx], minlength=d.n)
    assert np.linalg.norm(gap) <= 2e-9 * np.linalg.norm(d.b)


def test_rows_without_off_diagonals():
    n = 700
    rp, ci, v = np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), np.linspace(1.0, 5.0, n)
    # the last rows form a chain, so that slices without slots come before slices with some
    rows = [[(i, v[i])] for i in range(n)]
    for i in range(600, n - 1):
        rows[i].append((i + 1, -0.25))
        rows[i + 1].insert(0, (i, -0.25))
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    ci = np.array([c for r in rows for c, _ in r], np.int32)
    vals = np.array([a for r in rows for _, a in r])
    b = np.cos(np.arange(n))
    s = xp.PcgSolver(rp, ci, vals, sigma=1)
    r = s.solve(b, tau=1e-10, tau_mode=xp.XPLUS_TAU_REL_TRUE)
    assert r.metrics["kernel"] == "pcg_resident1_kernel" and r.status == "converged"
    dense = np.zeros((n, n))
    dense[np.repeat(np.arange(n), np.diff(rp)), ci] = vals
    np.testing.assert_allclose(r.solution, np.linalg.solve(dense, b), atol=1e-9)


def test_handles_of_different_size_live_together():
    solvers = [(d, xp.PcgSolver.from_dataset(d)) for d in (gen.fem2d(g, sigma=1.0, seed=g)[0] for g in (300, 60))]
    for d, s in solvers:  # the first handle needs more shared memory than the one made after it
        assert s.solve(d.b, tau=1e-8, tau_mode=xp.XPLUS_TAU_REL_TRUE).status == "converged"
