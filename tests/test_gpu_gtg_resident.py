"""The SM-resident G^T G kernel against the global-memory one, whose arithmetic and sums it keeps in order: the same
bits, over sizes at the edges of its bands and windows, value types, layouts, replacement policies and the fallback."""
import numpy as np
import pytest

import project_xplus_b200 as xp
from project_xplus_b200 import generators as gen
from project_xplus_b200.learned import fsai_lower

pytestmark = pytest.mark.gpu


def _system(dim, side):
    if dim == 2:
        return gen.fem2d(side, sigma=1.5, seed=side, perm_seed=1, rcm=True)[0]
    return gen.fem3d(side, sigma=1.0, seed=side)[0]


def _solve(d, fallback=0, **kw):
    s = xp.PcgSolver.from_dataset(d, **kw)
    s.set_gtg(fsai_lower(d.row_ptr, d.col_idx, d.values), fallback)
    r = s.solve(d.b, np.linspace(-1, 1, d.n), tau=1e-8, tau_mode=xp.XPLUS_TAU_REL_TRUE, max_iters=900, trace=True)
    s.close()
    return r


@pytest.mark.parametrize("dim,side", [(2, 2), (2, 6), (2, 23), (2, 91), (2, 274), (2, 275), (2, 520), (3, 9), (3, 40)])
@pytest.mark.parametrize("kw", [dict(), dict(chunk=2), dict(values_dtype="bf16"), dict(values_dtype="f16", replace_every=7),
                                dict(fallback=5), dict(restart_on_replace=3, replace_drop=0.3)],
                         ids=lambda k: "-".join(f"{a}={b}" for a, b in k.items()) or "default")
def test_same_bits_as_the_global_memory_kernel(dim, side, kw):
    d = _system(dim, side)
    # resident=False keeps the global-memory form
    a, b = _solve(d, **kw), _solve(d, resident=False, **kw)
    assert (a.status, a.iterations, a.replacements) == (b.status, b.iterations, b.replacements)
    assert a.metrics["jacobi_fallback_at"] == b.metrics["jacobi_fallback_at"]
    np.testing.assert_array_equal(a.solution, b.solution)
    assert [(t.alpha, t.beta, t.rz, t.rr) for t in a.iteration_trace] == \
        [(t.alpha, t.beta, t.rz, t.rr) for t in b.iteration_trace]


def test_barrier_timeout_ends_the_solve():
    """A block that withholds its first arrival: every bounded wait expires and the status says so."""
    from project_xplus_b200._lib import check, lib
    d = _system(2, 91)
    s = xp.PcgSolver.from_dataset(d, barrier_timeout_s=0.05)
    s.set_gtg(fsai_lower(d.row_ptr, d.col_idx, d.values))
    check(lib.xplus_pcg_debug_skip_arrival(s.handle, 3))
    assert s.solve(d.b, tau=1e-8).status == "timeout"
    check(lib.xplus_pcg_debug_skip_arrival(s.handle, -1))
    assert s.solve(d.b, tau=1e-8, tau_mode=xp.XPLUS_TAU_REL_TRUE).status == "converged"
    s.close()
