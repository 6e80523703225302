"""The windowed kernel (systems beyond the SM-resident one) against the global-memory kernel, whose arithmetic and
sums it keeps in order: the same bits."""
import numpy as np
import pytest

import project_xplus_b200 as xp
from project_xplus_b200 import generators as gen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def systems():
    return {"3d": gen.fem3d(104, sigma=1.0, seed=5)[0],  # a band's window of 29,000 rows
            "2d": gen.fem2d(1251, sigma=1.0, seed=5, perm_seed=1, rcm=True)[0]}


@pytest.mark.parametrize("which,kw", [("3d", dict()), ("3d", dict(chunk=2)), ("3d", dict(values_dtype="bf16")),
                                      ("3d", dict(values_dtype="f16", replace_every=9)), ("2d", dict()),
                                      ("2d", dict(restart_on_replace=3, replace_drop=0.5))],
                         ids=lambda v: v if isinstance(v, str) else "-".join(f"{a}={b}" for a, b in v.items()) or "default")
def test_same_bits_as_the_global_memory_kernel(systems, which, kw):
    d = systems[which]
    out = []
    for resident in (True, False):  # without resident the global-memory kernel runs
        s = xp.PcgSolver.from_dataset(d, resident=resident, **kw)
        r = s.solve(d.b, np.linspace(-1, 1, d.n), tau=1e-9, tau_mode=xp.XPLUS_TAU_REL_TRUE, max_iters=150, trace=True)
        assert r.metrics["kernel"] == "pcg_persistent_kernel"
        out.append((r.status, r.iterations, r.replacements, [(t.alpha, t.beta, t.rz, t.rr) for t in r.iteration_trace],
                    r.solution))
        s.close()
    assert out[0][:4] == out[1][:4]
    np.testing.assert_array_equal(out[0][4], out[1][4])


def test_barrier_timeout_ends_the_solve(systems):
    from project_xplus_b200._lib import check, lib
    d = systems["3d"]
    s = xp.PcgSolver.from_dataset(d, barrier_timeout_s=0.05)
    check(lib.xplus_pcg_debug_skip_arrival(s.handle, 7))
    assert s.solve(d.b, tau=1e-8).status == "timeout"
    check(lib.xplus_pcg_debug_skip_arrival(s.handle, -1))
    assert s.solve(d.b, tau=1e-6, tau_mode=xp.XPLUS_TAU_REL_TRUE).status == "converged"
    s.close()
