"""Which kernel a solve launches (metrics["kernel_form"]), on both sides of every line between them, and the bits of the
forms that share one arithmetic, each arm shown to be the kernel it is meant to be."""
import numpy as np
import pytest

import project_xplus_b200 as xp
from project_xplus_b200 import generators as gen
from project_xplus_b200._lib import check, lib
from project_xplus_b200.learned import fsai_lower

pytestmark = pytest.mark.gpu
F64 = dict(values_dtype="f64", vector_dtype="f64")
GENERAL, SMALL, WINDOW = "pcg_persistent_kernel", "pcg_small_kernel", "pcg_window_kernel"
RESIDENT, RESIDENT1, GTG, GTG_RES = "pcg_resident_kernel", "pcg_resident1_kernel", "pcg_gtg_kernel", "pcg_gtg_res_kernel"


def _chain(n):
    """Tridiagonal."""
    rp = np.concatenate([[0], np.cumsum(np.concatenate([[2], np.full(n - 2, 3), [2]]))]).astype(np.int32)
    ci = (np.arange(n)[:, None] + [-1, 0, 1]).reshape(-1)[1:-1].astype(np.int32)
    return rp, ci, np.tile([-1.0, 2.1, -1.0], n)[1:-1]


def _form(s, name, scheme):
    r = s.solve(np.cos(np.arange(s.n)), tau=1e-8, max_iters=3)
    assert (r.metrics["kernel_form"], r.metrics["kernel"]) == (name, scheme)


@pytest.mark.parametrize("n,kw,form,scheme", [
    # four slices of 32 rows per warp, 16 warps; four warps
    (2048, F64, SMALL, GENERAL), (2049, F64, GENERAL, GENERAL),
    (512, dict(F64, block_threads=128), SMALL, GENERAL), (513, dict(F64, block_threads=128), GENERAL, GENERAL),
    (2048, dict(values_dtype="bf16", vector_dtype="f64"), SMALL, GENERAL), (40, dict(resident=False), GENERAL, GENERAL),
    # 24 bytes of shared memory per row of a band of a chain; 4
    (1_200_000, dict(), RESIDENT1, RESIDENT1), (1_200_000, dict(barriers_per_iter=2), RESIDENT, RESIDENT),
    (1_600_000, dict(), WINDOW, GENERAL), (1_600_000, dict(values_dtype="bf16", chunk=2), WINDOW, GENERAL),
    (1_600_000, dict(chunk=1), GENERAL, GENERAL), (1_600_000, dict(index16=False), GENERAL, GENERAL),
    (1_600_000, dict(resident=False), GENERAL, GENERAL), (1_600_000, dict(row_sum_form=False), GENERAL, GENERAL),
    (1_600_000, dict(vector_dtype="f64"), GENERAL, GENERAL)], ids=str)
def test_jacobi(n, kw, form, scheme):
    s = xp.PcgSolver(*_chain(n), **kw)
    _form(s, form, scheme)
    s.close()


@pytest.mark.parametrize("n,kw,form", [
    (40, dict(), GTG_RES), (400_000, dict(), GTG_RES), (400_000, dict(chunk=2, values_dtype="f16"), GTG_RES),
    (1_600_000, dict(), GTG), (400_000, dict(chunk=1), GTG), (400_000, dict(index16=False), GTG),
    (400_000, dict(resident=False), GTG)], ids=str)
def test_gtg_and_back(n, kw, form):
    s = xp.PcgSolver(*_chain(n), **kw)
    assert s.last_metrics()["kernel_form"] == "none"
    s.set_gtg(np.tile([0.0, 0.7], n)[1:])
    _form(s, form, GTG)
    s.set_gtg(None)
    r = s.solve(np.cos(np.arange(n)), tau=1e-8, max_iters=3)
    assert "gtg" not in r.metrics["kernel_form"] and r.metrics["jacobi_fallback_at"] == -1
    s.close()


def _outcome(s, d, tau=1e-9, max_iters=150):
    r = s.solve(d.b, np.linspace(-1, 1, d.n), tau=tau, tau_mode=xp.XPLUS_TAU_REL_TRUE, max_iters=max_iters, trace=True)
    return r, (r.status, r.iterations, r.replacements, r.residual_rel,
               [(t.alpha, t.beta, t.rz, t.rr) for t in r.iteration_trace])


def _same(a, b):
    assert a[1] == b[1]
    np.testing.assert_array_equal(a[0].solution, b[0].solution)


@pytest.mark.parametrize("dim,side", [(2, 3), (2, 6), (2, 69), (2, 97), (2, 151), (2, 390), (3, 5), (3, 31), (3, 45)])
@pytest.mark.parametrize("kw", [dict(), dict(chunk=2), dict(values_dtype="bf16"), dict(values_dtype="f16", chunk=2),
                                dict(sigma=1, replace_every=7)], ids=str)
def test_the_slot_ring_has_the_bits_of_the_plain_loop(dim, side, kw):
    """int32 columns in the same layout go through the loop that loads a group of slices and then gathers."""
    d = (gen.fem2d(side, sigma=1.0, seed=side, perm_seed=1, rcm=True) if dim == 2 else gen.fem3d(side, sigma=1.0, seed=side))[0]
    out = []
    for index16 in (True, False):
        s = xp.PcgSolver.from_dataset(d, index16=index16, **kw)
        out.append(_outcome(s, d))
        assert out[-1][0].metrics["kernel_form"] == RESIDENT1
        s.close()
    _same(*out)


@pytest.mark.parametrize("side", [1, 5, 6, 22, 32, 45])
@pytest.mark.parametrize("kw", [dict(values_dtype="f64"), dict(values_dtype="f64", chunk=1, index16=False),
                                dict(values_dtype="f32"), dict(values_dtype="f32", row_sum_form=False, chunk=2),
                                dict(values_dtype="bf16", replace_every=5)], ids=str)
def test_the_one_cta_kernel_has_the_bits_of_the_global_memory_kernel(side, kw):
    d, _ = gen.fem2d(side, sigma=1.0, seed=side, x_seed=side)
    s = xp.PcgSolver.from_dataset(d, vector_dtype="f64", **kw)
    a = _outcome(s, d)
    check(lib.xplus_pcg_debug_skip_arrival(s.handle, 1))  # there is no block 1: nothing is withheld
    b = _outcome(s, d)
    s.close()
    assert (a[0].metrics["kernel_form"], b[0].metrics["kernel_form"]) == (SMALL, GENERAL)
    _same(a, b)


@pytest.mark.parametrize("which,kw", [("3d", dict()), ("3d", dict(values_dtype="bf16")), ("2d", dict(chunk=2))], ids=str)
def test_the_windowed_kernel_has_the_bits_of_the_global_memory_kernel(which, kw):
    d = gen.fem3d(104, sigma=1.0, seed=5)[0] if which == "3d" else gen.fem2d(1251, sigma=1.0, seed=5, perm_seed=1, rcm=True)[0]
    out = []
    for resident, form in ((True, WINDOW), (False, GENERAL)):
        s = xp.PcgSolver.from_dataset(d, resident=resident, **kw)
        out.append(_outcome(s, d, max_iters=60))
        assert out[-1][0].metrics["kernel_form"] == form
        s.close()
    _same(*out)


@pytest.mark.parametrize("dim,side", [(2, 23), (2, 275), (2, 520), (3, 40)])
def test_the_resident_gtg_kernel_has_the_bits_of_the_global_memory_one(dim, side):
    d = (gen.fem2d(side, sigma=1.5, seed=side, perm_seed=1, rcm=True) if dim == 2 else gen.fem3d(side, sigma=1.0, seed=side))[0]
    out = []
    for resident, form in ((True, GTG_RES), (False, GTG)):
        s = xp.PcgSolver.from_dataset(d, resident=resident)
        s.set_gtg(fsai_lower(d.row_ptr, d.col_idx, d.values))
        out.append(_outcome(s, d))
        assert out[-1][0].metrics["kernel_form"] == form
        s.close()
    _same(*out)
