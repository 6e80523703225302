"""The network's kernels take eight lanes per row and sum gradients over blocks of nodes: rows around 8 and 32
pattern entries, and systems of fewer rows than a warp's four or a block's thirty-two."""
import numpy as np
import pytest

import project_xplus_b200 as xp
from project_xplus_b200 import learned as L

pytestmark = pytest.mark.gpu
SIZES = [(2, 1), (3, 1), (5, 4), (33, 7), (61, 8), (257, 31), (130, 33), (400, 70), (2500, 3)]


def _banded(n, half):
    """SPD band matrix: row i reaches i - half .. i + half."""
    rng = np.random.default_rng(n + half)
    i, j = np.nonzero(np.abs(np.subtract.outer(np.arange(n), np.arange(n))) <= half)
    a = np.zeros((n, n))
    a[i, j] = -rng.uniform(0.1, 1.0, len(i))
    a = (a + a.T) / 2
    np.fill_diagonal(a, 0.0)
    np.fill_diagonal(a, np.abs(a).sum(1) * rng.uniform(1.05, 1.5, n))
    rp = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))]).astype(np.int32)
    return rp, j.astype(np.int32), a[i, j], a


def _params():
    theta = L.init_params(3)
    return theta + np.random.default_rng(3).normal(0, 0.05, theta.size).astype(np.float32)


@pytest.mark.parametrize("n,half", SIZES)
def test_gradient_of_two_copies_is_that_of_one(n, half):
    """The losses are means over rows, so a block-diagonal pair of one system has its loss and its gradient; the two
    differ by the order of the FP32 sums only (the node values of the copies are the same bits)."""
    rp, ci, v, _ = _banded(n, half)
    pair = (np.concatenate([rp, rp[1:] + rp[-1]]), np.concatenate([ci, ci + n]), np.concatenate([v, v]))
    t = L.GnnTrainer([(rp, ci, v), pair], params=_params(), loss="kaporin")
    (l1, g1), (l2, g2) = t.loss_grad(0, 0), t.loss_grad(1, 0)
    t.close()
    assert abs(l1 - l2) <= 1e-6 * max(1.0, abs(l1))
    off = 0
    for name, shape in L.layout():
        m = int(np.prod(shape))
        a, b = g1[off:off + m].astype(np.float64), g2[off:off + m].astype(np.float64)
        assert np.abs(a - b).max() <= 2e-3 * max(np.abs(a).max(), 1e-12) + 1e-9, name
        off += m


@pytest.mark.parametrize("n,half", SIZES)
def test_normalized_rows(n, half):
    """set_gnn scales each row of G to (G A G^T)_ii = 1 (FP32 sums of at most 71 x 71 terms)."""
    rp, ci, v, dense = _banded(n, half)
    s = xp.PcgSolver(rp, ci, v)
    s.set_gnn(_params())
    low = s.get_gtg()
    s.close()
    g = np.zeros((n, n))
    rows = np.repeat(np.arange(n), np.diff(rp))
    keep = ci <= rows
    g[rows[keep], ci[keep]] = low
    np.testing.assert_allclose(np.einsum("ij,jk,ik->i", g, dense, g, optimize=True), 1.0, rtol=1e-4)
