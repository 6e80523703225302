"""The GPU ordering where its BFS kernels change their way: as many children of a node as they keep and one more, rows
of one and of several steps of eight lanes, levels of one node per group of lanes and of many, against the host's."""
import numpy as np
import pytest

from project_xplus_b200 import generators as g

pytestmark = pytest.mark.gpu


def _csr(n, edges, seed=None):
    """Pattern of an undirected graph with its diagonal; relabelled at random where a seed is given."""
    e = np.asarray(edges, np.int64).reshape(-1, 2)
    if seed is not None:
        e = np.random.default_rng(seed).permutation(n)[e]
    i = np.concatenate([e[:, 0], e[:, 1], np.arange(n)])
    j = np.concatenate([e[:, 1], e[:, 0], np.arange(n)])
    order = np.lexsort((j, i))
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(i, minlength=n), out=rp[1:])
    return rp, j[order].astype(np.int32)


def _same(rp, ci, on_gpu=True):
    dev, used = g.rcm_device(rp, ci)
    assert used == on_gpu
    np.testing.assert_array_equal(dev, g.rcm(rp, ci))


@pytest.mark.parametrize("leaves", [1, 7, 8, 9, 63, 64, 65])
def test_children_of_one_node(gpu, leaves):
    """A path of ten nodes whose far end has all the leaves: the order starts at node 0, the path's other end."""
    path = [(i, i + 1) for i in range(9)]
    _same(*_csr(10 + leaves, path + [(9, 10 + k) for k in range(leaves)]), on_gpu=leaves <= 64)


@pytest.mark.parametrize("fan", [(60, 60, 2, 1, 1), (50, 60, 7, 1), (40, 3, 1)])
def test_wide_levels(gpu, fan):
    """Trees whose levels go from one node to 7,200 and 21,000 nodes, with levels as wide behind them."""
    edges, level, n = [], [0], 1
    for f in fan:
        nxt = []
        for p in level:
            kids = range(n, n + f)
            n += f
            edges += [(p, k) for k in kids]
            nxt += kids
        level = nxt
    _same(*_csr(n, edges, seed=n))


def test_mesh_levels_wider_than_the_lane_groups(gpu):
    d = g.fem3d(112, perm_seed=2)[0]
    _same(d.row_ptr, d.col_idx)


def test_components_and_single_nodes(gpu):
    """Paths, cycles and nodes without neighbours, relabelled together."""
    edges = [(i, i + 1) for i in range(40)] + [(50 + i, 50 + (i + 1) % 17) for i in range(17)] + [(80, 81)]
    _same(*_csr(100, edges, seed=3))


@pytest.mark.parametrize("leaves", [64, 65, 200])
def test_a_wide_root_is_seen_in_the_first_search(gpu, leaves):
    """Node 0, where the first search starts, has a path of ten nodes and the leaves: as many children as neighbours there,
    one fewer in the order from the far end.  The host takes over as soon as a search counts more than 64."""
    path = [(i, i + 1) for i in range(9)]
    _same(*_csr(10 + leaves, path + [(0, 10 + k) for k in range(leaves - 1)]), on_gpu=leaves <= 64)
