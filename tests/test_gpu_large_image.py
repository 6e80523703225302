"""A matrix whose SELL image has more than 2^31 slots: the solve kernels number slots in 32 bits and refuse it, the
product counts in 64 and takes it."""
import numpy as np
import pytest

import project_xplus_b200 as xp

pytestmark = pytest.mark.gpu


def test_solve_refuses_and_spmv_takes_2_31_slots():
    # one row of 4100 entries in each slice of 32, which makes all its rows that wide; the others have a diagonal only
    slices, wide = 16_500, 4100
    n = 32 * slices
    lens = np.ones(n, np.int64)
    lens[::32] = wide
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    first = np.clip(np.arange(0, n, 32) - wide // 2, 0, n - wide)
    ci = np.repeat(np.arange(n, dtype=np.int32), lens)
    at = np.zeros(n + 1, np.int64)
    at[1:] = np.cumsum(lens)
    cols = (first[:, None] + np.arange(wide)).astype(np.int32)
    np.put(ci, (at[:-1:32, None] + np.arange(wide)).reshape(-1), cols.reshape(-1))
    v = np.full(len(ci), -1.0)
    v[ci == np.repeat(np.arange(n, dtype=np.int32), lens)] = 8192.0
    s = xp.PcgSolver(rp, ci, v, sigma=1, keep_fp64=False)
    try:
        assert s.info()["slots"] >= 1 << 31
        x = np.random.default_rng(1).uniform(-1, 1, n)
        y = s.spmv(x)
        # a serial FP32 sum of 4100 terms |x_j - x_i| <= 2 is off by at most 4100^2 / 2 * 2 * 2^-24 = 1.0, the rest by 0.01
        run = np.concatenate([[0.0], np.cumsum(x)])
        rows = np.arange(0, n, 32)
        expect = 8193.0 * x[rows] - (run[first + wide] - run[first])
        assert np.abs(y[rows] - expect).max() < 1.01
        np.testing.assert_allclose(y[1::32], 8192.0 * x[1::32], rtol=1e-6)
        with pytest.raises(RuntimeError, match="2\\^31 slots"):
            s.solve(x, max_iters=1)
    finally:
        s.close()
