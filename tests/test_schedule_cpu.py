"""The device schedule at the worker counts where its bundles and cuts can go wrong (CPU, serial
execution with a race check per level, double precision): one worker, one per warp, a warp not
filled, 2 to 32 workers a warp; grids whose levels are narrower than a warp, a chain (one
pivot a level), a hub (one row with a pair from every other) and a lattice."""

import numpy as np
import pytest

from p3s_gb300.synthetic import build_ybus, grid_118, make_grid
from test_host_cpu import _selftest, _shaped_grid


@pytest.mark.parametrize("workers", [1, 2, 16, 32, 48, 128, 256, 512, 1024])
@pytest.mark.parametrize("cap", [0.0, 1.0])
def test_warp_programs_solve_the_jacobian(workers, cap):
    for g in (grid_118(), make_grid(30, seed=4), make_grid(501, seed=2, max_drop_pu=0.05)):
        err, _ = _selftest(g, workers, chain_cap=cap)
        assert err < 1e-9, err  # test_host_cpu's bound against scipy's solve of the same Jacobian


def _hub(n):
    """Every bus but the slack's neighbour hangs on that neighbour: one row takes a pair from every other."""
    g = _shaped_grid("star", n)
    f, t = np.r_[0, np.ones(n - 2, int)], np.r_[1, np.arange(2, n)]
    y = 1.0 / (0.01 + 0.1j)
    stamp = np.tile(np.array([y + 0.01j, -y, -y, y + 0.01j]), (n - 1, 1))
    g.Yp, g.Yj, g.Yx, _ = build_ybus(n, f.astype(np.int32), t.astype(np.int32), stamp)
    g.nnz = len(g.Yj)
    return g


@pytest.mark.parametrize("make", [lambda: _shaped_grid("chain", 200), lambda: _hub(200), lambda: _shaped_grid("mesh", 225)],
                         ids=["chain", "hub", "mesh"])
@pytest.mark.parametrize("workers", [1, 32, 1024])
def test_warp_programs_on_extreme_trees(make, workers):
    err, _ = _selftest(make(), workers)
    assert err < 1e-9, err
