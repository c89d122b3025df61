"""The CTA shape rules without a GPU: batches of every size up to where the rule is constant, small to
very large grids, both precisions, with and without outages; and the edges of the plan check's arguments."""

import ctypes as C

import numpy as np
import pytest

from p3s_gb300 import _lib
from p3s_gb300.synthetic import make_grid
from test_host_cpu import _selftest

GRIDS = (1, 13, 64, 65, 117, 250, 251, 399, 400, 600, 601, 1500, 1999, 3500, 4096, 4097, 8192, 16384, 16385, 19999)


def _rule(nsm, nv, units, mixed, outages, slot_budget=0):
    nt, g = C.c_int(), C.c_int()
    assert _lib.load().gbpf_selftest_shape(nsm, nv, units, mixed, outages, slot_budget, C.byref(nt), C.byref(g)) == 0
    return nt.value, g.value


def _prepared(nsm, nv, most):
    out = np.zeros(64, np.int32)
    k = _lib.load().gbpf_selftest_shapes(nsm, nv, most, _lib.i32(out), 32)
    assert 0 < k <= 32, _lib.last_error()
    return {(int(a), int(b)) for a, b in out[: 2 * k].reshape(-1, 2)}


@pytest.mark.parametrize("nsm", [8, 148, 152])
def test_every_shape_of_a_launch_is_prepared(nsm):
    """Up to 70 cases an SM every batch, then every seventh up to 200 an SM, and a batch that fills any device."""
    sizes = [*range(1, 70 * nsm + 1), *range(70 * nsm, 200 * nsm, 7), 1 << 40]
    if nsm != 152:
        sizes = sizes[::11]
    for nv in GRIDS:
        seen = {_rule(nsm, nv, units, mixed, outages) for units in sizes for mixed in (0, 1) for outages in (0, 1)}
        for most in (1, 4, 32):
            used = {(nt, g) for nt, g in seen if g <= most}
            used |= {(nt, 1) for nt, _ in used} | {(1024, 1)}  # a CTA's last case, the shared start
            # a group of several grids: 512 threads, or 1,024 with up to four slots
            used |= {(nt, g) for nt in (512, 1024) for g in (1, 2, 4, 8, 16, 32) if g <= min(most, 4 if nt == 1024 else 32)}
            prepared = _prepared(nsm, nv, most)
            assert used <= prepared, (nv, most, used - prepared)
            assert max(g for _, g in prepared) <= most


@pytest.mark.parametrize("budget", [1, 8192, 16384, 65536])
def test_group_shapes_keep_within_the_slot_budget(budget):
    """Variable buses x slots of a CTA stay within a group's budget (one slot at least), and a server's warm-up,
    which prepares as many slots as the budget allows, has the shape."""
    for nv in GRIDS:
        most = 1
        while most < 32 and 2 * most * nv <= budget:
            most *= 2
        prepared = _prepared(152, nv, most)
        for units in (*range(1, 152 * 70, 97), 1 << 40):
            nt, g = _rule(152, nv, units, 0, 0, budget)
            assert g == 1 or nv * g <= budget, (nv, units, nt, g)
            assert {(nt, g), (nt, 1)} <= prepared, (nv, units, nt, g)


@pytest.mark.parametrize("workers", [0, -3])
def test_a_plan_for_no_workers_is_checked_with_one(workers):
    err, _ = _selftest(make_grid(30, seed=4), workers)
    assert err < 1e-9, err  # the bound of the other plan checks
