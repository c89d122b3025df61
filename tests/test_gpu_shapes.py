"""CTA shapes on the GPU: what is told is launched, and group launches of a single job take the batch rule's
shape unless the caller set a slot budget or device memory does not hold its slots; the same bits by every route."""

import numpy as np
import pytest

from p3s_gb300.group import GpuGroup, GroupJob
from p3s_gb300.solver import GpuSolver
from p3s_gb300.synthetic import make_grid, scenario_injections

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_a_slot_budget_that_was_set_holds_for_an_only_job():
    """16,384, the default's figure, set by the caller (a server does so): the shape of the group rule, whose
    schedules the server's warm-up has built, and not the batch rule's."""
    g = make_grid(257, seed=257, max_drop_pu=0.05)
    S = scenario_injections(g, 744, seed=1)
    s = GpuSolver(g.Yp, g.Yj, g.Yx, g.pv, g.pq)
    grp = GpuGroup()
    p = GpuSolver.params(precision="mixed")
    first = None
    for budget in (0, 16384, 16385, 16383, 1, 0):
        grp.set_shape(0, budget)
        r = grp.solve([GroupJob(s, S, g.V0)], p)[0]
        first = first or r
        assert (grp.stats["threads_per_cta"] == 512) == (budget > 0)
        assert np.array_equal(r["V"], first["V"]) and np.array_equal(r["iterations"], first["iterations"])


def test_an_only_job_runs_where_memory_holds_the_group_rules_slots_only():
    """4,864 cases of 2,000 buses: the batch rule's 32 slots an SM take 4,864 slots, the group rule's 8 a CTA
    2,432. With room for about 3,600 of them (and the call's arrays) the launch takes the group rule."""
    g = make_grid(2000, seed=7, max_drop_pu=0.05)
    T = 4864
    S = np.ascontiguousarray(scenario_injections(g, 16, seed=5)[:, np.arange(T) % 16])
    s = GpuSolver(g.Yp, g.Yj, g.Yx, g.pv, g.pq)
    p = GpuSolver.params(precision="mixed", shared_start=False)
    s.prepare_shapes(32)
    want = GpuGroup().solve([GroupJob(s, S, g.V0)], p)[0]
    nf = s.info["n_blocks"] + s.info["n_var_bus"]
    slot = nf * 64 + s.info["n_var_bus"] * 40 + g.n * 93
    grp = GpuGroup()
    grp.solve([GroupJob(s, np.ascontiguousarray(S[:, :1]), g.V0)], p)
    room = 3600 * slot + 2 * S.nbytes + (256 << 20)
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
    try:
        got = grp.solve([GroupJob(s, S, g.V0)], p)[0]
        shape = grp.stats["threads_per_cta"], grp.stats["cases_per_cta"]
    finally:
        del held
        torch.cuda.empty_cache()
    assert shape == (512, 16)  # (the most slots that the group rule gives any job)
    assert np.array_equal(got["V"], want["V"]) and np.array_equal(got["iterations"], want["iterations"])


@pytest.mark.parametrize("n,cases", [(118, 1), (118, 4000), (490, 96), (490, 6500)])
def test_the_shape_told_is_the_shape_launched(n, cases):
    """Batches whose shape differs between the precisions; without a word the precision is the parameters'
    default, double."""
    g = make_grid(n, seed=n, max_drop_pu=0.05)
    S = scenario_injections(g, cases, seed=1)
    s = GpuSolver(g.Yp, g.Yj, g.Yx, g.pv, g.pq)
    told = {precision: s.shape(cases, precision) for precision in ("double", "mixed")}
    assert told["double"] != told["mixed"] and s.shape(cases) == told["double"]
    for precision, shape in told.items():
        s.solve_batch(S, g.V0, GpuSolver.params(precision=precision))
        assert (s.stats["threads_per_cta"], s.stats["cases_per_cta"]) == shape


@pytest.mark.parametrize("shared_start", [-1, 0, 1, 2, 3])
def test_a_group_shares_the_start_for_the_values_a_solver_does(shared_start):
    """Any value but 0 (never) and 2 (where it pays: not for 200 cases of 65 buses) shares the start."""
    g = make_grid(65, seed=65, max_drop_pu=0.05)
    S = scenario_injections(g, 200, seed=1)
    s = GpuSolver(g.Yp, g.Yj, g.Yx, g.pv, g.pq)
    p = GpuSolver.params()
    p.shared_start = shared_start
    grp = GpuGroup()
    got, want = grp.solve([GroupJob(s, S, g.V0)], p)[0], s.solve_batch(S, g.V0, p)
    assert grp.stats["first_steps"] == s.stats["first_steps"] == (0 if shared_start in (0, 2) else 200)
    assert np.array_equal(got["V"], want["V"]) and np.array_equal(got["iterations"], want["iterations"])
