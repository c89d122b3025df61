"""Cases that outlive the others of their CTA, on the GPU: an hour without a solution among hours that
converge in a few steps, CTAs of 16 and 32 slots with one case left."""

import numpy as np
import pytest

from p3s_gb300.solver import GpuSolver
from p3s_gb300.synthetic import make_grid, scenario_injections

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["double", "mixed"])
@pytest.mark.parametrize("nt,slots", [(256, 16), (512, 16), (512, 32), (1024, 32)])
def test_the_last_case_of_a_cta_has_all_its_threads(nt, slots, precision):
    """A case alone in a CTA of many slots forms and evaluates its points in at most six times the cycles of
    the CTA of the same threads with one slot: both deal NT threads to its rows, and beside 15 or 31 empty
    slots its 8- to 32-byte items lie in sectors of their own, at most four times the memory sectors. With
    the NT / slots threads of one slot in a full CTA it would be 16 or 32 times the instructions."""
    g = make_grid(2000, seed=7, max_drop_pu=0.05)
    S = scenario_injections(g, 1, seed=5)
    s = GpuSolver(g.Yp, g.Yj, g.Yx, g.pv, g.pq)
    p = GpuSolver.params(precision=precision, phase_timers=True)
    cycles, V = {}, {}
    for k in (1, slots):
        s.set_shape(1, nt, k)
        runs = []
        for _ in range(5):
            V[k] = s.solve_batch(S, g.V0, p)["V"]
            assert s.stats["threads_per_cta"] == nt and s.stats["cases_per_cta"] == k
            runs.append([s.stats["phase_cycles"][phase] for phase in ("step", "eval")])
        cycles[k] = np.min(np.asarray(runs, dtype=float), axis=0)
    assert np.array_equal(V[1], V[slots])
    assert (cycles[slots] < 6 * cycles[1]).all(), cycles


@pytest.mark.parametrize("precision", ["double", "mixed"])
@pytest.mark.parametrize("line_search", [True, False])
def test_an_hour_without_a_solution_changes_no_other(precision, line_search):
    """One hour with 30 times the load among 70: the others' bits as without it, its own as alone, whatever the
    slots of its CTA."""
    g = make_grid(257, seed=257, max_drop_pu=0.05)
    S = scenario_injections(g, 70, seed=8)
    bad = S.copy()
    bad[:, 37] *= 30.0
    s = GpuSolver(g.Yp, g.Yj, g.Yx, g.pv, g.pq)
    p = GpuSolver.params(precision=precision, line_search=line_search)
    others = np.arange(70) != 37
    alone = s.solve_batch(np.ascontiguousarray(bad[:, 37:38]), g.V0, p)
    assert not alone["converged"][0]
    for nt, slots in ((1024, 1), (256, 16), (512, 16), (512, 32), (1024, 32)):
        s.set_shape(70, nt, slots)
        want, got = s.solve_batch(S, g.V0, p), s.solve_batch(bad, g.V0, p)
        assert want["converged"].all()
        for key in ("V", "iterations", "converged"):
            assert np.array_equal(got[key][..., others], want[key][..., others])
            assert np.array_equal(got[key][..., 37], alone[key][..., 0], equal_nan=True)
