"""Launches of few cases per CTA on the GPU, where one lane or four work on a factorization task:
grids around the sizes where levels change over, 1 to 8 slots a CTA, both precisions. Every
CTA shape forms the same numbers, so a case's result must be bit-identical whatever its launch,
and within the double path's 1e-11 of the oracle."""

from fractions import Fraction

import numpy as np
import pytest

from oracle import cpu
from oracle import islands as oislands
from p3s_gb300 import _lib, contingency
from p3s_gb300.group import GpuGroup, GroupJob
from p3s_gb300.solver import GpuSolver
from p3s_gb300.synthetic import make_grid, scenario_injections

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 30, 65, 257, 1031])
def test_small_shapes_agree_bit_for_bit(n):
    g = make_grid(n, seed=n, max_drop_pu=0.05)
    S = scenario_injections(g, 13, seed=n)
    ref = cpu.Solver(g.Yp, g.Yj, g.Yx, g.pv, g.pq).solve_batch(S, g.V0)
    s = GpuSolver(g.Yp, g.Yj, g.Yx, g.pv, g.pq)
    # (the reference's votes take every mixed case through a double Jacobian and factorization)
    for precision, rule in (("double", "gb300"), ("mixed", "gb300"), ("mixed", "reference")):
        p = GpuSolver.params(precision=precision, vote_rule=rule)
        first = None
        for nt, slots in ((1024, 1), (1024, 4), (512, 1), (512, 2), (512, 8), (256, 4), (512, 16), (512, 32)):
            s.set_shape(13, nt, slots)
            r = s.solve_batch(S, g.V0, p)
            if first is None:
                first = r
            assert np.array_equal(r["V"], first["V"]) and np.array_equal(r["iterations"], first["iterations"])
        assert np.array_equal(first["converged"], ref["converged"]) and ref["converged"].all()
        if precision == "double":
            assert np.array_equal(first["iterations"], ref["iterations"])
            assert np.abs(first["V"] - ref["V"]).max() < 1e-11


@pytest.mark.parametrize("cases", [15, 16, 153, 3200])
def test_shared_start_where_it_pays_changes_no_result(cases):
    """Below 16 cases never, then only where the prologue pays (3,200 cases of 257 buses: double yes, mixed
    no): the same bits as always and never sharing the start."""
    g = make_grid(257, seed=257, max_drop_pu=0.05)
    S = scenario_injections(g, cases, seed=3)
    s = GpuSolver(g.Yp, g.Yj, g.Yx, g.pv, g.pq)
    for precision in ("double", "mixed"):
        r, first = {}, {}
        for how in (True, False, "auto"):
            r[how] = s.solve_batch(S, g.V0, GpuSolver.params(precision=precision, shared_start=how))
            first[how] = s.stats["first_steps"]
        assert first[True] == (cases if cases >= 16 else 0) and first[False] == 0
        assert first["auto"] == (cases if cases == 3200 and precision == "double" else 0)
        for how in (False, "auto"):
            assert np.array_equal(r[how]["V"], r[True]["V"])
            assert np.array_equal(r[how]["iterations"], r[True]["iterations"])
        assert r[True]["converged"].all()


@pytest.mark.parametrize("cases", [3084, 3085, 52428, 52429])
def test_results_by_the_staging_block_and_directly(cases):
    """5 buses: voltages, iterations and flags of 3,084 cases fit the page-locked block, of 3,085 only the
    iterations and flags, of 52,429 nothing: the same bits from each, for a solver and a group."""
    g = make_grid(5, seed=5, max_drop_pu=0.05)
    S3 = scenario_injections(g, 3, seed=2)
    s = GpuSolver(g.Yp, g.Yj, g.Yx, g.pv, g.pq)
    p = GpuSolver.params()
    want = s.solve_batch(S3, g.V0, p)
    S = np.ascontiguousarray(S3[:, np.arange(cases) % 3])
    grp = GpuGroup()
    few, many = grp.solve([GroupJob(s, S3, g.V0), GroupJob(s, S, g.V0)], p)
    for got in (s.solve_batch(S, g.V0, p), many):
        assert np.array_equal(got["V"], want["V"][:, np.arange(cases) % 3])
        assert np.array_equal(got["iterations"], want["iterations"][np.arange(cases) % 3])
        assert got["converged"].all()
    assert np.array_equal(few["V"], want["V"]) and few["converged"].all()


def test_dc_starts_share_work_arrays():
    """Few, many (work arrays freed after the call) and few cases again, with and without DC stamps."""
    g = make_grid(257, seed=257, max_drop_pu=0.05)
    s = GpuSolver(g.Yp, g.Yj, g.Yx, g.pv, g.pq)
    is_slack = np.zeros(g.n, np.uint8)
    is_slack[np.asarray(g.ref)] = 1
    s.set_branches(g.f, g.t, g.stamp_pos, g.stamp, is_slack)
    P3 = np.ascontiguousarray(scenario_injections(g, 3, seed=4).real)
    for stamps in (None, g.stamp):
        want = [s.dc_start(np.ascontiguousarray(P3[:, k]), g.V0, dc_stamps=stamps)[0] for k in range(3)]
        for cases in (3, 17000, 3):
            V, used = s.dc_start(np.ascontiguousarray(P3[:, np.arange(cases) % 3]), g.V0, dc_stamps=stamps)
            assert used.all()
            for k in range(3):
                assert np.array_equal(V[:, k::3], np.repeat(want[k][:, None], len(range(k, cases, 3)), axis=1))


@pytest.mark.parametrize("n,cases", [(1, 1), (4, 7), (28, 8), (29, 9), (36, 17), (37, 3), (1000, 33),
                                     (1256, 9), (1257, 9), (2536, 5), (2537, 5), (4096, 5), (4097, 5)])
def test_islands_at_the_edges_of_both_kernels(n, cases):
    """Labels in shared memory with four, two and one case a CTA up to 1,256, 2,536 and 4,096 buses, in
    global memory beyond: random graphs with many components, self-loops, parallel and dead branches,
    equal priorities."""
    rng = np.random.default_rng(n + cases)
    m = int(1.1 * n)
    f, t = rng.integers(0, n, m).astype(np.int32), rng.integers(0, n, m).astype(np.int32)
    t[: m // 2] = np.minimum(f[: m // 2] + 1, n - 1)  # long chains: the deepest trees
    live = rng.random(m) < 0.9
    groups = [rng.choice(m, size=min(m, int(rng.integers(0, 4))), replace=False) for _ in range(cases)]
    prio = rng.integers(-1, 3, n).astype(float)
    ref = np.unique(rng.integers(0, n, max(1, n // 50)))
    batch = contingency.ContingencyBatch(None, None, None, n, groups, None, None, ref, f, t, live, None)
    for reslack in (True, False):
        got = contingency.islands(batch, reslack, prio)
        want = oislands.islands(n, f, t, live, groups, ref, reslack, prio)
        for a, b in zip(got, want):
            assert np.array_equal(a, b)


def test_stamps_beside_plain_jobs_of_other_slot_counts():
    """A group launch's outage stamps lie behind the slots of each job: an outage job of few slots beside a
    plain one of many, and the other way round, give the bits of each job alone."""
    g = make_grid(65, seed=65, max_drop_pu=0.05)
    s = GpuSolver(g.Yp, g.Yj, g.Yx, g.pv, g.pq)
    is_slack = np.zeros(g.n, np.uint8)
    is_slack[np.asarray(g.ref)] = 1
    s.set_branches(g.f, g.t, g.stamp_pos, g.stamp, is_slack, np.maximum(g.p_gen, 0.0))
    S = scenario_injections(g, 40, seed=6)
    groups = [[], *[[b] for b in range(39)]]
    out = contingency.outage_lists(groups)
    grp = GpuGroup()
    for precision in ("double", "mixed"):
        p = GpuSolver.params(precision=precision)
        for few, many in ((1, 32), (32, 1), (4, 4)):
            jobs = [GroupJob(s, S, g.V0, cases_per_cta=many),
                    GroupJob(s, np.asarray(g.Sbus), g.V0, n_cases=40, outages=out, reslack=True, cases_per_cta=few)]
            both = grp.solve(jobs, p)
            for r, job in zip(both, jobs):
                alone = grp.solve([job], p)[0]
                assert np.array_equal(r["V"], alone["V"], equal_nan=True)
                assert np.array_equal(r["iterations"], alone["iterations"])
                assert np.array_equal(r["converged"], alone["converged"])
        assert not np.array_equal(both[1]["V"][:, 1], both[1]["V"][:, 0])


@pytest.mark.parametrize("exponent", [-126, -32, -31, -1, 0, 1, 30, 31, 125])
def test_reciprocal_seed_is_rounded_to_nearest(exponent):
    """Inside and outside the range whose seed is converted on the integer pipes (2^-31 to 2^31): the bits
    of a float reciprocal of the nearest float, refined by two fused Newton steps; ties, carries into the
    exponent and neighbours of powers of two."""
    rng = np.random.default_rng(exponent + 200)
    man = np.concatenate([rng.integers(0, 1 << 52, 200), rng.integers(0, 1 << 23, 50) << 29,
                          (rng.integers(0, 1 << 23, 50) << 29) + (1 << 28), [0, 1, (1 << 52) - 1, (1 << 28) - 1, 1 << 28]])
    x = np.ldexp(1.0 + man.astype(np.float64) * 2.0 ** -52, exponent)
    outs = [np.empty(len(x)) for _ in range(5)]
    rc = _lib.load().gbpf_selftest_math(_lib.d(x), len(x), *[_lib.d(o) for o in outs], None, None)
    assert rc == 0, _lib.last_error()
    seed = (np.float32(1.0) / x.astype(np.float32)).astype(np.float64)
    for a, r, got in zip(x, seed, outs[0]):
        for _ in range(2):
            r = float(r) * float(2 - Fraction(float(a)) * Fraction(float(r)))
        assert got == r


@pytest.mark.parametrize("n", [14, 65, 257, 617])
@pytest.mark.parametrize("cases", [1, 153, 305, 457])
def test_shapes_of_small_shares_agree_bit_for_bit(n, cases):
    """One to four cases an SM on grids below and above the lines between 256, 512 and 1,024 threads: the
    chosen shape's results are those of one 1,024-thread CTA with four slots."""
    g = make_grid(n, seed=n, max_drop_pu=0.05)
    S = scenario_injections(g, cases, seed=n)
    s = GpuSolver(g.Yp, g.Yj, g.Yx, g.pv, g.pq)
    for precision in ("double", "mixed"):
        p = GpuSolver.params(precision=precision)
        auto = s.solve_batch(S, g.V0, p)
        s.set_shape(cases, 1024, 4)
        r = s.solve_batch(S, g.V0, p)
        s.set_shape(cases, 0, 0)
        for key in ("V", "iterations", "converged"):
            assert np.array_equal(auto[key], r[key])
        assert auto["converged"].all()
