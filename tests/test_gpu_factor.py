"""The factorization and the solves at the sizes where their tiles, slices and
cluster splits change: dense tails around one and several 32- and 64-wide
panels, remainders, grids without a head, and every cluster size."""

import numpy as np
import pytest

from conftest import TOL_V_FP64, TOL_V_MIXED
from gpusim2grid_b200 import (AcPfGPU, ContingencyAnalysisGPU, InjectionSweepGPU, RowStatus, ScenarioSweepGPU,
                              compute_many)
from gpusim2grid_b200.synthetic import grid_by_name, injection_scenarios, make_grid, n1_branches, scenario_outages
from oracle.nr_oracle import nr_solve

pytestmark = pytest.mark.gpu


def _grid(n):
    branches = min(n * (n - 1) // 2, max(n - 1, int(1.58 * n)))
    return make_grid(n, branches, n // 5, max(1, int(0.75 * n)), seed=n, load_scale=0.1)


# tails (default plan): from a handful of unknowns to several panels, whole and ragged;
# 130 to 210: where a row's workspace stops fitting in shared memory (FP64, then FP32)
SIZES = [2, 3, 9, 40, 83, 84, 95, 118, 130, 140, 150, 190, 210, 231, 402, 700]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_solves_match_the_oracle(n, precision):
    g = _grid(n)
    p, q = injection_scenarios(g, 5, seed=3)
    Y, V0, _, _, _, pv, pq = g.as_tuple()
    sw = InjectionSweepGPU(g.as_tuple(), init_from_n_powerflow=False, precision=precision, nb_iter=10,
                           scheduling="continuous", start="flat")
    sw.set_injections(p, q, g.sn_mva)
    for policy in (0, 1):  # the exact trailing clique, and the cost model's tail
        sw.session.replan(policy, 40.0, -1)
        sw.compute()
        V, _, st, it = sw.results_view()
        for r in range(5):
            Vo, so, io, _ = nr_solve(Y, V0, (p[r] + 1j * q[r]) / g.sn_mva, pv, pq, max_iter=10, tol=1e-8)
            assert st[r] == so == 0
            if precision == "fp64":
                assert it[r] == io
            assert np.abs(V[r] - Vo).max() <= (TOL_V_FP64 if precision == "fp64" else TOL_V_MIXED)


# (buses, rows, CTAs per row): dense tails of 133 (no clusters), 150 (none of 2), 204 (an SM
# to each CTA) and 341 (two on an SM); rows well inside what any B200 holds of each size
CLUSTERS = [(402, 1, 0), (402, 20, 0), (500, 1, 16), (500, 10, 8), (500, 25, 4), (500, 50, 0), (700, 1, 16),
            (700, 12, 8), (700, 25, 4), (700, 60, 2), (700, 100, 0), (1200, 1, 16), (1200, 20, 8), (1200, 50, 4),
            (1200, 100, 2), (1200, 149, 0)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,rows,size", CLUSTERS)
def test_small_batches_on_clusters_equal_one_cta_per_row(n, rows, size, precision):
    """Clusters of 16, 8, 4 and 2 CTAs and none, by the dense tail and the number of rows."""
    g = _grid(n)
    p, q = injection_scenarios(g, rows, seed=5)
    out = []
    for cluster in (1, 0):
        sw = InjectionSweepGPU(g.as_tuple(), init_from_n_powerflow=False, precision=precision, nb_iter=10,
                               scheduling="continuous", start="flat")
        sw.session.set_handoff(cluster)
        sw.set_injections(p, q, g.sn_mva)
        sw.compute()
        assert sw.session.cluster_size() == (size if cluster else 0)
        out.append([a.copy() for a in sw.results_view()])
        assert np.all(out[-1][2] == 0)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


FORMS = {
    "chunked": dict(nb_iter=6),
    "rounds": dict(scheduling="continuous", nb_iter=6, nb_iter_per_round=2),
    "adaptive": dict(scheduling="continuous", nb_iter=10, strategy="adaptive"),
    "scaled": dict(scheduling="continuous", nb_iter=10, scaling_max_voltage_change=True, max_dVa=0.05, max_dVm=0.01),
    "masked": dict(scheduling="continuous", nb_iter=10, handle_disconnected_grid=True),
    "base_chord": dict(scheduling="continuous", nb_iter=10, strategy="base_chord"),
}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("form", FORMS)
def test_options_on_clusters_equal_one_cta_per_row(form, precision):
    """Outage rows (some split the grid, one has a start that is not finite) in every
    schedule and option, on clusters and on one CTA each: the same bits."""
    g = _grid(700)
    safe = set(int(b) for b in n1_branches(g))
    splits = [b for b in range(g.n_branch) if b not in safe][:4]
    rows = [[b] for b in splits] + [[b] for b in sorted(safe)[:6]] + [sorted(safe)[8:10]]
    out = []
    for cluster in (1, 0):
        ca = ContingencyAnalysisGPU(g.as_tuple(), init_from_n_powerflow=False, precision=precision, **FORMS[form])
        ca.set_branch_data(*g.branch_data())
        ca.set_branch_limits(np.full(g.n_branch, 50.0))
        ca.add_contingencies_by_branch_id(rows)
        ca.session.set_handoff(cluster)
        if form == "base_chord":
            ca.session.set_chord(0)  # every row in the single-row sweep
        start = np.tile(g.vinit(), (len(rows), 1))
        start[5] = np.nan
        ca.set_start_voltages(start)
        ca.compute()
        if form != "masked":  # (there the FP64 re-solve of a failed row may be the last run)
            assert ca.session.cluster_size() == (8 if cluster else 0)
        out.append([ca.V_results, ca.get_row_status(), ca.get_row_iterations(), ca.get_row_factorizations(),
                    *ca.branch_loading()])
    assert len(splits) == 4 and np.any(out[0][1] == RowStatus.CONVERGED)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n_ctas,sizes", [(0, {16}), (4, {0}), (8, {2}), (64, {16}), (63, {8})])
def test_a_callers_cta_count_bounds_the_clusters(n_ctas, sizes):
    """n_ctas is the number of CTAs a run may have, clusters included."""
    from gpusim2grid_b200._native import lib
    g = _grid(900)
    p, q = injection_scenarios(g, 4, seed=5)
    sw = InjectionSweepGPU(g.as_tuple(), init_from_n_powerflow=False, precision="fp64", nb_iter=10,
                           scheduling="continuous", start="flat")
    sw.set_injections(p, q, g.sn_mva)
    s = sw.session
    for rows in (None, np.arange(4, dtype=np.int32)):  # the whole batch, then a subset of it
        if rows is None:
            s.run(10, 1e-8, False, lib.PREC_FP64, lib.START_VINIT, n_ctas=n_ctas)
        else:
            s.run_subset(rows, 10, 1e-8, False, lib.PREC_FP64, lib.START_VINIT, n_ctas=n_ctas)
        assert s.cluster_size() in sizes
        assert np.all(s.results()[2] == 0)
    # a base solve, whose callers give no count, has the device
    s.solve_base(10, 1e-8, lib.PREC_FP64)
    assert s.cluster_size() == 16


def _leaving(g, rows, seed):
    """A mixed sweep whose rows all leave the chord for their own factor."""
    p, q = injection_scenarios(g, rows, seed=seed)
    sw = InjectionSweepGPU(g.as_tuple(), init_from_n_powerflow=False, precision="mixed", nb_iter=10,
                           scheduling="continuous", strategy="base_chord")
    sw.refactor_ratio = 1e-9
    sw.set_injections(p, q, g.sn_mva)
    return sw


@pytest.mark.parametrize("multi", [False, True])
def test_handoffs_get_clusters_by_the_chip(multi):
    """The rows that a chord sweep hands off share the chip, however few rows
    the batch had."""
    sweeps = [_leaving(_grid(n), 3, n) for n in ((900, 700) if multi else (900,))]
    compute_many(sweeps) if multi else sweeps[0].compute(batch_size=0)
    for sw in sweeps:
        assert np.all(sw.get_row_factorizations() > 0)
        assert sw.session.cluster_size() in (8, 16)


def test_single_solve_on_a_cluster_equals_one_cta():
    g = grid_by_name("case2000_synth", 0)
    got = []
    for cluster in (1, 0):
        ac = AcPfGPU(g.as_tuple(), init_from_n_powerflow=False)
        ac.session.set_handoff(cluster)
        t = ac.resolve(g.vinit(), 1.05 * g.sbus())
        got.append((ac.solve(), t.nb_iter, t.residual))
    np.testing.assert_array_equal(got[0][0], got[1][0])
    assert got[0][1:] == got[1][1:]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("rows,size", [(1, 16), (10, 8), (25, 4), (50, 2), (90, 0)])
def test_multi_grid_handoffs_on_clusters_equal_one_cta_per_row(rows, size, precision):
    """Every row of a small and a large grid leaves the chord; the small grid's
    (dense tail 42) are run by one CTA of their cluster."""
    grids = [grid_by_name("case118_synth", 0), grid_by_name("case2000_synth", 0)]
    out = []
    for cluster in (1, 0):
        sweeps = []
        for i, g in enumerate(grids):
            p, q = injection_scenarios(g, rows, seed=20 + i)
            f = ScenarioSweepGPU(g.as_tuple(), init_from_n_powerflow=False, precision=precision, nb_iter=10,
                                 scheduling="continuous", strategy="base_chord")
            f.refactor_ratio = 1e-9
            f.set_branch_data(*g.branch_data())
            f.set_injections(p, q, g.sn_mva)
            f.set_topology(scenario_outages(g, rows, seed=40 + i))
            f.session.set_handoff(cluster)
            sweeps.append(f)
        compute_many(sweeps)
        for f in sweeps:
            ran = f.results_view()[2] != RowStatus.NOT_SIMULATED  # an outage that splits the grid is not simulated
            assert np.any(ran) and np.all(f.get_row_factorizations()[ran] > 0)
            assert f.session.cluster_size() == (size if cluster else 0)
        out.append([a.copy() for f in sweeps for a in f.results_view()])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n", [84, 402])
def test_base_chord_rows_match_the_oracle(n):
    g = _grid(n)
    rows = [[int(b)] for b in n1_branches(g)[:60]]
    Y, V0, S, _, _, pv, pq = g.as_tuple()
    from oracle.nr_oracle import trip_branches
    ca = ContingencyAnalysisGPU(g.as_tuple(), init_from_n_powerflow=False, precision="mixed", nb_iter=10,
                                scheduling="continuous", strategy="base_chord")
    ca.set_branch_data(*g.branch_data())
    ca.add_contingencies_by_branch_id(rows)
    ca.compute()
    V, _, st, _ = ca.results_view()
    for r, ids in enumerate(rows):
        Yr = trip_branches(Y, ids, g.branch_from, g.branch_to, g.yff, g.yft, g.ytf, g.ytt)
        Vo, so, _, _ = nr_solve(Yr, V0, S, pv, pq, max_iter=10, tol=1e-8)
        assert st[r] == so == 0
        assert np.abs(V[r] - Vo).max() <= TOL_V_MIXED


def test_small_results_in_every_run_and_session():
    """A session's first run and results are copied one by one, later ones
    through a pinned block, of which there are 32: every copy is the same."""
    g = _grid(40)
    p, q = injection_scenarios(g, 3, seed=4)
    sweeps = []
    ref = None
    for _ in range(34):
        sw = InjectionSweepGPU(g.as_tuple(), init_from_n_powerflow=False, precision="fp64", nb_iter=10,
                               scheduling="continuous", start="flat")
        sw.set_injections(p, q, g.sn_mva)
        for _ in range(3):
            sw.compute()
            got = [a.copy() for a in sw.session.results()] + [sw.session.timings()["total_iters"]]
            ref = ref or got
            for a, b in zip(got, ref):
                np.testing.assert_array_equal(a, b)
        sweeps.append(sw)
    assert ref[-1] == ref[3].sum()
