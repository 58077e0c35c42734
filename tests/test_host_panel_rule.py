"""Which jobs are evaluated as panels, checked on the CPU: a job whose panels cost more than its forms, or more memory,
keeps the forms; one whose pairs are products of waves takes panels."""
import numpy as np
import pytest
import torch

import bench
from dwba_b200 import engine as E

N, L_MAX = 160, 6


def _job(sets, n_i, n_f, T, one_ui=True, disjoint=False, eng="semisep", k0=1.0, **kw):
    from dwba_b200.dwba_matrix_elements import _make_job
    from dwba_b200.plan import GridInfo
    g = bench.make_grid(N, 0.05, 300.0)

    class Cache:
        info = GridInfo(g.r, g.w_simpson, g.w_trapz)
        dg = E.DeviceGrid(info, torch.device("cpu"))
    rng = np.random.default_rng(3)
    pairs = []
    for s in range(sets):
        wi = [bench._Wave(l % 5, k0 + 0.01 * s, 0.0, rng.normal(size=N)) for l in range(n_i)]
        wf = [bench._Wave(l % 5, 0.7, 0.0, rng.normal(size=N)) for l in range(n_f)]
        pairs += list(zip(wi, wf)) if disjoint else [(a, b) for a in wi for b in wf]
    u = [np.exp(-(1 + 0.1 * t) * g.r) for t in range(T)]
    b_i = [bench._Bound(0, u[0] if one_ui else u[t]) for t in range(T)]
    b_f = [bench._Bound(1, g.r * u[t]) for t in range(T)]
    z = np.zeros(N)
    job = _make_job(g, z, z, b_i, b_f, pairs, L_MAX, z, {}, Cache)
    assert E.panel_work(job) >= E.PANEL_MIN_WORK
    return E.PreparedJob(job, Cache.dg, eng, rebuild_nodesets=True, **kw)


@pytest.mark.parametrize("sets,n_i,n_f,T,one_ui,disjoint,part,want", [
    (40, 1, 1, 8, True, False, False, False),     # one pair per node set: nothing shared on the direct side
    (40, 1, 1, 16, True, False, False, False),
    (100, 2, 2, 4, True, False, False, False),     # many small products
    (40, 4, 4, 4, False, False, False, False),    # a potential per transition and wave
    (1, 60, 60, 8, False, True, False, False),    # pairs of one node set that share no wave
    (1, 20, 20, 1, True, False, False, True),     # an energy point
    (1, 20, 20, 1, True, False, True, True),
    (4, 20, 20, 2, True, False, False, True),
    (1, 6, 6, 8, True, False, False, True),       # transitions of an ejected energy
])
def test_panels_where_they_cost_less(sets, n_i, n_f, T, one_ui, disjoint, part, want):
    pj = _job(sets, n_i, n_f, T, one_ui, disjoint, part=part)
    assert (pj.direct_plan.panels is not None) == want
    if want:
        assert pj.direct_plan.dot_fo.size == pj.direct_plan.ss_fo.size == 0


def test_sets_of_a_job_are_judged_one_by_one():
    """A node set with a product of waves beside many with one pair each: panels for the product alone."""
    big = _job(1, 20, 20, 8)
    small = _job(40, 1, 1, 8, k0=1.1)
    job = big.job
    job.pairs, job._packed = big.job.pairs + small.job.pairs, None
    job._waves, job._wave_idx = None, (None, None)
    pj = E.PreparedJob(job, big.dg, "semisep", rebuild_nodesets=True)
    pp = pj.direct_plan.panels
    assert pp is not None and len(pp.direct.fo) == len(pp.exchange.fo) == 8 * 400
    assert len(pj.direct_plan.dot_fo) == len(pj.direct_plan.ss_fo) == 8 * 40


def test_memory_bound(monkeypatch):
    """With many multipoles the potentials and psi blocks outgrow the forms' operand rows."""
    args = (1, 20, 20, 2)
    assert _job(*args).direct_plan.panels is not None
    monkeypatch.setattr(E, "PANEL_FREE_BYTES", 0)
    assert _job(*args).direct_plan.panels is not None  # 42 blocks of 7 rows against 3200 rows
    monkeypatch.setattr(E.SharedOperands, "nbytes", staticmethod(lambda y, n, N, nl: 32 * N * n + 1))
    assert _job(*args).direct_plan.panels is None
    assert _job(*args, panels=True).direct_plan.panels is not None  # asked for


def test_other_engines_share_wherever_every_form_can():
    assert _job(40, 1, 1, 8, eng="dense").dense_panels
    assert not _job(40, 1, 1, 8, one_ui=False, eng="dense").dense_panels  # no operand twice


def test_parts_of_a_split_sweep_follow_the_exact_rule():
    """In a ragged launch only the direct forms of a split-BF16 job are panels."""
    assert _job(40, 1, 1, 8, eng="tc_bf16x3").tc_panels
    assert _job(40, 1, 1, 8, eng="tc_bf16x3", part=True).direct_plan.panels is None
    assert _job(1, 20, 20, 1, eng="tc_bf16x3", part=True).direct_plan.panels is not None
