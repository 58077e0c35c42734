"""The engine tuner keeps a choice for jobs that share their operands apart from one for jobs that do not: the plain
form is the faster engine for some of the first and hundreds of times slower for the others."""
import numpy as np
import pytest
import torch

import bench
from dwba_b200 import tune
from dwba_b200 import engine as E

CANDS = ("semisep", "dense")


def _call(n, shared, L, n_t=1):
    """64 pairs of one grid: 8 x 8 waves, or 128 waves of which every pair has its own two."""
    rng = np.random.default_rng(7)
    g = bench.make_grid(n, 0.01, 200.0)
    wave = lambda l, k: bench._Wave(l, k, 0.0, np.sin(k * g.r + rng.uniform(0, 3)))  # noqa: E731
    if shared:
        wi, wf = [wave(l, 2.0) for l in range(8)], [wave(l, 1.5) for l in range(8)]
        pairs = [(a, b) for a in wi for b in wf]
    else:
        pairs = [(wave(s % 8, 2.0 + 0.01 * s), wave(s // 8, 1.5)) for s in range(64)]
    z = np.zeros(n)
    b_i = [bench._Bound(0, g.r * np.exp(-g.r))] * n_t
    b_f = [bench._Bound(1, g.r ** 2 * np.exp(-(0.5 + 0.1 * t) * g.r)) for t in range(n_t)]
    return g, (z, z), b_i, b_f, pairs, L


def _class(n, shared, L, n_t=1):
    from dwba_b200.dwba_matrix_elements import _make_job
    from dwba_b200.plan import GridInfo
    g, (V, U), b_i, b_f, pairs, L = _call(n, shared, L, n_t)

    class Cache:
        info = GridInfo(g.r, g.w_simpson, g.w_trapz)
        dg = E.DeviceGrid(info, torch.device("cpu"))
    job = _make_job(g, V, U, b_i, b_f, pairs, L, U, {}, Cache)
    return job, E.plan_job(job)


@pytest.mark.parametrize("n_t", [1, 3])
def test_shared_and_unshared_jobs_have_different_keys(n_t):
    a, b, c = _class(150, True, 4, n_t), _class(150, False, 4, n_t), _class(150, True, 4, n_t)
    key = lambda *jobs: tune.TUNER.key(150, 128 * n_t, 4, CANDS, E.sharing_class(jobs, CANDS))  # noqa: E731
    assert key(a)[:4] == key(b)[:4] == (256, tune._pow2(128 * n_t), 4, CANDS)
    assert key(a) == key(c) != key(b)
    assert E.sharing_class([a], CANDS)[:3] == ({1: 8, 3: 32}[n_t], 8, 64)
    assert E.sharing_class([b], CANDS)[:3] == ({1: 1, 3: 4}[n_t], 1, 1)
    assert key(a, a) == key(a) and key(a, b) not in (key(a), key(b))


def test_key_names_the_panels_of_one_call(monkeypatch):
    a = _class(150, True, 4)
    before = E.sharing_class([a], CANDS)
    monkeypatch.setattr(E, "PANEL_ONCE_DENSE", 1.0)  # now one evaluation by the plain form uses panels
    assert before[3:] == (False, False) and E.sharing_class([a], CANDS)[3:] == (False, True)


@pytest.mark.gpu
def test_auto_keeps_a_choice_per_sharing():
    from dwba_b200.dwba_matrix_elements import radial_ME_all_L_batch
    seen = set(tune.TUNER.choices)
    for shared in (True, False):
        g, (V, U), b_i, b_f, pairs, L = _call(1111, shared, 3)
        radial_ME_all_L_batch(g, V, U, b_i, b_f, pairs, L, engine="auto")
    new = set(tune.TUNER.choices) - seen
    assert len(new) == 2 and len({k[:4] for k in new}) == 1
