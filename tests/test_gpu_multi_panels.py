"""Panels of several jobs in one launch (MultiPrepared): grids whose potentials fall in different length classes, more
potentials than one launch takes together, jobs with and without panels side by side, and a captured graph. Reference:
the same jobs by per-pair forms, the same sums in another order: 1e-14 of the sum of the terms' magnitudes, with 1e-12
of the result for the L = 0 corrections and tails added on the host. And the sized potentials at the lengths where the
number of warps changes and where a launch is sized too small, against long-double sums."""
import numpy as np
import pytest

import bench

pytestmark = pytest.mark.gpu


def _job(N, n_i, n_f, L, seed, n_t=1):
    from dwba_b200.dwba_matrix_elements import GPUCache, _make_job
    rng = np.random.default_rng(seed)
    g = bench.make_grid(N, 1e-3, 80.0)
    r = g.r

    def wave(l, k):
        return bench._Wave(l % 7, k, 0.0, np.sin(k * r + rng.uniform(0, 3)) * (1 - np.exp(-(r * k) ** (1 + l % 7))))
    wi, wf = [wave(l, 1.9 + 0.01 * seed) for l in range(n_i)], [wave(l, 1.6) for l in range(n_f)]
    z = np.zeros(N)
    cache = GPUCache.from_grid(g)
    b_f = [bench._Bound(1, r * r * np.exp(-(0.5 + 0.1 * t) * r)) for t in range(n_t)]
    return _make_job(g, z, z, [bench._Bound(0, r * np.exp(-r))] * n_t, b_f, [(a, b) for a in wi for b in wf], L, z, {},
                     cache), cache


def _scale(pj, L):
    """The forms of a per-pair job on the magnitudes of their operands."""
    import torch
    from dwba_b200 import _lib
    ab, f = pj.ops.abs(), pj.forms_host.copy()
    for k in ("a", "b"):
        f[k] = f[k] - pj.ops.data_ptr() + ab.data_ptr()
    fd = torch.from_numpy(f.view(np.uint8).copy()).cuda()
    S = torch.empty((len(f), L + 1), dtype=torch.float64, device="cuda")
    r = pj.job.grid.r
    _lib.check(_lib.load().dwba_bilinear_semisep_fp64(fd.data_ptr(), len(f), L, pj.ds.ctypes.data, float(r[0]), float(r[-1]),
                                                      S.data_ptr(), torch.cuda.current_stream().cuda_stream), "scale")
    return S.cpu().numpy().reshape(pj.T, pj.P, 2, L + 1)


def _check(mp, jobs, L, got):
    from dwba_b200.engine import PreparedJob
    for k, ((job, cache), res) in enumerate(zip(jobs, got)):
        ref = PreparedJob(job, cache.dg, "semisep", rebuild_nodesets=True, fuse_folds=False, panels=False)
        ref.launch()
        want, S = ref.collect(), _scale(ref, L)
        for e in (0, 1):
            assert np.all(np.isfinite(res[e]))
            assert np.all(np.abs(res[e] - want[e]) <= 1e-14 * S[:, :, e] + 1e-12 * np.abs(want[e])), (k, e)


def test_exact_engine_over_length_classes():
    from dwba_b200.engine import MultiPrepared, PreparedJob
    L, sizes = 5, (2040, 2050, 4090, 4100, 8200)
    jobs = [_job(N, 11, 16, L, s, n_t=1 + s % 2) for s, N in enumerate(sizes)] + [_job(1300, 3, 5, L, 9)]
    parts = [PreparedJob(j, c.dg, "semisep", rebuild_nodesets=True, panels=k < len(sizes), part=k % 2 == 0)
             for k, (j, c) in enumerate(jobs)]
    mp = MultiPrepared(parts)
    fl = mp.form_launch
    assert fl.n_pots > 64 and len(fl.pot_runs) == 4 and sum(n for _, n, _ in fl.pot_runs) == fl.n_pots
    assert [p.direct_plan.panels is not None for p in parts] == [True] * 5 + [False]
    mp.launch()
    got = mp.collect()
    _check(mp, jobs, L, got)
    mp.capture()
    mp.out.fill_(float("nan"))
    mp.replay()
    for a, b in zip(got, mp.collect()):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("with_panels", [(True, False, True), (False, True, False, False), (False, False), (True, True)])
def test_plain_engine_with_and_without_panels(with_panels):
    from dwba_b200.engine import MultiPrepared, PreparedJob
    L = 6
    jobs = [_job(N, 4 + s, 5, L, s) for s, N in zip(range(len(with_panels)), (300, 421, 500, 333))]
    parts = [PreparedJob(j, c.dg, "dense", rebuild_nodesets=True, panels=p, part=True)
             for (j, c), p in zip(jobs, with_panels)]
    assert [p.dense_panels for p in parts] == list(with_panels)
    mp = MultiPrepared(parts)
    mp.launch()
    _check(mp, jobs, L, mp.collect())


@pytest.mark.parametrize("engine", ["tc_bf16x6"])
def test_split_engine_direct_forms_of_several_jobs(engine):
    """The exchange forms of a ragged sweep go one column each, the direct forms of all jobs as panels."""
    from dwba_b200.engine import MultiPrepared, PreparedJob
    L = 4
    jobs = [_job(N, 6, 7, L, s) for s, N in enumerate((400, 555, 640))]
    res = []
    for panels in (True, False):
        mp = MultiPrepared([PreparedJob(j, c.dg, engine, rebuild_nodesets=True, panels=panels, part=True) for j, c in jobs])
        mp.launch()
        res.append(mp.collect())
    for (job, cache), a, b in zip(jobs, *res):
        ref = PreparedJob(job, cache.dg, "semisep", rebuild_nodesets=True, fuse_folds=False, panels=False)
        ref.launch()
        S = _scale(ref, L)
        assert np.all(np.abs(a[0] - b[0]) <= 1e-14 * S[:, :, 0] + 1e-12 * np.abs(b[0]))
        assert np.all(np.abs(a[1] - b[1]) <= 1e-14 * S[:, :, 1] + 1e-12 * np.abs(b[1]))


@pytest.mark.parametrize("n,max_len", [(1, 1), (255, 255), (256, 256), (257, 257), (2047, 2047), (2048, 2048), (2049, 2049),
                                       (4096, 4096), (4097, 4097), (8192, 8192), (8193, 8193), (16385, 16385),
                                       (4097, 1), (8193, 2048), (5000, 4096)])
def test_sized_potentials(n, max_len):
    import torch
    from dwba_b200 import _lib
    from dwba_b200.plan import diag_scale
    L_max = 4 if n < 9000 else 1
    rng = np.random.default_rng(n)
    r = np.geomspace(1e-3, 60.0, max(n, 2))[:n]
    b = rng.normal(size=(3, n)) * np.exp(-r / 10)
    rows, cols = (n, n, max(1, n // 3)), (n, max(1, n // 2), n)
    rd, bd = torch.as_tensor(r, device="cuda"), torch.as_tensor(b, device="cuda")
    phi = torch.full((3, L_max + 1, n), np.nan, dtype=torch.float64, device="cuda")
    rec = np.zeros(3, dtype=_lib.POTENTIAL_DTYPE)
    for k in range(3):
        rec[k] = (rd.data_ptr(), bd[k].data_ptr(), phi[k].data_ptr(), rows[k], cols[k], n, 0)
    recd = torch.from_numpy(rec.view(np.uint8).copy()).cuda()
    ds = diag_scale(L_max)
    _lib.check(_lib.load().dwba_multipole_potentials_sized(
        recd.data_ptr(), 3, max_len, L_max, ds.ctypes.data, float(r[0]), float(r[-1]),
        torch.cuda.current_stream().cuda_stream), "potentials")
    got, x = phi.cpu().numpy(), r.astype(np.longdouble)
    for k in range(3):
        y = np.where(np.arange(n) < cols[k], b[k], 0.0).astype(np.longdouble)
        for L in range(L_max + 1):
            lo, hi = x ** L, x ** -(L + 1)

            def f(z):
                suf = np.cumsum((z * hi)[::-1])[::-1] - z * hi
                return (hi * (np.cumsum(z * lo) - z * lo) + lo * suf + (1 - 1e-12) ** L * z / x)[:rows[k]]
            assert np.all(np.abs(got[k, L, :rows[k]] - f(y)) <= 1e-14 * f(np.abs(y))), (k, L)
            assert np.all(np.isnan(got[k, L, rows[k]:]))
