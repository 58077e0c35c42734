"""Handles of one grid on several streams: what the grid shares is made with the grid, not by the first handle that
uses it. (On the GPU: two handles on two streams, the first stream busy when the second handle is built, launched
and read; the direct integrals of its panels read the grid's ones.)"""
import numpy as np
import pytest

import bench


def _points(n, device, energies):
    import torch
    from dwba_b200.dwba_matrix_elements import _make_job
    from dwba_b200.engine import DeviceGrid
    from dwba_b200.plan import GridInfo
    g = bench.make_grid(n, 1e-3, 100.0)

    class Cache:
        info = GridInfo(g.r, g.w_simpson, g.w_trapz)
        dg = DeviceGrid(info, torch.device(device))
    rng = np.random.default_rng(11)
    u_i, u_f = g.r * np.exp(-g.r), g.r ** 2 * np.exp(-0.5 * g.r)
    z = np.zeros(n)
    jobs = []
    for k in energies:
        w = [[bench._Wave(l, kk, 0.0, np.sin(kk * g.r + rng.uniform(0, 3))) for l in range(6)] for kk in (k, 0.8 * k)]
        pairs = [(a, b) for a in w[0] for b in w[1]]
        jobs.append(_make_job(g, z, z, [bench._Bound(0, u_i)], [bench._Bound(1, u_f)], pairs, 5, z, {}, Cache))
    return Cache.dg, jobs


def test_handles_share_nothing_made_by_the_first_one(monkeypatch):
    import torch
    from dwba_b200.engine import PreparedJob
    dg, jobs = _points(200, "cpu", (2.0, 1.7))
    ptr = dg.ones.data_ptr()
    assert np.array_equal(dg.ones.numpy(), np.ones(200))
    real, made = torch.ones, []
    monkeypatch.setattr(torch, "ones", lambda *a, **k: made.append(a) or real(*a, **k))
    for job in jobs:
        pj = PreparedJob(job, dg, "semisep", rebuild_nodesets=True, panels=True)
        assert pj.direct_plan.panels.ones == ptr
    assert not made and dg.ones.data_ptr() == ptr


@pytest.mark.gpu
def test_second_handle_does_not_wait_for_the_first_stream():
    import torch
    from dwba_b200.engine import PreparedJob
    warm, (job0,) = _points(500, "cuda", (2.0,))  # tables of the device, not of a grid
    PreparedJob(job0, warm, "semisep", rebuild_nodesets=True, panels=True).launch()
    dg, (job_a, job_b) = _points(3000, "cuda", (2.0, 1.7))
    torch.cuda.synchronize()
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(s1):
        torch.cuda._sleep(200_000_000)  # about 0.1 s
        a = PreparedJob(job_a, dg, "semisep", rebuild_nodesets=True, panels=True)
        a.launch()
    with torch.cuda.stream(s2):
        b = PreparedJob(job_b, dg, "semisep", rebuild_nodesets=True, panels=True)
        b.launch()
    s2.synchronize()
    got_b = b.out.cpu().numpy()
    torch.cuda.synchronize()
    got_a = a.out.cpu().numpy()
    for job, got in ((job_a, got_a), (job_b, got_b)):
        want = PreparedJob(job, dg, "semisep", rebuild_nodesets=True, panels=True)
        want.launch()
        torch.cuda.synchronize()
        assert np.all(np.isfinite(got)) and np.array_equal(got, want.out.cpu().numpy())
