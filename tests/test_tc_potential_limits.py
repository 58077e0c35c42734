"""Split-BF16 engine: potentials past the 32-bit stride of a panel leave the exchange forms to one column per form."""
import pytest
import torch

import bench
import numpy as np
from dwba_b200 import _lib
from dwba_b200 import engine as E


def _job():
    from dwba_b200.dwba_matrix_elements import _make_job
    from dwba_b200.plan import GridInfo
    n = 200
    g = bench.make_grid(n, 0.05, 300.0)

    class Cache:
        info = GridInfo(g.r, g.w_simpson, g.w_trapz)
        dg = E.DeviceGrid(info, torch.device("cpu"))
    rng = np.random.default_rng(1)
    w = [[bench._Wave(l, k, 0.0, rng.normal(size=n)) for l in range(6)] for k in (1.5, 1.0)]
    z = np.zeros(n)
    job = _make_job(g, z, z, [bench._Bound(0, np.exp(-g.r))], [bench._Bound(1, g.r * np.exp(-g.r))],
                    [(a, b) for a in w[0] for b in w[1]], 4, z, {}, Cache)
    return job, Cache.dg


@pytest.mark.parametrize("terms,engine", [(2, "tc_bf16x3"), (3, "tc_bf16x6")])
def test_sizes_past_the_panels_stride_take_forms(monkeypatch, terms, engine):
    job, dg = _job()
    assert E.PreparedJob(job, dg, engine, panels=True).tc_panels
    lib = _lib.load()
    real, asked = lib.dwba_tc_potentials_layout, []

    def large(n, N, L, t, row, lrow):  # 2^31 / N operands or more
        ws = real(n, N, L, t, row, lrow)
        asked.append((n, N, L, t))
        lrow._obj.value = 0x80000000
        return ws
    monkeypatch.setattr(lib, "dwba_tc_potentials_layout", large)
    pj = E.PreparedJob(job, dg, engine, panels=True)
    assert asked == [(6, 200, 4, terms)] and not pj.tc_panels
    ex = pj.forms_host[1::2]  # every exchange form has its operands, shared or not
    assert np.all(ex["a"] != 0) and np.all(ex["b"] != 0) and len(np.unique(ex["b"])) == 6
    assert pj.form_launch.panels.n_exchange == 0 and pj.form_launch.panels.n_direct > 0
    assert pj.tc_ws.numel() >= lib.dwba_tc_workspace_bytes(36, 200, 4, terms)
