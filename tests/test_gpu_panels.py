"""dwba_panel_forms at the edges of its tiles (64 rows x 64 columns, steps of 16 grid points, chunks of 256 and more),
dwba_multipole_potentials past its one-tile length (16384 points), and the panels of a job against its per-pair forms."""
import numpy as np
import pytest

import bench

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


@pytest.mark.parametrize("M,F,L_max,n,mul", [
    (1, 1, 0, 1, False), (8, 3, 4, 15, True), (9, 2, 6, 17, False), (63, 64, 0, 255, True), (64, 16, 3, 256, False),
    (65, 9, 6, 257, True), (21, 21, 6, 4097, False), (130, 5, 10, 1000, True), (3, 33, 1, 4113, True), (2, 2, 40, 300, False)])
def test_panels_at_tile_edges(M, F, L_max, n, mul):
    import ctypes
    import torch
    from dwba_b200 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(M * F + n)
    nl, stride = L_max + 1, n + 3
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda")  # noqa: E731
    a, phi, mu = rng.normal(size=(M, n)), rng.normal(size=(F, nl, stride)), rng.normal(size=(F, n))
    ad, pd, md = t(a), t(phi), t(mu)
    out = torch.full((M * F + 1, nl), np.nan, dtype=torch.float64, device="cuda")
    hole = (M * F) // 2 if M * F > 2 else -1
    rows = ad.data_ptr() + 8 * n * np.arange(M, dtype=np.uint64)
    cols = np.zeros(F, dtype=_lib.PANEL_COL_DTYPE)
    cols["phi"] = pd.data_ptr() + 8 * nl * stride * np.arange(F, dtype=np.uint64)
    if mul:
        cols["mul"] = md.data_ptr() + 8 * n * np.arange(F, dtype=np.uint64)
    outs = out.data_ptr() + 8 * nl * np.arange(M * F, dtype=np.uint64)
    if hole >= 0:
        outs[hole] = 0
    rd, cd, od = (t(x.view(np.uint8)) for x in (rows, cols, outs))
    P = np.zeros(1, dtype=_lib.PANEL_DTYPE)
    P["rows"], P["cols"], P["out"], P["M"], P["F"], P["n"], P["stride"] = rd.data_ptr(), cd.data_ptr(), od.data_ptr(), M, F, n, stride
    part = ctypes.c_int64(0)
    n_cta = lib.dwba_panel_plan(P.ctypes.data, 1, L_max, None, ctypes.byref(part))
    ctas = np.zeros(n_cta, dtype=_lib.PANEL_CTA_DTYPE)
    assert lib.dwba_panel_plan(P.ctypes.data, 1, L_max, ctas.ctypes.data, ctypes.byref(part)) == n_cta
    Pd, Cd = t(P.view(np.uint8)), t(ctas.view(np.uint8))
    w = torch.full((part.value,), np.nan, dtype=torch.float64, device="cuda")
    _lib.check(lib.dwba_panel_forms(Pd.data_ptr(), 1, Cd.data_ptr(), n_cta, 0, L_max, w.data_ptr(),
                                    torch.cuda.current_stream().cuda_stream), "panels")
    got = out.cpu().numpy()
    assert np.all(np.isnan(got[M * F]))
    b = phi[:, :, :n] * (mu[:, None, :] if mul else 1.0)
    want, scale = np.einsum("mx,flx->mfl", a, b).reshape(-1, nl), np.einsum("mx,flx->mfl", abs(a), abs(b)).reshape(-1, nl)
    for q in range(M * F):
        if q == hole:
            assert np.all(np.isnan(got[q]))
        else:  # n products and sums, each rounded once
            assert np.all(np.abs(got[q] - want[q]) <= 4 * EPS * np.sqrt(n) * scale[q]), q


@pytest.mark.parametrize("n_rows,n_cols,L_max", [(16384, 16384, 1), (16385, 16390, 2), (40001, 33000, 0), (700, 17000, 4)])
def test_potentials_past_one_tile(n_rows, n_cols, L_max):
    import torch
    from dwba_b200 import _lib
    from dwba_b200.plan import diag_scale
    rng = np.random.default_rng(n_rows)
    n, nl = max(n_rows, n_cols), L_max + 1
    r = np.geomspace(1e-3, 60.0, n)
    b = rng.normal(size=n_cols) * np.exp(-r[:n_cols] / 10)
    rd, bd = torch.as_tensor(r, device="cuda"), torch.as_tensor(b, device="cuda")
    phi = torch.full((nl, n_rows), np.nan, dtype=torch.float64, device="cuda")
    rec = np.zeros(1, dtype=_lib.POTENTIAL_DTYPE)
    rec[0] = (rd.data_ptr(), bd.data_ptr(), phi.data_ptr(), n_rows, n_cols, n_rows, 0)
    recd = torch.from_numpy(rec.view(np.uint8).copy()).cuda()
    ds = diag_scale(L_max)
    _lib.check(_lib.load().dwba_multipole_potentials(recd.data_ptr(), 1, L_max, ds.ctypes.data, float(r[0]), float(r[-1]),
                                                     torch.cuda.current_stream().cuda_stream), "potentials")
    got = phi.cpu().numpy()
    x, y = r.astype(np.longdouble), np.zeros(n, dtype=np.longdouble)
    y[:n_cols] = b
    for L in range(nl):
        lo, hi = x ** L, x ** -(L + 1)

        def f(z):
            suf = np.cumsum((z * hi)[::-1])[::-1] - z * hi
            return (hi * (np.cumsum(z * lo) - z * lo) + lo * suf + (1 - 1e-12) ** L * z / x)[:n_rows]
        assert np.all(np.abs(got[L] - f(y)) <= 1e-14 * f(np.abs(y)))


def test_panel_jobs_match_per_pair_forms():
    """A Coulomb energy point with tails and an unfiltered list with a missing pair: panels against the per-pair
    forms of the same job. Both sum the same products in another order: 1e-14 of the sum of their magnitudes."""
    from dwba_b200.dwba_matrix_elements import GPUCache, _make_job
    from dwba_b200.engine import PreparedJob
    for pt in bench.make_ragged_points(64, l_max_wave=13, select=[40]):
        pairs = pt["pairs"][:-1] + [(pt["pairs"][3][0], pt["pairs"][-1][1])]  # a hole, and one of another parity
        cache = GPUCache.from_grid(pt["grid"])
        job = _make_job(pt["grid"], pt["V_core_array"], pt["U_i_array"], pt["bound_i"], pt["bound_f"], pairs, 8,
                        pt["U_f_array"], {}, cache)
        res = []
        for panels in (True, False):
            pj = PreparedJob(job, cache.dg, "semisep", panels=panels)
            pj.launch()
            res.append(pj.collect())
            if panels:
                n = len(pj.direct_plan.panels.direct.fo) + len(pj.direct_plan.panels.exchange.fo)
                assert n > pj.n_forms // 2
        import torch
        ab = pj.ops.abs()
        f = pj.forms_host.copy()
        for k in ("a", "b"):
            f[k] = f[k] - pj.ops.data_ptr() + ab.data_ptr()
        from dwba_b200 import _lib
        fd = torch.from_numpy(f.view(np.uint8).copy()).cuda()
        S = torch.empty((len(f), 9), dtype=torch.float64, device="cuda")
        _lib.check(_lib.load().dwba_bilinear_semisep_fp64(fd.data_ptr(), len(f), 8, pj.ds.ctypes.data, float(job.grid.r[0]),
                                                          float(job.grid.r[-1]), S.data_ptr(),
                                                          torch.cuda.current_stream().cuda_stream), "scale")
        S = S.cpu().numpy().reshape(len(pairs), 2, 9)
        for e in (0, 1):
            assert np.all(np.abs(res[0][e][0] - res[1][e][0]) <= 1e-14 * S[:, e] + 1e-12 * np.abs(res[1][e][0]))


@pytest.mark.parametrize("n_rows,n_cols,n,L_max", [(1, 1, 1, 0), (31, 700, 8, 4), (32, 32, 9, 5), (33, 1, 3, 2), (700, 257, 17, 11)])
def test_dense_potentials_at_tile_edges(n_rows, n_cols, n, L_max):
    """Runs of eight, row tiles of 32, column tiles of 128 and passes of five multipoles, padded runs; reference: K_L in
    long double, 1e-14 of the sum of the terms' magnitudes."""
    import torch
    from dwba_b200 import _lib
    from dwba_b200.engine import _dense_runs
    from dwba_b200.plan import diag_scale
    rng = np.random.default_rng(n_rows + n)
    nl, N = L_max + 1, max(n_rows, n_cols)
    r = np.geomspace(1e-3, 60.0, max(N, 2))
    b = rng.normal(size=(n, n_cols))
    rd, bd = torch.as_tensor(r, device="cuda"), torch.as_tensor(b, device="cuda")
    phi = torch.full((n, nl, n_rows), np.nan, dtype=torch.float64, device="cuda")
    p = np.zeros(n, dtype=_lib.POTENTIAL_DTYPE)
    p["r"], p["n_rows"], p["n_cols"], p["stride"] = rd.data_ptr(), n_rows, n_cols, n_rows
    p["b"] = bd.data_ptr() + 8 * n_cols * np.arange(n, dtype=np.uint64)
    p["phi"] = phi.data_ptr() + 8 * nl * n_rows * np.arange(n, dtype=np.uint64)
    p = _dense_runs(p)
    pd = torch.from_numpy(p.view(np.uint8).copy()).cuda()
    ds = diag_scale(L_max)
    _lib.check(_lib.load().dwba_dense_potentials(pd.data_ptr(), len(p), n_rows, L_max, ds.ctypes.data,
                                                 torch.cuda.current_stream().cuda_stream), "dense potentials")
    x = r.astype(np.longdouble)
    lo, hi = np.minimum(x[:n_rows, None], x[None, :n_cols]), np.maximum(x[:n_rows, None], x[None, :n_cols])
    for L in range(nl):
        K = np.minimum(lo / hi, np.longdouble(1) - np.longdouble(1e-12)) ** L / hi
        d = np.abs(phi[:, L].cpu().numpy() - (b @ K.T).astype(float))
        assert np.all(d <= 1e-14 * (np.abs(b) @ K.T).astype(float)), L


@pytest.mark.parametrize("engine,n_l", [("dense", 12), ("tc_bf16x3", 12), ("tc_bf16x6", 12), ("tc_bf16x3", 70), ("tc_bf16x3", 130)])
def test_engine_panels_match_per_pair_forms(engine, n_l):
    """The plain FP64 and the split-BF16 engines with panels against their per-form launches: the same products (K_L
    elements, or K_L b from the same tensor-core tiles) summed in another order. n_l waves of one momentum: 12, 70
    and 130 distinct operands (the three tile widths of the split product)."""
    import torch
    from dwba_b200.dwba_matrix_elements import GPUCache, _make_job
    from dwba_b200.engine import PreparedJob
    N, L = (1500, 6) if n_l == 12 else (700, 2)
    rng = np.random.default_rng(n_l)
    g = bench.make_grid(N, 1e-4, 80.0)
    r = g.r

    def wave(l, k):
        return bench._Wave(l % 9, k, 0.0, np.sin(k * r + rng.uniform(0, 3)) * (1 - np.exp(-(r * k) ** (1 + l % 9))))
    wi, wf = [wave(l, 1.9) for l in range(5 if n_l > 12 else 12)], [wave(l, 1.6) for l in range(n_l)]
    pairs = [(a, b) for a in wi for b in wf]
    u = [bench._Bound(0, r * np.exp(-r)), bench._Bound(1, r * r * np.exp(-0.5 * r))]
    z = np.zeros(N)
    cache = GPUCache.from_grid(g)
    job = _make_job(g, z, z, u[0], u[1], pairs, L, z, {}, cache)
    jobs = [PreparedJob(job, cache.dg, engine, panels=p) for p in (True, False)]
    assert jobs[0].dense_panels or jobs[0].tc_panels
    res = []
    for pj in jobs:
        pj.launch()
        res.append(pj.collect())
    pj = PreparedJob(job, cache.dg, "semisep", panels=False)
    pj.launch()
    ab, f = pj.ops.abs(), pj.forms_host.copy()
    for k in ("a", "b"):
        f[k] = f[k] - pj.ops.data_ptr() + ab.data_ptr()
    from dwba_b200 import _lib
    fd = torch.from_numpy(f.view(np.uint8).copy()).cuda()
    S = torch.empty((len(f), L + 1), dtype=torch.float64, device="cuda")
    _lib.check(_lib.load().dwba_bilinear_semisep_fp64(fd.data_ptr(), len(f), L, pj.ds.ctypes.data, float(r[0]), float(r[-1]),
                                                      S.data_ptr(), torch.cuda.current_stream().cuda_stream), "scale")
    S = S.cpu().numpy().reshape(len(pairs), 2, L + 1)
    for e in (0, 1):
        assert np.all(np.isfinite(res[0][e]))
        assert np.all(np.abs(res[0][e][0] - res[1][e][0]) <= 1e-14 * S[:, e] + 1e-12 * np.abs(res[1][e][0])), e
