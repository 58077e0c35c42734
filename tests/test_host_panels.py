"""Host logic of the panels, checked on the CPU: a prepared job's descriptors (folds, potentials, psi folds, panels)
are emulated with NumPy on random operators and waves, and every result row must equal the bilinear form of its
pair, a^T K_L b with a = T (u_f chi_i) or T (chi_f chi_i) and b = B (chi_f u_i) or w u_f u_i, formed pair by pair.
Covered: parity-filtered and complete pair lists, one and several transitions, pairs whose integration limit
differs (node sets of their own, left to the per-pair forms), repeated pairs (no panels), a combination missing
from an otherwise complete block, and the rule that keeps unshared batches on the per-pair forms."""
import ctypes

import numpy as np
import pytest
import torch

import bench
from dwba_b200 import _lib
from oracle.folded import semiseparable_eval

N, L_MAX = 150, 9  # ten multipoles: two psi multi-folds per block


def _view(ptr, n, t=ctypes.c_double):
    return np.ctypeslib.as_array((t * int(n)).from_address(int(ptr)))


def _wave(g, l, k, rng, match=-1):
    w = bench._Wave(l, k, 0.0, rng.normal(size=N))
    w.idx_match = match
    return w


def _job(kind, panels=True):
    from dwba_b200.dwba_matrix_elements import GPUCache, _make_job  # noqa: F401
    from dwba_b200.engine import DeviceGrid, PreparedJob
    from dwba_b200.plan import GridInfo
    rng = np.random.default_rng(4)
    g = bench.make_grid(N, 0.05, 300.0)  # every l at its matching radius (no limit pushed out)
    n_t = 3 if kind == "transitions" else 1
    u0 = rng.normal(size=N) * np.exp(-g.r)
    b_i = [bench._Bound(0, u0)] * n_t
    b_f = [bench._Bound(1, rng.normal(size=N) * np.exp(-g.r)) for _ in range(n_t)]
    wi = [_wave(g, l, 2.0, rng, 120) for l in range(8)]
    wf = [_wave(g, l, 1.5, rng, 120) for l in range(8)]
    pairs = [(a, b) for a in wi for b in wf if kind == "complete" or (a.l + b.l) % 2 == 0]
    if kind == "limits":  # two waves with another matching radius
        wi[6].idx_match = wf[7].idx_match = 90
    if kind == "hole":
        del pairs[5]
    if kind == "repeated":
        pairs.append(pairs[3])
    if kind == "unshared":
        pairs = [(_wave(g, 0, 2.0, rng), _wave(g, 0, 1.5, rng)) for _ in range(20)]

    class Cache:
        info = GridInfo(g.r, g.w_simpson, g.w_trapz)
        dg = DeviceGrid(info, torch.device("cpu"))
    z = np.zeros(N)
    job = _make_job(g, z, z, b_i, b_f, pairs, L_MAX, z, {}, Cache)
    pj = PreparedJob(job, Cache.dg, "semisep", rebuild_nodesets=True, panels=panels)
    for q, pl in enumerate(pj.plans.nodesets):  # random operators, T symmetric
        n1 = pl.key.n1
        ta = _view(pj.nodesets.ta_all[q], 3 * n1).reshape(n1, 3)
        ta[:] = rng.normal(size=(n1, 3))
        ta[1:, 0] = ta[:-1, 2]
        _view(pj.nodesets.bx_all[q], 5 * N)[:] = rng.normal(size=5 * N)
    return pj, g


def _band(op, h, f, n_out, n_src):
    out = np.zeros(n_out)
    for d in range(-h, h + 1):
        k = np.arange(n_out) + d
        ok = (k >= 0) & (k < n_src)
        out[ok] += op.reshape(-1, 2 * h + 1)[:n_out][ok, d + h] * f[k[ok]]
    return out


def _multi(m):
    g = _view(m["g"], m["n_src"])
    op = _view(m["op"], (2 * m["half_band"] + 1) * m["n_out"])
    for q in range(m["n_f"]):
        r = _band(op, int(m["half_band"]), _view(m["f"][q], m["n_src"]) * g, int(m["n_out"]), int(m["n_src"]))
        _view(m["out"][q], m["n_clear"])[:] = np.concatenate([r, np.zeros(m["n_clear"] - m["n_out"])])


def _emulate(pj, r):
    nl = pj.nl
    for f in pj.folds_host:
        assert f["half_band"] == 0
        n = int(f["n_out"])
        _view(f["out"], n)[:] = _view(f["op"], n) * _view(f["f"], n) * _view(f["g"], n)
    for m in pj.multi_host:
        _multi(m)
    fl = pj.form_launch
    rl, rg = np.minimum(r[:, None], r[None, :]), np.maximum(r[:, None], r[None, :])
    K = [(1 / rg) * np.minimum(rl / rg, 1 - 1e-12) ** L for L in range(nl)]
    for p in fl.pots_host:
        dst = _view(p["phi"], nl * p["stride"]).reshape(nl, p["stride"])
        b = _view(p["b"], p["n_cols"])
        for L in range(nl):
            dst[L, :p["n_rows"]] = K[L][:p["n_rows"], :p["n_cols"]] @ b
    for d in fl.dots_host:
        if d["n_rows"]:
            phi = _view(d["phi"], nl * d["stride"]).reshape(nl, d["stride"])
            _view(d["out"], nl)[:] = phi[:, :d["n_rows"]] @ _view(d["a"], d["n_rows"])
    if fl.n_ss:
        for f, row in zip(fl.ss_forms_host, fl.ss_rows_d.numpy()):
            a, b = np.zeros(len(r)), np.zeros(len(r))
            a[:f["n_rows"]], b[:f["n_cols"]] = _view(f["a"], f["n_rows"]), _view(f["b"], f["n_cols"])
            fl.out.numpy()[row] = semiseparable_eval(r, a, b, nl - 1)
    if fl.panels is None:
        return 0
    for m in fl.panels.psi_host:
        _multi(m)
    n = 0
    ctas = _view(fl.panels.ctas_ptr, 4 * fl.panels.n_cta, ctypes.c_int32).reshape(-1, 4)
    for q, P in enumerate(fl.panels.panels_host):
        cols = _view(P["cols"], 2 * P["F"], ctypes.c_uint64).reshape(-1, 2)
        rows, outs = _view(P["rows"], P["M"], ctypes.c_uint64), _view(P["out"], P["M"] * P["F"], ctypes.c_uint64)
        mine = ctas[ctas[:, 0] == q]
        assert len(np.unique(mine, axis=0)) == len(mine) > 0
        assert (mine[:, 1].max() + 1) * 64 >= P["M"] and (mine[:, 2].max() + 1) * 64 >= P["F"] * nl
        for m in range(P["M"]):
            for f in range(P["F"]):
                o = outs[m * P["F"] + f]
                if not o:
                    continue
                phi = _view(cols[f, 0], nl * P["stride"]).reshape(nl, P["stride"])[:, :P["n"]]
                x = _view(rows[m], P["n"]) * (_view(cols[f, 1], P["n"]) if cols[f, 1] else 1.0)
                _view(o, nl)[:] = phi @ x
                n += 1
    return n


@pytest.mark.parametrize("kind,expect", [("parity", "all"), ("complete", "all"), ("transitions", "all"), ("hole", "all"),
                                         ("limits", "some"), ("repeated", "none"), ("unshared", "none")])
def test_panels_evaluate_every_form(kind, expect):
    pj, g = _job(kind)
    r = g.r
    pj.out.fill_(np.nan)
    pj.ops.fill_(np.nan)
    n = _emulate(pj, r)
    assert (n == pj.n_forms) if expect == "all" else (0 < n < pj.n_forms) if expect == "some" else n == 0
    out, job = pj.out.numpy(), pj.job
    for t, tr in enumerate(job.transitions):
        for p, (ci, cf) in enumerate(job.pairs):
            q, n1 = int(pj.plans.ns_index[t, p]), int(pj.plans.n1[t, p])
            ta, bx = _view(pj.nodesets.ta_all[q], 3 * n1), _view(pj.nodesets.bx_all[q], 5 * N)
            nb = min(N, n1 + 2)
            for e, a, b in ((0, _band(ta, 1, cf.chi_of_r * ci.chi_of_r, n1, n1), g.w_simpson * tr.u_f * tr.u_i),
                            (1, _band(ta, 1, tr.u_f * ci.chi_of_r, n1, n1), _band(bx, 2, cf.chi_of_r * tr.u_i, nb, N))):
                x, y = np.zeros(N), np.zeros(N)
                x[:n1], y[:len(b)] = a, b
                # |Tx| can cancel where T|x| does not: the scale is that of the operator's terms
                ax = _band(np.abs(ta), 1, np.abs(cf.chi_of_r if e == 0 else tr.u_f) * np.abs(ci.chi_of_r), n1, n1)
                sx = np.zeros(N)
                sx[:n1] = ax
                scale = semiseparable_eval(r, sx, np.abs(y), L_MAX)
                got = out[2 * (t * pj.P + p) + e]
                assert np.all(np.abs(got - semiseparable_eval(r, x, y, L_MAX)) <= 1e-12 * scale), (t, p, e)


def test_backward_jobs_keep_one_operand_per_form():
    pj, _ = _job("parity", panels=False)
    assert pj.form_launch.panels is None and np.all(pj.forms_host["a"] != 0)
