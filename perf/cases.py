"""Workloads of the radial matrix-element engine, as a user's program calls them.

``listed()`` gives the cases, ``draw(rng)`` another one of the same ranges, ``prepare(case, seed)`` the inputs and
handles a program has in hand before the call, ``run(state)`` one pass through the public entry points with its whole
outputs, ``work(case)`` the bytes and operations the pass cannot do without, and ``exact(case, seed)`` the same outputs
from plain torch in 64 bits (None where that would take too long).

The waves are the synthetic stand-ins of the benchmark: sin(k r - l pi/2 + d) with an (r/r0)^(l+1) onset, on exponential
grids from 1e-5 a0; Coulomb-like ones add eta log(2 k r) with eta = -1/k and a matching radius inside the grid, so that
the outer tails take part.
"""
import math
from types import SimpleNamespace

import numpy as np
import torch

HARTREE = 27.211386245988
DEV = "cuda"


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the reference driver's loop: one call per (l_i, l_f) pair, the grid's cache kept over one energy (H 1s->2p, 50 eV
        # sizes), with the default engine: the smallest call, where latency and launches count
        dict(name="pair_call", kind="pair", n=3000, L=4, engine="default"),
        # all 128 pairs of that energy point in one batched call from host arrays; a new energy has new node sets
        dict(name="point_call", kind="point_call", n=3000, l_max=15, L=4, engine="semisep"),
        # the same energy point through the plain FP64 engine (the default one), its handle kept
        dict(name="point_dense", kind="point", n=3000, l_max=15, L=4, engine="dense"),
        # one energy point through the split-BF16 tensor-core engine with its accuracy guard
        dict(name="point_split_bf16", kind="point", n=6000, l_max=25, L=6, engine="tc_bf16x3"),
        # excitation sweep: He+-like 1s->2s and 1s->2p, 45..1000 eV, every energy on its own grid (2000..15000 points,
        # most sizes odd), Coulomb-like waves with outer tails, all energies in shared launches
        dict(name="sweep", kind="sweep", energies=8, n_lo=2000, n_hi=15000, l_max=40, L=6, engine="semisep"),
        # a short sweep of few partial waves: few forms per launch
        dict(name="sweep_small", kind="sweep", energies=3, n_lo=1201, n_hi=4003, l_max=9, L=5, engine="semisep"),
        # one ejected energy of an ionization SDCS: a transition per ejected partial wave, all pairs of matching parity
        dict(name="ionization", kind="ionization", n=8000, l_max=30, L=10, engine="semisep"),
        # the benchmark's batch, its handle kept: every pair at energies of its own, 4 transitions
        dict(name="batch_step", kind="batch", n=15000, pairs=2048, transitions=4, L=8, engine="semisep"),
        # a quarter of that batch through the batched call, from pinned host arrays to result arrays
        dict(name="batch_call", kind="batch_call", n=15000, pairs=512, transitions=4, L=8, engine="semisep"),
        # differentiation: integrals and all input gradients of one transition (Na-like 3s->3p sizes)
        dict(name="gradient", kind="gradient", n=6000, l_max=25, L=4, engine="semisep"),
        # the backward of the bilinear forms alone, through the C interface, at those sizes
        dict(name="forms_backward", kind="forms_backward", n=6000, forms=676, L=4),
        # DCS and TCS of one energy of the sweep from its integrals (s->p, 181 angles)
        dict(name="cross_sections", kind="cross_sections", l_max=40, L=6, angles=181),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair", "point_call", "point", "sweep", "ionization", "batch", "batch_call", "gradient",
                       "forms_backward", "cross_sections"])
    if kind == "pair":
        return dict(kind=kind, n=_log_int(rng, 1000, 15000), L=rng.randint(0, 10),
                    engine=rng.choice(["default", "semisep"]))
    if kind == "point_call":
        return dict(kind=kind, n=_log_int(rng, 1500, 8000), l_max=rng.randint(3, 20), L=rng.randint(2, 8),
                    engine="semisep")
    if kind == "point":
        eng = rng.choice(["dense", "semisep", "tc_bf16x3"])
        hi = 4000 if eng == "dense" else 8000
        return dict(kind=kind, n=_log_int(rng, 1500, hi), l_max=rng.randint(5, 20), L=rng.randint(2, 8), engine=eng)
    if kind == "sweep":
        return dict(kind=kind, energies=rng.randint(2, 6), n_lo=_log_int(rng, 1000, 3000), n_hi=_log_int(rng, 3001, 12000),
                    l_max=rng.randint(5, 35), L=rng.randint(2, 9), engine="semisep")
    if kind == "ionization":
        return dict(kind=kind, n=_log_int(rng, 2000, 7000), l_max=rng.randint(6, 26), L=rng.randint(4, 10), engine="semisep")
    if kind in ("batch", "batch_call"):
        return dict(kind=kind, n=_log_int(rng, 3000, 14000), pairs=_log_int(rng, 70, 450), transitions=rng.randint(1, 5),
                    L=rng.randint(3, 10), engine="semisep")
    if kind == "gradient":
        return dict(kind=kind, n=_log_int(rng, 1500, 6000), l_max=rng.randint(5, 20), L=rng.randint(2, 6), engine="semisep")
    if kind == "forms_backward":
        return dict(kind=kind, n=_log_int(rng, 1500, 8000), forms=_log_int(rng, 40, 600), L=rng.randint(2, 10))
    return dict(kind=kind, l_max=rng.randint(8, 36), L=rng.randint(2, 8), angles=rng.choice([91, 181, 361]))


# ------------------------------------------------------------------------------------------------ inputs
def _grid(n, r_max):
    """Exponential grid with trapezoid and non-uniform Simpson weights."""
    r = 1e-5 * ((r_max / 1e-5) ** np.linspace(0.0, 1.0, n))
    dr = np.diff(r)
    wt = np.zeros(n)
    wt[0], wt[-1] = 0.5 * dr[0], 0.5 * dr[-1]
    wt[1:-1] = 0.5 * (r[2:] - r[:-2])
    ws = np.zeros(n)
    h1, h2 = dr[0:n - 2:2], dr[1:n - 1:2]
    c = (h1 + h2) / 6.0
    ws[0:n - 2:2] += c * (2.0 - h2 / h1)
    ws[1:n - 1:2] += c * ((h1 + h2) ** 2 / (h1 * h2))
    ws[2:n:2] += c * (2.0 - h1 / h2)
    if n % 2 == 0:
        ws[-2] += 0.5 * dr[-1]
        ws[-1] += 0.5 * dr[-1]
    return SimpleNamespace(r=r, dr=np.append(dr, dr[-1]), w_trapz=wt, w_simpson=ws)


def _waves(g, l, k, d, eta=None, sigma=None, pinned=False):
    """chi of many waves as the rows of one host matrix (formed on the GPU)."""
    t = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=DEV)[:, None]  # noqa: E731
    r = torch.as_tensor(g.r, device=DEV)[None, :]
    rows = len(l)
    out = torch.empty((rows, len(g.r)), dtype=torch.float64, pin_memory=pinned)
    for a in range(0, rows, 512):
        s = slice(a, a + 512)
        kk, ll = t(k[s]), t(l[s])
        ph = kk * r - 0.5 * math.pi * ll + t(d[s])
        if eta is not None:
            ph += t(eta[s]) * torch.log(2 * kk * r) + t(sigma[s])
        out[s] = torch.sin(ph) * (1.0 - torch.exp(-(r * kk / (ll + 1.0)) ** (ll + 1.0)))
    return out.numpy()


def _wave(l, k, d, chi, eta=0.0, sigma=0.0, match=-1):
    return SimpleNamespace(l=int(l), k_au=float(k), phase_shift=float(d), chi_of_r=chi, idx_match=int(match),
                           eta=float(eta), sigma_l=float(sigma))


def _ejected(w):
    """A continuum final state: carries chi_of_r, and u_of_r as the reference's does."""
    w.u_of_r, w.energy_au = w.chi_of_r, 0.5 * w.k_au ** 2
    return w


def _bound(l, u, g):
    return SimpleNamespace(l=l, energy_au=-0.5, n_index=1, u_of_r=u / np.sqrt(np.sum(g.w_trapz * u * u)))


def _point_inputs(case, seed):
    """One energy point: neutral waves of two momenta, an s->p transition, U_i different from V_core, so that the L=0
    corrections are live; all (l_i, l_f) of odd parity."""
    rng = np.random.default_rng(seed)
    g = _grid(case["n"], 200.0)
    r, lm = g.r, case.get("l_max", 3)
    V = -(1.0 + np.exp(-2.0 * r)) / r
    U = V + rng.uniform(0.2, 0.4) * np.exp(-r)
    bi = _bound(0, r * np.exp(-rng.uniform(0.9, 1.1) * r), g)
    bf = _bound(1, r * r * np.exp(-rng.uniform(0.45, 0.55) * r), g)
    k_i = rng.uniform(1.85, 2.0)
    k_f = math.sqrt(k_i ** 2 - 0.75)
    l = np.arange(lm + 1)
    d = rng.uniform(0.0, math.pi, (2, lm + 1))
    wi = [_wave(*a) for a in zip(l, [k_i] * (lm + 1), d[0], _waves(g, l, [k_i] * (lm + 1), d[0]))]
    wf = [_wave(*a) for a in zip(l, [k_f] * (lm + 1), d[1], _waves(g, l, [k_f] * (lm + 1), d[1]))]
    pairs = [(wi[a], wf[b]) for a in range(lm + 1) for b in range(lm + 1) if (a + b) % 2 == 1]
    if case["kind"] == "pair":
        pairs = [pairs[int(rng.integers(len(pairs)))]]
    return SimpleNamespace(g=g, V=V, U=U, U_f=U, bi=[bi], bf=[bf], pairs=pairs, rng=rng)


def _batch_inputs(case, seed):
    """Pairs at energies of their own (k in 0.5..8, l in 0..63), bound products r^a e^(-b r) times a quadratic."""
    rng = np.random.default_rng(seed)
    g = _grid(case["n"], 400.0)
    P = case["pairs"]
    l, k, d = rng.integers(0, 64, 2 * P), rng.uniform(0.5, 8.0, 2 * P), rng.uniform(0.0, math.pi, 2 * P)
    chi = _waves(g, l, k, d, pinned=True)
    w = [_wave(*a) for a in zip(l, k, d, chi)]
    u = []
    for _ in range(2 * case["transitions"]):
        c = rng.uniform(-1, 1, 3)
        u.append(g.r ** int(rng.integers(1, 3)) * np.exp(-rng.uniform(0.5, 2.0) * g.r) * (c[0] + c[1] * g.r + c[2] * g.r ** 2))
    z = np.zeros(case["n"])
    return SimpleNamespace(g=g, V=z, U=z, U_f=z, bi=[_bound(0, x, g) for x in u[0::2]], bf=[_bound(1, x, g) for x in u[1::2]],
                           pairs=[(w[2 * p], w[2 * p + 1]) for p in range(P)], chi=chi)


def _coulomb(g, l, k, rng, match):
    eta = np.full(len(l), -1.0 / k)
    d, sig = rng.uniform(0, math.pi, len(l)), rng.uniform(-1, 1, len(l))
    kk = np.full(len(l), k)
    return [_wave(a, k, b, c, e, s, match) for a, b, c, e, s in zip(l, d, _waves(g, l, kk, d, eta, sig), eta, sig)]


def _sweep_points(case, seed):
    rng = np.random.default_rng(seed)
    lm, ne = case["l_max"], case["energies"]
    l, pts = np.arange(lm + 1), []
    for e, E in enumerate(np.geomspace(45.0, 1000.0, ne)):
        n = int(round(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** (e / max(1, ne - 1))))
        g = _grid(n, 200.0)
        r = g.r
        V = -2.0 / r
        match = int(np.searchsorted(r, 120.0))
        u1s = r * np.exp(-2.0 * r)
        for par, u2 in ((0, r * (1.0 - r) * np.exp(-r)), (1, r * r * np.exp(-r))):
            k_i, k_f = math.sqrt(2 * E / HARTREE), math.sqrt(2 * E / HARTREE - 3.0)
            wi, wf = _coulomb(g, l, k_i, rng, match), _coulomb(g, l, k_f, rng, match)
            pairs = [(wi[a], wf[b]) for a in range(lm + 1) for b in range(lm + 1) if (a + b) % 2 == par]
            pts.append(SimpleNamespace(g=g, V=V, U=V, U_f=V, bi=[_bound(0, u1s, g)], bf=[_bound(par, u2, g)], pairs=pairs))
    return pts


def _ionization_points(case, seed):
    rng = np.random.default_rng(seed)
    g = _grid(case["n"], 200.0)
    r, lm = g.r, case["l_max"]
    V = -1.0 / r
    b = _bound(0, r * np.exp(-r), g)
    match = int(np.searchsorted(r, 120.0))
    E_ej = rng.uniform(0.5, 99.0)
    l = np.arange(lm + 1)
    inc = _coulomb(g, l, math.sqrt(2 * 200.0 / HARTREE), rng, match)
    sc = _coulomb(g, l, math.sqrt(2 * (186.394307 - E_ej) / HARTREE), rng, match)
    ej = [_ejected(w) for w in _coulomb(g, l, math.sqrt(2 * E_ej / HARTREE), rng, match)]
    pts = []
    for par in (0, 1):
        pairs = [(inc[a], sc[c]) for a in range(lm + 1) for c in range(lm + 1) if (a + c) % 2 == par]
        fin = ej[par::2]
        pts.append(SimpleNamespace(g=g, V=V, U=V, U_f=V, bi=[b] * len(fin), bf=fin, pairs=pairs))
    return pts


def _prepared(p, L, engine, cache=None):
    """The kept handle of one point: its functions and descriptors on the device, node sets rebuilt on every launch."""
    from dwba_b200.dwba_matrix_elements import GPUCache
    from dwba_b200.engine import Job, PreparedJob, Transition
    from dwba_b200.plan import is_excitation
    cache = cache or GPUCache.from_grid(p.g)
    job = Job(grid=cache.info, V_core=p.V, U_i=p.U, U_f=p.U_f, pairs=p.pairs, L_max=L,
              transitions=[Transition(u_i=a.u_of_r, u_f=b.u_of_r, excitation=is_excitation(b)) for a, b in zip(p.bi, p.bf)])
    return PreparedJob(job, cache.dg, engine, rebuild_nodesets=True)


def _backward_inputs(case, seed):
    rng = np.random.default_rng(seed)
    g = _grid(case["n"], 200.0)
    n, nf, nl = case["n"], case["forms"], case["L"] + 1
    r = torch.as_tensor(g.r, device=DEV)
    t = lambda a: torch.as_tensor(a, device=DEV)  # noqa: E731
    dr = torch.as_tensor(g.w_simpson, device=DEV)
    f = lambda: (torch.sin(t(rng.uniform(0.5, 3, (nf, 1))) * r + t(rng.uniform(0, 3, (nf, 1))))  # noqa: E731
                 * torch.exp(-r * t(rng.uniform(0.05, 1.0, (nf, 1)))) * r * dr)
    a, b = f(), f()
    grad = t(rng.normal(size=(nf, nl)))
    rows = np.where(np.arange(nf) % 2 == 0, n, n - rng.integers(2, n // 4, nf)).astype(np.int32)
    cols = np.where(np.arange(nf) % 2 == 0, n, np.minimum(n, rows + 2)).astype(np.int32)
    return SimpleNamespace(g=g, r=r, a=a, b=b, grad=grad, rows=rows, cols=cols)


def _cross_inputs(case, seed):
    rng = np.random.default_rng(seed)
    lm = case["l_max"]
    ch = [(a, b) for a in range(lm + 1) for b in range(lm + 1) if (a + b) % 2 == 1]
    scale = np.exp(-0.1 * np.array([a + b for a, b in ch]))[:, None]
    I = rng.normal(size=(2, len(ch), case["L"] + 1)) * scale * 0.05
    k_i = rng.uniform(1.9, 8.0)
    return ch, I, k_i, math.sqrt(k_i ** 2 - 3.0)


# ------------------------------------------------------------------------------------------------ the passes
def prepare(case, seed):
    kind, L = case["kind"], case.get("L")
    eng = None if case.get("engine") == "default" else case.get("engine")
    s = SimpleNamespace(kind=kind, L=L, engine=eng)
    if kind in ("pair", "point_call", "batch_call"):
        from dwba_b200.dwba_matrix_elements import GPUCache
        s.p = _batch_inputs(case, seed) if kind == "batch_call" else _point_inputs(case, seed)
        s.cache = GPUCache.from_grid(s.p.g)
    elif kind == "point":
        s.job = _prepared(_point_inputs(case, seed), L, eng)
    elif kind == "batch":
        s.job = _prepared(_batch_inputs(case, seed), L, eng)
    elif kind in ("sweep", "ionization"):
        from dwba_b200.dwba_matrix_elements import GPUCache
        from dwba_b200.engine import MultiPrepared
        pts = _sweep_points(case, seed) if kind == "sweep" else _ionization_points(case, seed)
        caches = {}
        for p in pts:
            caches.setdefault(id(p.g), GPUCache.from_grid(p.g))
        s.job = MultiPrepared([_prepared(p, L, eng, caches[id(p.g)]) for p in pts])
    elif kind == "gradient":
        from dwba_b200.autograd import RadialIntegrals
        p = _point_inputs(case, seed)
        s.model = RadialIntegrals(p.g, p.bi[0], p.bf[0], p.pairs, L, U_f_array=p.U_f, engine=eng)
        s.x, s.c = _gradient_tensors(p, L)
    elif kind == "forms_backward":
        from dwba_b200 import _lib
        from dwba_b200.plan import diag_scale
        b = s.b = _backward_inputs(case, seed)
        s.ga, s.gb = torch.zeros_like(b.a), torch.zeros_like(b.b)
        step = 8 * case["n"] * np.arange(case["forms"], dtype=np.uint64)
        d = np.zeros(case["forms"], dtype=_lib.FORM_GRAD_DTYPE)
        d["r"], d["n_rows"], d["n_cols"] = b.r.data_ptr(), b.rows, b.cols
        for name, x in (("a", b.a), ("b", b.b), ("ga", s.ga), ("gb", s.gb)):
            d[name] = np.uint64(x.data_ptr()) + step
        s.desc, s.ds, s.lib = torch.from_numpy(d.view(np.uint8)).to(DEV), diag_scale(L), _lib.load()
        s.n, s.lo, s.hi = len(d), float(b.g.r[0]), float(b.g.r[-1])
    elif kind == "cross_sections":
        from dwba_b200.coupling import CouplingTables
        ch, I, k_i, k_f = _cross_inputs(case, seed)
        s.tab = CouplingTables(np.linspace(0.0, math.pi, case["angles"]), ch, L, k_i, k_f, 0, 1)
        s.I = torch.as_tensor(I, device=DEV)
        s.tab.cross_sections_gpu(s.I[0], s.I[1])  # its tables go to the device once
    return s


def run(s):
    kind = s.kind
    if kind == "pair":
        from dwba_b200.dwba_matrix_elements import radial_ME_all_L_gpu
        p = s.p
        res = radial_ME_all_L_gpu(p.g, p.V, p.U, p.bi[0], p.bf[0], p.pairs[0][0], p.pairs[0][1], s.L, gpu_cache=s.cache,
                                  U_f_array=p.U_f, engine=s.engine)
        return {"direct": np.array(list(res.I_L_direct.values())), "exchange": np.array(list(res.I_L_exchange.values()))}
    if kind in ("point_call", "batch_call"):
        from dwba_b200.dwba_matrix_elements import radial_ME_all_L_batch
        p = s.p
        d, e = radial_ME_all_L_batch(p.g, p.V, p.U, p.bi, p.bf, p.pairs, s.L, U_f_array=p.U_f, gpu_cache=s.cache,
                                     engine=s.engine, as_arrays=True)
        s.cache.clear()  # one call per energy: the next one has node sets of its own
        return {"direct": d, "exchange": e}
    if kind == "gradient":
        x = {k: v.detach().requires_grad_(True) for k, v in s.x.items()}
        I = s.model(**x)
        (I * s.c).sum().backward()
        return {"I": I.detach(), **{"d_" + k: v.grad for k, v in x.items()}}
    if kind == "forms_backward":
        from dwba_b200 import _lib
        _lib.check(s.lib.dwba_bilinear_semisep_backward_fp64(s.desc.data_ptr(), s.n, s.L, s.ds.ctypes.data,
                                                             s.b.grad.data_ptr(), s.lo, s.hi,
                                                             torch.cuda.current_stream().cuda_stream), "forms_backward")
        return {"ga": s.ga, "gb": s.gb}
    if kind == "cross_sections":
        dcs, tcs = s.tab.cross_sections_gpu(s.I[0], s.I[1])
        return {"dcs": dcs, "tcs": tcs}
    s.job.launch()
    if s.engine == "tc_bf16x3":
        return {"direct": s.job.out_dir, "exchange": s.job.out_ex}
    return {"integrals": s.job.out}


def _gradient_tensors(p, L):
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=DEV)  # noqa: E731
    x = dict(V_core=t(p.V), U_i=t(p.U), u_i=t(p.bi[0].u_of_r), u_f=t(p.bf[0].u_of_r),
             chi_i=t(np.stack([a.chi_of_r for a, _ in p.pairs])), chi_f=t(np.stack([b.chi_of_r for _, b in p.pairs])))
    return x, t(p.rng.normal(size=(len(p.pairs), 2, L + 1)))


# ------------------------------------------------------------------------------------------------ bytes and operations
def _n_parity(lm, par):
    return sum(1 for a in range(lm + 1) for b in range(lm + 1) if (a + b) % 2 == par)


def work(case):
    """Bytes: every input function and grid array read once, every output written once. Operations: per distinct wave
    product and multipole one multiply-add over the grid, for the direct and the exchange integral, beside the
    O(N L) sums of every distinct density."""
    kind, nl = case["kind"], case.get("L", 0) + 1
    if kind == "cross_sections":
        P, na = _n_parity(case["l_max"], 1), case["angles"]
        return dict(bytes=8.0 * (3 * P * (4 * nl + 2 * na) + 2 * P * nl + 2 * na), flops=3.0 * P * (8 * nl + 8 * na))
    if kind == "forms_backward":
        n, nf = case["n"], case["forms"]
        return dict(bytes=8.0 * n * (4 * nf + 1), flops=float(nf) * n * nl * 16)
    if kind == "sweep":
        tot, byt, lm, ne = 0.0, 0.0, case["l_max"], case["energies"]
        for e in range(ne):
            n = case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** (e / max(1, ne - 1))
            P = _n_parity(lm, 0) + _n_parity(lm, 1)
            tot += n * nl * (4.0 * P + 40.0 * (lm + 1))
            byt += 8.0 * (n * (4 * (lm + 1) + 5) + 2 * P * nl)
        return dict(bytes=byt, flops=tot)
    n, lm = case["n"], case.get("l_max", 0)
    if kind == "ionization":
        forms = sum(_n_parity(lm, q) * len(range(q, lm + 1, 2)) for q in (0, 1))
        return dict(bytes=8.0 * (n * (3 * (lm + 1) + 4) + 2 * forms * nl), flops=n * nl * (4.0 * forms + 40.0 * (lm + 1)))
    if kind in ("batch", "batch_call"):
        P, T = case["pairs"], case["transitions"]
        return dict(bytes=8.0 * (n * (2 * P + 2 * T + 3) + 2 * P * T * nl), flops=n * nl * P * T * 12.0)
    P = 1 if kind == "pair" else _n_parity(lm, 1)
    waves = 2 if kind == "pair" else 2 * (lm + 1)
    if kind == "gradient":
        return dict(bytes=8.0 * (n * (4 * P + 12) + 4 * P * nl), flops=n * nl * P * 40.0)
    return dict(bytes=8.0 * (n * (waves + 7) + 2 * P * nl), flops=n * nl * (4.0 * P + 20.0 * waves))


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _operators(r, k_total):
    """Bands of T (outer quadrature) and B (exchange inner quadrature) of one neutral node set over the whole grid: phase
    intervals of at most pi/4, refined down to pi/16 where the grid undersamples the phase, 5 nodes each."""
    n = len(r)
    d = math.pi / 4
    mx = k_total * float((r[1:] - r[:-1]).max())
    if mx > math.pi / 4:
        d = min(max(d * max(0.25, min(1.0, (math.pi / 4) / mx)), math.pi / 16), math.pi / 4)
    r0, r1 = float(r[0]), float(r[-1])
    br = torch.as_tensor(np.linspace(r0, r1, int(math.ceil((r1 - r0) / (d / k_total))) + 1), device=r.device)
    x5 = torch.cos(torch.arange(5, device=r.device, dtype=torch.float64) * (math.pi / 4))
    w5 = torch.tensor([1.0, 9.0, 11.0, 9.0, 1.0], device=r.device, dtype=torch.float64) / 15.0
    hw = 0.5 * (br[1:] - br[:-1])
    X = torch.minimum(torch.maximum(hw[:, None] * (x5 + 1.0) + br[:-1, None], br[:-1, None]), br[1:, None]).reshape(-1)
    W = (hw[:, None] * w5).reshape(-1)
    j = (torch.searchsorted(r, X, right=True) - 1).clamp(0, n - 2)
    t = torch.log1p((X - r[j]) / r[j]) / torch.log1p((r[j + 1] - r[j]) / r[j])
    c = torch.searchsorted(r, X).clamp(1, n - 1) - 1
    q = (X - r[c]) / (r[c + 1] - r[c] + 1e-30)
    T = torch.zeros((n, 3), dtype=torch.float64, device=r.device)
    B = torch.zeros((n, 5), dtype=torch.float64, device=r.device)

    def put(M, row, off, v, half):
        M.view(-1).index_add_(0, row * (2 * half + 1) + (off + half), v)
    for da, wa in ((0, 1 - t), (1, t)):
        for db, wb in ((0, 1 - t), (1, t)):
            put(T, j + da, db - da, W * wa * wb, 1)
        for dc, wc in ((0, 1 - q), (1, q)):
            put(B, c + dc, j + da - c - dc, W * wa * wc, 2)
    return T, B


def _band(M, f):
    """M f for rows of f, M a band given by its diagonals."""
    h = M.shape[1] // 2
    p = torch.nn.functional.pad(f, (h, h))
    return sum(M[:, k] * p[..., k:k + f.shape[-1]] for k in range(2 * h + 1))


def _bilinear(r, a, b, nl):
    """a^T K_L b for the rows of a and b, L = 0..nl-1 (last axis of the result)."""
    out = []
    for L in range(nl):
        lo, hi = r ** L, r ** (-(L + 1.0))
        A, B = torch.cumsum(a * lo, -1) - a * lo, torch.cumsum(b * lo, -1) - b * lo
        out.append((hi * (a * B + b * A)).sum(-1) + (a * b / r).sum(-1) * (1.0 - 1e-12) ** L)
    return torch.stack(out, -1)


def _exact_point(g, V, U, u_i, u_f, chi_i, chi_f, k_total, nl, chunk=64):
    """(P, 2, nl) integrals of one transition whose pairs share k_total, differentiable in the functions."""
    r, w = torch.as_tensor(g.r, device=DEV), torch.as_tensor(g.w_simpson, device=DEV)
    T, B = _operators(r, k_total)
    vd, rows = V - U, []
    for p in range(0, len(chi_i), chunk):
        ci, cf = chi_i[p:p + chunk], chi_f[p:p + chunk]
        d = _bilinear(r, _band(T, cf * ci), (w * u_f * u_i).expand_as(ci), nl)
        e = _bilinear(r, _band(T, u_f * ci), _band(B, cf * u_i), nl)
        zero = torch.zeros_like(d[:, 0])
        s, se = (w * u_f * u_i).sum(), (w * cf * u_i).sum(-1)
        cd = torch.where(s.abs() > 1e-12, (w * cf * ci * vd).sum(-1) * s, zero)
        ce = torch.where(se.abs() > 1e-12, (w * u_f * ci * vd).sum(-1) * se, zero)
        pad = lambda c: torch.nn.functional.pad(c[:, None], (0, nl - 1))  # noqa: E731
        rows.append(torch.stack([d + pad(cd), e + pad(ce)], 1))
    return torch.cat(rows)


def _point_tensors(p):
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=DEV)  # noqa: E731
    return (t(p.V), t(p.U), t(p.bi[0].u_of_r), t(p.bf[0].u_of_r), t(np.stack([a.chi_of_r for a, _ in p.pairs])),
            t(np.stack([b.chi_of_r for _, b in p.pairs])))


def exact(case, seed):
    kind, nl = case["kind"], case.get("L", 0) + 1
    if kind in ("pair", "point_call", "point"):
        p = _point_inputs(case, seed)
        V, U, u_i, u_f, ci, cf = _point_tensors(p)
        I = _exact_point(p.g, U if kind == "point" else V, U, u_i, u_f, ci, cf, p.pairs[0][0].k_au + p.pairs[0][1].k_au, nl)
        d, e = I[:, 0].cpu(), I[:, 1].cpu()
        if kind == "pair":
            return {"direct": d[0].numpy(), "exchange": e[0].numpy()}
        if kind == "point_call":
            return {"direct": d[None].numpy(), "exchange": e[None].numpy()}
        if case["engine"] == "tc_bf16x3":
            return {"direct": d, "exchange": e}
        return {"integrals": torch.stack([d, e], 1).reshape(-1, nl)}
    if kind == "gradient":
        p = _point_inputs(case, seed)
        x, c = _gradient_tensors(p, case["L"])
        x = {k: v.requires_grad_(True) for k, v in x.items()}
        g = {k: torch.zeros_like(v) for k, v in x.items()}
        rows = []
        for q in range(0, len(p.pairs), 32):  # pairs are independent: their gradients add up
            s = slice(q, q + 32)
            I = _exact_point(p.g, x["V_core"], x["U_i"], x["u_i"], x["u_f"], x["chi_i"][s], x["chi_f"][s],
                             p.pairs[0][0].k_au + p.pairs[0][1].k_au, nl)
            for k, v in zip(x, torch.autograd.grad((I * c[s]).sum(), list(x.values()))):
                g[k] += v
            rows.append(I.detach())
        return {"I": torch.cat(rows), **{"d_" + k: v for k, v in g.items()}}
    if kind in ("batch", "batch_call"):
        p = _batch_inputs(case, seed)
        if case["n"] * case["pairs"] > 15000 * 2048:
            return None
        r, w = torch.as_tensor(p.g.r, device=DEV), torch.as_tensor(p.g.w_simpson, device=DEV)
        ui = torch.as_tensor(np.stack([b.u_of_r for b in p.bi]), device=DEV)
        uf = torch.as_tensor(np.stack([b.u_of_r for b in p.bf]), device=DEV)
        out = torch.empty((case["transitions"], case["pairs"], 2, nl), dtype=torch.float64, device=DEV)
        for q, (a, b) in enumerate(p.pairs):
            T, B = _operators(r, a.k_au + b.k_au)
            ci, cf = (torch.as_tensor(x.chi_of_r, device=DEV) for x in (a, b))
            A = torch.cat([_band(T, cf * ci).expand_as(uf), _band(T, uf * ci)])
            I = _bilinear(r, A, torch.cat([w * uf * ui, _band(B, cf * ui)]), nl)
            out[:, q, 0], out[:, q, 1] = I[:len(uf)], I[len(uf):]
        if kind == "batch":
            return {"integrals": out.reshape(-1, nl)}
        return {"direct": out[:, :, 0].cpu().numpy(), "exchange": out[:, :, 1].cpu().numpy()}
    if kind == "forms_backward":
        x = _backward_inputs(case, seed)
        r = x.r
        at = torch.arange(case["n"], device=DEV)
        in_a, in_b = at < torch.as_tensor(x.rows, device=DEV)[:, None], at < torch.as_tensor(x.cols, device=DEV)[:, None]
        a, b = x.a * in_a, x.b * in_b
        ga, gb = torch.zeros_like(a), torch.zeros_like(b)
        for y, z in ((b, ga), (a, gb)):
            for L in range(nl):
                lo, hi = r ** L, r ** (-(L + 1.0))
                pre = torch.cumsum(y * lo, -1) - y * lo
                suf = torch.flip(torch.cumsum(torch.flip(y * hi, (-1,)), -1), (-1,)) - y * hi
                z += x.grad[:, L:L + 1] * (hi * pre + lo * suf + (1.0 - 1e-12) ** L * y / r)
        return {"ga": ga * in_a, "gb": gb * in_b}
    if kind == "cross_sections":
        from dwba_b200.coupling import CouplingTables  # its coupling tables are inputs here
        ch, I, k_i, k_f = _cross_inputs(case, seed)
        th = np.linspace(0.0, math.pi, case["angles"])
        t = CouplingTables(th, ch, case["L"], k_i, k_f, 0, 1)
        f = np.einsum("ap,apt->at", np.einsum("apl,pl->ap", t.cf, I[0]), t.yd)
        g = np.einsum("ap,apt->at", np.einsum("apl,pl->ap", t.cg, I[1]), t.ye)
        dcs = np.clip((t.pref * (0.25 * np.abs(f + g) ** 2 + 0.75 * np.abs(f - g) ** 2)).sum(0), 0.0, None)
        return {"dcs": dcs, "tcs": np.array([2.0 * math.pi * np.trapezoid(np.sin(th) * dcs, th)])}
    return None  # sweep, ionization: Coulomb phase intervals and outer tails pair by pair take far over 20 s
