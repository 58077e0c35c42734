"""L=0 corrections and the routing of outer tails, formed natively for all pairs of a transition."""
import numpy as np
import pytest

from dwba_b200 import _lib


@pytest.mark.parametrize("N", [1, 3, 4, 255, 256, 257, 1003])
def test_l0_corrections(N):
    rng = np.random.default_rng(N)
    P = 7
    w, v = rng.random(N) + 0.1, rng.standard_normal(N)
    u_i, u_f = rng.standard_normal(N), rng.standard_normal(N)
    chi = rng.standard_normal((2 * P, N))
    rows_i, rows_f = rng.integers(0, 2 * P, P), rng.integers(0, 2 * P, P)
    n1 = rng.integers(1, N + 1, P)
    n1[3] = n1[2]
    base, step = chi.ctypes.data, 8 * N
    got = _lib.l0_corrections(base + step * rows_i, base + step * rows_f, n1, w, u_i, u_f, v, 1e-12)
    ld = np.longdouble
    for p in range(P):
        wl = np.where(np.arange(N) < n1[p], w, 0.0).astype(ld)
        ci, cf = chi[rows_i[p]].astype(ld), chi[rows_f[p]].astype(ld)
        terms = ((wl * cf * ci * v, wl * u_f * u_i), (wl * u_f * ci * v, wl * cf * u_i))
        for k, (a, b) in enumerate(terms):
            # a term is a product of four factors, a block's running sums take at most 64 additions each
            eps = np.finfo(float).eps
            tol = (64 + 8) * eps * (np.abs(a).sum() * np.abs(b.sum()) + np.abs(a.sum()) * np.abs(b).sum() +
                                    72 * eps * np.abs(a).sum() * np.abs(b).sum())
            assert abs(got[k][p] - a.sum() * b.sum()) <= tol
            alone = _lib.l0_corrections(base + step * rows_i[p:p + 1], base + step * rows_f[p:p + 1], n1[p:p + 1], w,
                                        u_i, u_f, v, 1e-12)
            assert alone[k][0] == got[k][p]


def test_l0_corrections_gate_and_lengths():
    N = 40
    x = np.ones((1, N))
    z = np.zeros(N)
    addr = np.array([x.ctypes.data])
    one, n1 = np.ones(N), np.array([N])
    assert _lib.l0_corrections(addr, addr, n1, one, z, one, one, 1e-12)[0][0] == 0.0
    assert _lib.l0_corrections(addr, addr, n1, one, one, one, np.full(N, np.nan), 1e-12)[0][0] != 0.0
    with pytest.raises(ValueError):
        _lib.l0_corrections(addr, addr, n1, one, one[:-1], one, one, 1e-12)


def test_tails_on_device_rows():
    rng = np.random.default_rng(5)
    waves = np.abs(rng.standard_normal((20, 10))) + 0.2
    waves[::3, 5:] = waves[::3, :5]  # equal waves: the difference phase stands still
    r_m = rng.uniform(5.0, 50.0, 20)
    got = _lib.tails_on_device(waves, r_m, 200.0)
    assert got.tolist() == [_lib.tail_on_device(w, m, 200.0) for w, m in zip(waves, r_m)]
    assert got.any() and not got.all()
    assert _lib.tails_on_device(np.zeros((0, 10)), np.zeros(0), 200.0).shape == (0,)
