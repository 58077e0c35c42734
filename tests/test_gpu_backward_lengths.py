"""Backward of the bilinear forms over the lengths that are laid out differently: up to 1664 points one CTA per gradient,
above that half a cluster with 8 points per thread (to 2048) or 16 (to 4096), then a cluster (one tile up to 8192
points). The lengths sit on both sides of each line and on the segments' (a multiple of 128) edges. A form's gradient
must not depend on how many forms, of whatever lengths, share its launch. Reference and tolerance: those of the tests
at the tiles' edges."""
import numpy as np
import pytest

from test_gpu_backward_edges import EPS, _grads

pytestmark = pytest.mark.gpu


def _run(r, a, b, g, nr, nc, L_max):
    import torch
    from dwba_b200 import _lib
    from dwba_b200.plan import diag_scale
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda")  # noqa: E731
    rd, A, B, G = t(r), t(a), t(b), t(g)
    GA, GB = torch.full_like(A, np.nan), torch.full_like(B, np.nan)
    d = np.zeros(len(a), dtype=_lib.FORM_GRAD_DTYPE)
    for f in range(len(a)):
        d[f] = (rd.data_ptr(), A[f].data_ptr(), B[f].data_ptr(), GA[f].data_ptr(), GB[f].data_ptr(), nr[f], nc[f])
    dd = torch.from_numpy(d.view(np.uint8).copy()).cuda()
    ds = diag_scale(L_max)
    _lib.check(_lib.load().dwba_bilinear_semisep_backward_fp64(
        dd.data_ptr(), len(a), L_max, ds.ctypes.data, G.data_ptr(), float(r[0]), float(r[-1]),
        torch.cuda.current_stream().cuda_stream), "backward")
    return GA.cpu().numpy(), GB.cpu().numpy()


def _forms(n, nr, nc, L_max, seed):
    rng = np.random.default_rng(seed)
    a, b = rng.normal(size=(2, len(nr), n))
    a[np.arange(n)[None, :] >= np.asarray(nr)[:, None]] = 0.0
    b[np.arange(n)[None, :] >= np.asarray(nc)[:, None]] = 0.0
    return a, b, rng.normal(size=(len(nr), L_max + 1))


@pytest.mark.parametrize("L_max", [0, 4, 7, 8, 10, 17])
def test_lengths(L_max):
    n = 3001  # the reference by cumulative sums
    m = np.array([1, 2, 127, 128, 129, 1279, 1281, 1536, 1537, 1663, 1664, 1665, 2047, 2048, 2049, 2800])
    nr, nc = np.concatenate([m, m, np.minimum(m, 900)]), np.concatenate([m, np.maximum(1, m // 2), m])
    r = np.geomspace(1e-2, 60.0, n)
    a, b, g = _forms(n, nr, nc, L_max, L_max)
    ga, gb = _run(r, a, b, g, nr, nc, L_max)
    for f in range(len(nr)):
        wa, wb = _grads(r, a[f], b[f], g[f])
        sa, sb = _grads(r, np.abs(a[f]), np.abs(b[f]), np.abs(g[f]))
        for got, want, scale, k in ((ga[f], wa, sa, nr[f]), (gb[f], wb, sb, nc[f])):
            assert np.all(np.isnan(got[k:]))
            assert np.all(np.abs(got[:k] - want[:k]) <= 4 * EPS * np.sqrt(n) * scale[:k] + 1e-300), (f, nr[f], nc[f])


@pytest.mark.parametrize("n", [4095, 4096, 4097, 8193])
def test_long_forms(n):
    r = np.geomspace(1e-2, 60.0, n)
    nr, nc = np.array([n, n - 3]), np.array([n, n])
    a, b, g = _forms(n, nr, nc, 5, n)
    ga, gb = _run(r, a, b, g, nr, nc, 5)
    for f in range(2):
        wa, wb = _grads(r, a[f], b[f], g[f])
        sa, sb = _grads(r, np.abs(a[f]), np.abs(b[f]), np.abs(g[f]))
        for got, want, scale, k in ((ga[f], wa, sa, nr[f]), (gb[f], wb, sb, nc[f])):
            assert np.all(np.abs(got[:k] - want[:k]) <= 4 * EPS * np.sqrt(n) * scale[:k] + 1e-300)


@pytest.mark.parametrize("L_max", [3, 9])
def test_a_gradient_does_not_depend_on_the_launch(L_max):
    n = 4200
    r = np.geomspace(1e-2, 60.0, n)
    m = np.array([100, 700, 1500, 1600, 1800, 2048, 3000, 4200])
    nr, nc = np.tile(m, 30), np.tile(m[::-1], 30)  # 240 forms
    nr[:len(m)] = nc[:len(m)] = m
    a, b, g = _forms(n, nr, nc, L_max, 5)
    ga, gb = _run(r, a, b, g, nr, nc, L_max)
    for k in (1, len(m)):
        xa, xb = _run(r, a[:k], b[:k], g[:k], nr[:k], nc[:k], L_max)
        assert np.array_equal(xa, ga[:k], equal_nan=True) and np.array_equal(xb, gb[:k], equal_nan=True)
