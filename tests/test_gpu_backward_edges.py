"""Backward of the bilinear forms at the edges of its tiles.

The backward splits a form's points into runs of 16 per thread, 512 per warp and 2048 per CTA, four CTAs per
gradient (up to 8192 points in one tile each); longer forms walk their tiles. The sizes below sit on and around
those edges, with n_rows != n_cols and multipoles in one and in several launches. Reference: the oracle's dense
gradients below 3000 points, else the same sums as long-double cumulative sums. The error of an entry is bounded
by the rounding of about n additions on its terms: 4 eps sqrt(n) times the sum of their magnitudes.
"""
import numpy as np
import pytest

from oracle.backward import form_grads

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _grads(r, a, b, g):
    if len(r) <= 3000:
        return form_grads(r, a, b, g)
    x = r.astype(np.longdouble)
    out = []
    for y in (b, a):
        z = np.zeros_like(x)
        for L, gl in enumerate(g):
            lo, hi = x ** L, x ** -(L + 1)
            pre = np.cumsum(y * lo) - y * lo
            suf = np.cumsum((y * hi)[::-1])[::-1] - y * hi
            z += gl * (hi * pre + lo * suf + (1.0 - 1e-12) ** L * y / x)
        out.append(z.astype(float))
    return out


@pytest.mark.parametrize("n,nr,nc,L_max", [
    (2, 1, 2, 0), (17, 16, 15, 3), (513, 512, 511, 4), (2049, 2048, 2049, 8), (2049, 2049, 700, 7), (2100, 3, 2100, 9),
    (8192, 8192, 8191, 2), (8193, 8193, 8193, 4), (12001, 9000, 12001, 8), (16500, 16500, 2, 1)])
def test_backward_at_tile_edges(n, nr, nc, L_max):
    import torch
    from dwba_b200 import _lib
    from dwba_b200.plan import diag_scale
    rng = np.random.default_rng(n + L_max)
    r = np.geomspace(1e-3, 60.0, n)
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda")  # noqa: E731
    a, b = np.zeros((2, n)), np.zeros((2, n))
    a[:, :nr], b[:, :nc] = rng.normal(size=(2, nr)), rng.normal(size=(2, nc))
    g = rng.normal(size=(2, L_max + 1))
    rd, A, B, G = t(r), t(a), t(b), t(g)
    GA, GB = torch.full_like(A, np.nan), torch.full_like(B, np.nan)
    d = np.zeros(2, dtype=_lib.FORM_GRAD_DTYPE)
    for f in range(2):
        d[f] = (rd.data_ptr(), A[f].data_ptr(), B[f].data_ptr(), GA[f].data_ptr(), GB[f].data_ptr(), nr, nc)
    dd = torch.from_numpy(d.view(np.uint8).copy()).cuda()
    ds = diag_scale(L_max)
    _lib.check(_lib.load().dwba_bilinear_semisep_backward_fp64(
        dd.data_ptr(), 2, L_max, ds.ctypes.data, G.data_ptr(), float(r[0]), float(r[-1]),
        torch.cuda.current_stream().cuda_stream), "backward")
    ga, gb = GA.cpu().numpy(), GB.cpu().numpy()
    for f in range(2):
        wa, wb = _grads(r, a[f], b[f], g[f])
        sa, sb = _grads(r, np.abs(a[f]), np.abs(b[f]), np.abs(g[f]))
        for got, want, scale, m in ((ga[f], wa, sa, nr), (gb[f], wb, sb, nc)):
            assert np.all(np.isnan(got[m:]))  # rows past the operand are not written
            assert np.all(np.abs(got[:m] - want[:m]) <= 4 * EPS * np.sqrt(n) * scale[:m] + 1e-300)
