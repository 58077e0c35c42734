"""Backward of many forms: short ones (up to 1536 points) take a kernel of their own, in one launch with longer ones."""
import numpy as np
import pytest

from test_gpu_backward_edges import EPS, _grads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L_max", [0, 7, 10])
def test_short_and_long_forms_together(L_max):
    import torch
    from dwba_b200 import _lib
    from dwba_b200.plan import diag_scale
    rng = np.random.default_rng(L_max)
    n, F = 2100, 210
    r = np.geomspace(1e-3, 60.0, n)
    nr = rng.choice([1, 2, 127, 129, 1500, 1535, 1536, 1537, 2100], F)
    nc = rng.choice([1, 128, 1501, 1535, 1536, 1537, 2100], F)
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda")  # noqa: E731
    a, b = rng.normal(size=(2, F, n))
    a[np.arange(n)[None, :] >= nr[:, None]] = 0.0
    b[np.arange(n)[None, :] >= nc[:, None]] = 0.0
    g = rng.normal(size=(F, L_max + 1))
    rd, A, B, G = t(r), t(a), t(b), t(g)
    GA, GB = torch.full_like(A, np.nan), torch.full_like(B, np.nan)
    d = np.zeros(F, dtype=_lib.FORM_GRAD_DTYPE)
    for f in range(F):
        d[f] = (rd.data_ptr(), A[f].data_ptr(), B[f].data_ptr(), GA[f].data_ptr(), GB[f].data_ptr(), nr[f], nc[f])
    dd = torch.from_numpy(d.view(np.uint8).copy()).cuda()
    ds = diag_scale(L_max)
    _lib.check(_lib.load().dwba_bilinear_semisep_backward_fp64(
        dd.data_ptr(), F, L_max, ds.ctypes.data, G.data_ptr(), float(r[0]), float(r[-1]),
        torch.cuda.current_stream().cuda_stream), "backward")
    ga, gb = GA.cpu().numpy(), GB.cpu().numpy()
    for f in range(0, F, 14):
        wa, wb = _grads(r, a[f], b[f], g[f])
        sa, sb = _grads(r, np.abs(a[f]), np.abs(b[f]), np.abs(g[f]))
        for got, want, scale, m in ((ga[f], wa, sa, nr[f]), (gb[f], wb, sb, nc[f])):
            assert np.all(np.isnan(got[m:]))
            # rounding of about n additions on the terms, as at the tiles' edges
            assert np.all(np.abs(got[:m] - want[:m]) <= 4 * EPS * np.sqrt(n) * scale[:m] + 1e-300)
