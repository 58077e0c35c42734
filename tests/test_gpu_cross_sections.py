"""The cross-section kernel at the edges of its angle tiles (32 angles) and channel chunks (256 channels of each of a
cluster's eight CTAs), against the amplitudes as NumPy sums. An amplitude is off by at most eps (P + nl) times the sum
of its terms' magnitudes, which bounds the DCS."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


@pytest.mark.parametrize("n_M,P,nl,n_theta", [(1, 1, 1, 1), (3, 7, 5, 32), (2, 9, 3, 33), (5, 2049, 7, 181), (1, 2056, 11, 31)])
def test_cross_sections_at_tile_edges(n_M, P, nl, n_theta):
    import torch
    from dwba_b200 import _lib
    rng = np.random.default_rng(P + n_theta)
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda")  # noqa: E731
    cf, cg = (rng.normal(size=(n_M, P, nl)) + 1j * rng.normal(size=(n_M, P, nl)) for _ in range(2))
    yd, ye = rng.normal(size=(2, n_M, P, n_theta))
    I = rng.normal(size=(2, P, nl))
    th = np.linspace(0.0, np.pi, n_theta) if n_theta > 1 else np.array([0.3])
    dev = [t(cf.view(float)), t(cg.view(float)), t(yd), t(ye), t(I[0]), t(I[1]), t(th)]
    dcs = torch.full((n_theta,), np.nan, dtype=torch.float64, device="cuda")
    tcs = torch.full((1,), np.nan, dtype=torch.float64, device="cuda")
    _lib.check(_lib.load().dwba_cross_sections(*(x.data_ptr() for x in dev), n_M, P, nl, n_theta, 0.7, dcs.data_ptr(),
                                               tcs.data_ptr(), torch.cuda.current_stream().cuda_stream), "dcs")
    f = np.einsum("ap,apt->at", np.einsum("apl,pl->ap", cf, I[0]), yd)
    g = np.einsum("ap,apt->at", np.einsum("apl,pl->ap", cg, I[1]), ye)
    want = 0.7 * (0.25 * np.abs(f + g) ** 2 + 0.75 * np.abs(f - g) ** 2).sum(0)
    # an amplitude is off by at most eps (P + nl) times the sum of its terms' magnitudes
    s = np.einsum("ap,apt->at", np.einsum("apl,pl->ap", np.abs(cf), np.abs(I[0])), np.abs(yd)) + \
        np.einsum("ap,apt->at", np.einsum("apl,pl->ap", np.abs(cg), np.abs(I[1])), np.abs(ye))
    tol = 0.7 * 8 * (np.abs(f) + np.abs(g) + EPS * (P + nl) * s).max() * EPS * (P + nl) * s.sum(0)
    got = dcs.cpu().numpy()
    assert np.all(np.abs(got - want) <= tol + 1e-14 * want)
    if n_theta > 1:
        ref = 2 * np.pi * np.trapezoid(np.sin(th) * got, th)
        assert abs(float(tcs) - ref) <= 1e-13 * 2 * np.pi * np.trapezoid(np.sin(th) * np.abs(got), th)
    else:
        assert float(tcs) == 0.0
