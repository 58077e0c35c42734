"""Potentials of a launch that does not know their lengths, few and many of them together: a potential takes the CTAs of
its cluster that it fills. Lengths on both sides of one CTA's and one cluster's tile; reference: long-double sums, 1e-14
of the sum of the terms' magnitudes. (Few: the whole cluster each.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies,L_max", [(1, 3), (3, 0), (3, 12), (3, 25)])
def test_lengths_mixed_in_one_launch(copies, L_max):
    import torch
    from dwba_b200 import _lib
    from dwba_b200.plan import diag_scale
    lens = np.array([1, 255, 256, 257, 1023, 1024, 1025, 2049, 3000, 7169, 8191, 8192, 8193, 9300])
    shapes = [(a, b) for n in lens for a, b in ((n, n), (n, max(1, n // 3)), (max(1, n // 2), n))][:37 if copies == 1 else 99]
    shapes *= copies
    n, nl = int(lens.max()), L_max + 1
    rng = np.random.default_rng(L_max)
    r = np.geomspace(1e-2, 60.0, n)
    b = rng.normal(size=(len(shapes), n)) * np.exp(-r / 10)
    rd, bd = torch.as_tensor(r, device="cuda"), torch.as_tensor(b, device="cuda")
    phi = torch.full((len(shapes), nl, n), np.nan, dtype=torch.float64, device="cuda")
    rec = np.zeros(len(shapes), dtype=_lib.POTENTIAL_DTYPE)
    for k, (nr, nc) in enumerate(shapes):
        rec[k] = (rd.data_ptr(), bd[k].data_ptr(), phi[k].data_ptr(), nr, nc, n, 0)
    recd = torch.from_numpy(rec.view(np.uint8).copy()).cuda()
    ds = diag_scale(L_max)
    _lib.check(_lib.load().dwba_multipole_potentials(recd.data_ptr(), len(shapes), L_max, ds.ctypes.data, float(r[0]),
                                                     float(r[-1]), torch.cuda.current_stream().cuda_stream), "potentials")
    x = r.astype(np.longdouble)
    rows = {L: (x ** L, x ** -(L + 1)) for L in {0, L_max // 2, L_max}}
    for k, (nr, nc) in enumerate(shapes):
        y = np.where(np.arange(n) < nc, b[k], 0.0).astype(np.longdouble)
        for L, (lo, hi) in rows.items():
            got = phi[k, L].cpu().numpy()

            def f(z):
                suf = np.cumsum((z * hi)[::-1])[::-1] - z * hi
                return (hi * (np.cumsum(z * lo) - z * lo) + lo * suf + (1 - 1e-12) ** L * z / x)[:nr]
            assert np.all(np.abs(got[:nr] - f(y)) <= 1e-14 * f(np.abs(y))), (nr, nc, L)
            assert np.all(np.isnan(got[nr:]))
