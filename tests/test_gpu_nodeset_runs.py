"""Node-set operators where whole phase intervals are summed in closed form: dwba_build_nodesets against the NumPy
model that sums node by node, entry by entry.

Cases: many, two, one and no whole intervals per grid interval; n1 < N; several rule sizes; log and linear taps (and
one of each); steps above and below 2^-9 and above 1/64 (no closed form); breakpoints that coincide with grid points;
a rule that is not symmetric (no closed form). A node's position carries a rounding of eps r, which moves a tap by
that over the grid step and an interval's width by that over the width; the closed form uses the exact positions, so
an entry may differ by those roundings times the weight that reaches its row, plus a few eps of that weight.
"""
import numpy as np
import pytest

import kernel_model as km

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _model(r, n1, nb, x_ref, w_ref, log1, log2, monkeypatch):
    monkeypatch.setattr(km, "cc_reference", lambda n: (x_ref, w_ref))
    return km.bands(r, n1, nb, None, len(x_ref), log1, log2), km.node_arrays(r, n1, nb, None, len(x_ref))


@pytest.mark.parametrize("N,n1,r_max,nb,n_cc,log1,log2,rule", [
    (3000, 3000, 400.0, 20000, 5, 1, 1, "cc"),    # up to 40 whole intervals, step 5.8e-3
    (15000, 15000, 400.0, 17000, 5, 1, 1, "cc"),  # step 1.2e-3
    (15000, 13017, 200.0, 9001, 5, 1, 1, "cc"),
    (2000, 1500, 100.0, 300, 7, 1, 1, "cc"),      # at most one or two
    (1000, 1000, 300.0, 4000, 5, 1, 1, "cc"),     # step above 1/64: node by node
    (1001, 1001, 50.0, 2001, 5, 0, 0, "linear"),  # every second breakpoint on a grid point
    (1001, 900, 50.0, 4501, 4, 0, 0, "linear"),
    (3000, 2500, 200.0, 6000, 2, 1, 0, "cc"),
    (3000, 3000, 200.0, 6000, 15, 0, 1, "cc"),
    (3000, 3000, 200.0, 6000, 5, 1, 1, "skew"),
])
def test_runs_match_node_by_node(N, n1, r_max, nb, n_cc, log1, log2, rule, monkeypatch):
    import torch
    from dwba_b200 import _lib
    from dwba_b200.plan import cc_reference
    x_ref, w_ref = cc_reference(n_cc)
    if rule == "skew":
        w_ref = w_ref * np.linspace(0.5, 1.5, n_cc)
    r = np.linspace(0.05, r_max + 0.05, N) if rule == "linear" else np.geomspace(1e-5, r_max, N)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")  # noqa: E731
    rd, ld, xd, wd = t(r), t(np.log(r)), t(x_ref), t(w_ref)
    ta = torch.full((3 * n1,), np.nan, dtype=torch.float64, device="cuda")
    bx = torch.full((5 * N,), np.nan, dtype=torch.float64, device="cuda")
    rec = np.zeros(1, dtype=_lib.NODESET_DTYPE)
    rec["r"], rec["logr"], rec["ta"], rec["bx"] = rd.data_ptr(), ld.data_ptr(), ta.data_ptr(), bx.data_ptr()
    rec["n_grid"], rec["n1"], rec["n_breaks"], rec["log1"], rec["log2"] = N, n1, nb, log1, log2
    recd = torch.from_numpy(rec.view(np.uint8).copy()).cuda()
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.check(_lib.load().dwba_build_nodesets(recd.data_ptr(), 1, N, xd.data_ptr(), wd.data_ptr(), n_cc, st.data_ptr(),
                                               torch.cuda.current_stream().cuda_stream), "nodesets")
    assert int(st.item()) == 0
    (mt, mb), (x, w) = _model(r, n1, nb, x_ref, w_ref, log1, log2, monkeypatch)
    # weight that reaches a row: nodes of its own and the two neighbouring grid intervals
    g = np.clip(np.searchsorted(r, x, side="right") - 1, 0, N - 1)
    per = np.bincount(g, np.abs(w), minlength=N)
    wt = per + np.roll(per, 1) + np.roll(per, 2) + np.roll(per, -1)
    dr = np.diff(r, append=r[-1] + (r[-1] - r[-2]))
    width = (r[n1 - 1] - r[0]) / (nb - 1)
    log_tap = 4 * EPS * np.abs(np.log(r)) / np.log(r[1] / r[0])  # log r_{g+1} - log r_g is a rounded difference
    tol = wt * (64 * EPS + 8 * EPS * r * (1.0 / dr + 1.0 / width) + (log_tap if log1 or log2 else 0.0)) + 1e-300
    for got, want, m, k in ((ta, mt, n1, 3), (bx, mb, N, 5)):
        d = np.abs(got.cpu().numpy().reshape(m, k) - want.reshape(m, k))
        assert np.all(d <= tol[:m, None]), (np.max(d / tol[:m, None]), np.unravel_index(np.argmax(d / tol[:m, None]), d.shape))
