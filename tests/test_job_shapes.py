"""A job whose functions do not fit its grid is refused when its L = 0 corrections are live."""
import numpy as np
import pytest
import torch

import bench
from dwba_b200 import engine as E


def _plan(**other):
    from dwba_b200.plan import GridInfo
    n = 150
    g = bench.make_grid(n, 0.05, 300.0)
    z = np.zeros(n)
    f = dict(V_core=-1.0 / g.r, U_i=z, u_i=g.r * np.exp(-g.r), u_f=g.r ** 2 * np.exp(-g.r))
    f.update(other)
    w = [bench._Wave(l, 2.0 - 0.5 * l, 0.0, np.sin(2 * g.r)) for l in range(2)]
    info = GridInfo(g.r, g.w_simpson, g.w_trapz)
    job = E.Job(grid=info, V_core=f["V_core"], U_i=f["U_i"], U_f=f.get("U_f"), pairs=[(w[0], w[1])], L_max=3,
                transitions=[E.Transition(u_i=f["u_i"], u_f=f["u_f"], excitation=True)])
    return E.plan_job(job)


@pytest.mark.parametrize("names", [("u_i",), ("u_f",), ("u_i", "u_f"), ("V_core", "U_i"),
                                   ("V_core", "U_i", "U_f")])
@pytest.mark.parametrize("n", [149, 151])
def test_functions_of_another_length_are_refused(names, n):
    assert np.all(_plan().corr_dir != 0)
    with pytest.raises((ValueError, IndexError)):
        _plan(**{k: np.linspace(0.1 * (i + 1), 1.0, n) for i, k in enumerate(names)})
