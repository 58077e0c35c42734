"""dwba_outer_tails_batch where its split can go wrong, against the native host path: one segment, intervals too short
to oscillate, more nodes than a CTA's threads take in one round, capped segment counts (more nodes per segment),
Levin branches, one and several multipole chunks, and one record, a few and enough that a CTA takes several.

Both sum the same node values; the composite sum differs by rounding: 1e-13 of the value plus 1e-14 of the integral
of the envelope (and 1e-16 times the condition number on Levin segments, whose systems two solvers solve apart; a
system that is singular to working precision has no value to compare)."""
import numpy as np
import pytest

from dwba_b200 import _lib
from golden_cases import levin_condition
from test_gpu_tails import _device_tails

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L_max", [1, 7, 8, 9, 17])
@pytest.mark.parametrize("copies", [1, 40])
def test_tails_at_the_edges(L_max, copies):
    rng = np.random.default_rng(L_max)
    waves, rm, rmax = [], [], []
    for k_i, k_f, l_i, l_f, a, b in ((1.3, 1.29, 0, 1, 40.0, 40.7), (1.3, 1.3004, 2, 1, 50.0, 50.5), (8.0, 7.5, 3, 40, 60.0, 400.0),
                                     (6.0, 5.0, 1, 0, 10.0, 3000.0), (0.9, 0.5, 14, 9, 30.0, 200.0), (2.0, 1.0, 0, 0, 120.0, 200.0),
                                     (1.9, 0.4, 25, 25, 20.0, 150.0)):
        for eta in (0.0, -1.0):
            d = rng.uniform(0, 3, 4)
            waves.append([k_i, l_i, d[0], eta / k_i, d[1], k_f, l_f, d[2], eta / k_f, d[3]])
            rm.append(a)
            rmax.append(b)
    keep = [q for q, w in enumerate(waves) if _lib.tail_on_device(w, rm[q], rmax[q])]
    assert len(keep) > 8
    mom = rng.normal(size=(len(waves), L_max + 1)) * 10.0 ** np.arange(L_max + 1)
    mom[0, 1:] = 0.0  # a record without moments
    idx = np.tile(keep, copies)
    got = _device_tails(np.array(waves)[idx], np.array(rm)[idx], np.array(rmax)[idx], mom[idx], 0, L_max)
    assert np.array_equal(got, np.tile(got[:len(keep)], (copies, 1)))  # independent of the records around
    for g, q in zip(got, keep):
        want = _lib.outer_tails(waves[q], rm[q], rmax[q], L_max, mom[q], 0, 4096, np.pi / 2)
        L = np.arange(L_max + 1)
        env = np.abs(mom[q]) * rm[q] ** -(L + 1.0) * (rmax[q] - rm[q])
        cond = levin_condition(waves[q], rm[q], rmax[q])
        if cond >= 1.0 / np.finfo(float).eps:
            assert np.all(np.isfinite(g))
            continue
        tol = 1e-13 * np.abs(want) + (1e-14 + 1e-16 * cond) * env
        assert g[0] == 0.0 and np.all(np.abs(g - want)[1:] <= tol[1:] + 1e-300), (q, g, want)
