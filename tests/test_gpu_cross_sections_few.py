"""Cross sections of few channels at many angles, on both sides of the line between its two kernels (320 angles per
channel), against NumPy sums; tolerance as at the tiles' edges."""
import pytest

from test_gpu_cross_sections import test_cross_sections_at_tile_edges as _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_M,P,nl,n_theta", [(1, 1, 1, 320), (1, 1, 1, 321), (3, 3, 5, 960), (3, 3, 5, 961), (2, 2, 33, 700),
                                              (2, 5, 7, 5003), (1, 40, 3, 13000)])
def test_few_channels_at_many_angles(n_M, P, nl, n_theta):
    _check(n_M, P, nl, n_theta)
