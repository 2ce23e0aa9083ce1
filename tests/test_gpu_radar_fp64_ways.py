"""Points formed in FP64 by their whole warp and by their own lane: the same sums in the same order. With the amplitudes
scaled by 2^-100 every point goes to FP64; a lone point of an image is formed by the warp (but with a single
element on either side), a whole warp of them by its lanes. Equal bit for bit, on both sides of 32 elements, and
not-a-number behind the transmitting elements in both."""
import numpy as np
import pytest
from test_gpu_radar_edges import _case

from em_lab_gb300.radar import RadarMonitor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,ntx", [(1, 2), (5, 3), (32, 32), (33, 31), (40, 65)])
def test_one_point_equals_its_place_in_an_image(C, ntx):
    array, z, g = _case(C, ntx, (4, 8, 16), C)
    array.tx_amp = array.tx_amp * 2.0 ** -100
    g.r0, g.dr = -8.0, 20.0  # the first range bin lies behind the array
    image = RadarMonitor.backproject(array, z, g)
    assert (image > 0).any() and np.isnan(image[0]).any()
    r0, az0, el0 = g.r0, g.az0, g.el0
    for ir, ie, ia in [(0, 0, 0), (0, 7, 15), (1, 3, 8), (2, 0, 15), (3, 7, 0), (3, 4, 5)]:
        g.nr = g.nel = g.naz = 1
        g.r0, g.el0, g.az0 = r0 + ir * g.dr, el0 + ie * g.del_, az0 + ia * g.daz
        np.testing.assert_array_equal(RadarMonitor.backproject(array, z, g)[0, 0, 0], image[ir, ie, ia])
