"""The record's way to the device: rows of z beyond every point's delay change nothing, on either side of the
128 KB up to which z travels in one copy with the other inputs."""
import numpy as np
import pytest
from test_gpu_radar_edges import _case

from em_lab_gb300.radar import RadarMonitor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [4095, 4096, 4097, 70000])
def test_long_records_are_copied_like_short_ones(M):
    array, z, g = _case(4, 3, (10, 9, 9), 11, M=400)
    want = RadarMonitor.backproject(array, z, g)
    assert (want > 0).any()
    longer = np.concatenate([z, np.full((M - len(z), 4), 7.0 + 3.0j, np.complex64)])
    np.testing.assert_array_equal(RadarMonitor.backproject(array, longer, g), want)
