"""The back-projection kernel sums pairs of FP32 and forms points it cannot decide again in FP64. Amplitudes
scaled by 2^-100 leave the image as it is (the delay is a ratio) but send every point down the FP64 path, which
is the reference's arithmetic: the two images agree to the 2e-8 of a point's power that the kernel lets a
rounding of the interpolation weight move, plus the pairs' own error (some 2^-45 of the sum of magnitudes)."""
import math

import numpy as np
import pytest

from em_lab_gb300 import abi
from em_lab_gb300.radar import RadarMonitor

pytestmark = pytest.mark.gpu


def _case(C, ntx, shape, seed, M=50):
    rng = np.random.default_rng(seed)
    g = abi.RadarGeometry()
    tx = np.array([20.3, 40.1, 39.7], np.float32)
    for k in range(3):
        g.tx[k], g.interior_min[k], g.interior_max[k] = float(tx[k]), 5.0, 110.0
    for k, v in enumerate([0, -1, 0, 0, 0, 1, 1, 0, 0]):
        g.axes[k] = float(v)
    g.omega, g.dt, g.sample_dt = 2 * math.pi / 16.0, 0.5, 3.0
    g.nr, g.nel, g.naz = shape
    g.r0, g.dr, g.daz, g.del_ = 2.0, 90.0 / g.nr, 2.0, 2.0
    g.az0, g.el0 = -2.0 * (g.naz // 2), -2.0 * (g.nel // 2)
    z = (rng.standard_normal((M, C)) + 1j * rng.standard_normal((M, C))).astype(np.complex64)

    class Array:
        elem_pos, weights = (tx + rng.uniform(-20, 20, (C, 3))).astype(np.float32), rng.uniform(0.3, 1.0, C)
        tx_pos = (tx + rng.uniform(-1, 1, (ntx, 3)) * [0.01, 20, 20]).astype(np.float32)
        tx_amp = rng.uniform(0.5, 1.5, ntx)
    return Array, z, g


@pytest.mark.parametrize("C,ntx,shape", [(1, 1, (1, 1, 1)), (1, 33, (9, 5, 7)), (4, 4, (40, 21, 31)), (9, 32, (16, 8, 1)),
                                         (33, 1, (7, 9, 11)), (65, 65, (30, 20, 17))])
def test_pairs_agree_with_the_fp64_sums(C, ntx, shape):
    array, z, g = _case(C, ntx, shape, C + ntx)
    got = RadarMonitor.backproject(array, z, g)
    array.tx_amp = array.tx_amp * 2.0 ** -100
    ref = RadarMonitor.backproject(array, z, g)
    assert np.array_equal(got < 0, ref < 0) and (ref >= 0).any()
    np.testing.assert_allclose(got, ref, rtol=2.5e-8, atol=1e-9 * ref.max())


def test_samples_that_are_not_finite_reach_the_same_points():
    array, z, g = _case(5, 3, (20, 9, 9), 3)
    z[20, 1], z[30, 4] = np.nan, np.inf
    got = RadarMonitor.backproject(array, z, g)
    array.tx_amp = array.tx_amp * 2.0 ** -100
    ref = RadarMonitor.backproject(array, z, g)
    assert np.isnan(ref).any() and np.array_equal(np.isnan(got), np.isnan(ref))
    fin = np.isfinite(ref)
    assert np.array_equal(np.isfinite(got), fin)
    np.testing.assert_allclose(got[fin], ref[fin], rtol=2.5e-8, atol=1e-9 * ref[fin].max())
