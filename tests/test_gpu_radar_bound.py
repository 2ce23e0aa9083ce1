"""The image from pairs of FP32 against the same kernel's FP64 way (amplitudes scaled by 2^-100, which changes no FP64
delay and sends every point there): within the 2e-10 of a point's power that the kernel promises, for arrays a
tenth of a wavelength to five wavelengths apart, near and far, with fine and coarse records."""
import math

import numpy as np
import pytest

from em_lab_gb300 import abi
from em_lab_gb300.radar import RadarMonitor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spacing", [0.1, 0.5, 5.0])
@pytest.mark.parametrize("side,wl,near,far,sdt", [(1, 16.0, 2.0, 90.0, 3.0), (3, 7.3, 2.0, 40.0, 0.7), (6, 16.0, 20.0, 140.0, 1.33),
                                                  (8, 31.0, 100.0, 900.0, 5.1)])
def test_image_is_within_its_bound_of_the_fp64_sums(side, wl, near, far, sdt, spacing):
    rng = np.random.default_rng([side, int(10 * spacing)])
    n = side * side
    tx = rng.uniform(900, 1000, 3).astype(np.float32)
    yz = np.stack([np.zeros(n), np.arange(n) % side - (side - 1) / 2, np.arange(n) // side - (side - 1) / 2], 1) * spacing * wl
    g = abi.RadarGeometry()
    for k in range(3):
        g.tx[k], g.interior_min[k], g.interior_max[k] = float(tx[k]), -1e4, 1e4
    for k, v in enumerate([0, -1, 0, 0, 0, 1, 1, 0, 0]):
        g.axes[k] = float(v)
    g.omega, g.dt, g.sample_dt = 2 * math.pi / wl, 0.5, sdt
    g.nr, g.nel, g.naz = 24, 11, 17
    g.r0, g.dr, g.daz, g.del_, g.az0, g.el0 = near, (far - near) / g.nr, 3.1, 3.3, -3.1 * 8, -3.3 * 5
    M = int((2.5 * far + 40 * spacing * wl) / sdt) + 3
    z = (rng.standard_normal((M, n)) + 1j * rng.standard_normal((M, n))).astype(np.complex64)

    class Array:
        elem_pos = tx_pos = (tx + yz + rng.uniform(-0.01, 0.01, yz.shape)).astype(np.float32)
        weights, tx_amp = rng.uniform(-1.0, 1.0, n), rng.uniform(0.5, 1.5, n)
    got = RadarMonitor.backproject(Array, z, g)
    Array.tx_amp = Array.tx_amp * 2.0 ** -100
    ref = RadarMonitor.backproject(Array, z, g)
    # a wide, sparse array's mean delay may lie before the record: no echo, power 0 both ways
    assert (ref >= 0).all() and (ref > 0).mean() > 0.9
    np.testing.assert_allclose(got, ref, rtol=2e-10, atol=0)


@pytest.mark.parametrize("scale", [2.0 ** -140, 2.0 ** 130])
def test_weights_beyond_the_pairs_take_the_fp64_way(scale):
    """Weights that FP32 cannot hold: the power scales with their square, exactly for a power of two."""
    rng = np.random.default_rng(5)
    tx = np.array([50.0, 50.0, 50.0], np.float32)
    g = abi.RadarGeometry()
    for k in range(3):
        g.tx[k], g.interior_min[k], g.interior_max[k] = float(tx[k]), -1e4, 1e4
    for k, v in enumerate([0, -1, 0, 0, 0, 1, 1, 0, 0]):
        g.axes[k] = float(v)
    g.omega, g.dt, g.sample_dt = 0.4, 0.5, 3.0
    g.nr, g.nel, g.naz = 9, 5, 7
    g.r0, g.dr, g.daz, g.del_ = 10.0, 9.0, 3.0, 3.0
    z = (rng.standard_normal((99, 6)) + 1j * rng.standard_normal((99, 6))).astype(np.complex64)

    class Array:
        elem_pos = tx_pos = (tx + rng.uniform(-9, 9, (6, 3))).astype(np.float32)
        weights, tx_amp = rng.uniform(0.3, 1.0, 6), np.full(6, 2.0 ** -100)
    ref = RadarMonitor.backproject(Array, z, g)
    Array.tx_amp, Array.weights = np.ones(6), Array.weights * scale
    got = RadarMonitor.backproject(Array, z, g)
    assert (ref > 0).all()
    np.testing.assert_array_equal(got / scale / scale, ref)
