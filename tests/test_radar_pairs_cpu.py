"""The radar kernel's pairs of FP32 on the host (the kernel's own functions): the bounds that it decides by hold.
Against the reference's formulas in FP64 and in extended precision, for arrays of 1 to 64 elements a tenth of a
wavelength to five wavelengths apart, 2 to 3000 cells away, with records from fine to coarse: the transmit delay is
within its bound of both; a sample index called certain is the FP64 one; and the FP32 interpolation weight that FP64
takes lies between the weights rounded from the ends of the interval. Nearly every
point in front of an array of up to half a wavelength's spacing is decided without FP64."""
import ctypes as C
import math

import numpy as np
import pytest

from em_lab_gb300 import abi
from em_lab_gb300.grid import EmlabError, _check, load_library

f32, LD = np.float32, np.longdouble


@pytest.fixture(scope="module")
def lib():
    try:
        lib = load_library()
    except EmlabError as e:
        pytest.skip(str(e))
    return lib


def length(v):
    """RadarMonitor's FP32 length, rounding by rounding."""
    return np.sqrt((v[..., 0] * v[..., 0] + v[..., 1] * v[..., 1]) + v[..., 2] * v[..., 2])


def tx_delay(points, tx, boresight, pos, amp, w, real):
    """RadarMonitor::txDelay in `real`, summed element by element, and |sum| / sum of magnitudes."""
    s = [np.zeros(len(points), real) for _ in range(5)]
    for q, a0 in zip(pos, amp):
        v = points - q
        d = np.maximum(length(v).astype(real), real(0.5))
        dot = (v[:, 0] * boresight[0] + v[:, 1] * boresight[1]) + v[:, 2] * boresight[2]
        a = real(a0) * np.maximum(dot.astype(real) / d, real(0)) / d
        tr, ti = a * np.cos(-real(w) * d), a * np.sin(-real(w) * d)
        for acc, term in zip(s, (tr, ti, d * tr, d * ti, a)):
            acc += term
    power = s[0] * s[0] + s[1] * s[1]
    return (s[2] * s[0] + s[3] * s[1]) / power, np.sqrt(power) / s[4]


def evaluate(lib, g, points, elems, pos, amp):
    n, c = len(points), len(elems)
    delays, samples = np.zeros((n, 2)), np.zeros((n, c, 5))
    fp, dp = C.POINTER(C.c_float), C.POINTER(C.c_double)
    arr = [np.ascontiguousarray(a, f32) for a in (points, elems, pos)]
    amp = np.ascontiguousarray(amp, np.float64)
    _check(lib.emlab_debug_radar_delays(C.byref(g), arr[0].ctypes.data_as(fp), n, arr[1].ctypes.data_as(fp), c,
                                        arr[2].ctypes.data_as(fp), amp.ctypes.data_as(dp), len(amp),
                                        delays.ctypes.data_as(dp), samples.ctypes.data_as(dp)))
    return delays, samples


@pytest.mark.parametrize("near,far", [(2.0, 30.0), (30.0, 300.0), (300.0, 3000.0)])
@pytest.mark.parametrize("spacing", [0.1, 0.5, 2.0, 5.0])
@pytest.mark.parametrize("side", [1, 2, 5, 8])
def test_bounds_hold(lib, side, spacing, near, far):
    rng = np.random.default_rng([side, int(10 * spacing), int(far)])
    wl = float(np.exp(rng.uniform(math.log(6.0), math.log(60.0))))
    w, dt, sdt = 2 * math.pi / wl, float(rng.uniform(0.2, 0.57)), float(np.exp(rng.uniform(math.log(0.6), math.log(8.0))))
    tx = rng.uniform(20, 200, 3).astype(f32)
    k = np.arange(side * side)
    yz = np.stack([0 * k, k % side - (side - 1) / 2, k // side - (side - 1) / 2], 1) * spacing * wl
    pos = (tx + yz + rng.uniform(-0.01, 0.01, yz.shape)).astype(f32)
    elems = (tx + yz[rng.permutation(len(yz))[:9]]).astype(f32)
    amp = rng.uniform(0.3, 1.5, len(pos))
    boresight = np.array([1, 0, 0], f32)
    g = abi.RadarGeometry()
    for a in range(3):
        g.tx[a], g.axes[6 + a] = float(tx[a]), float(boresight[a])
    g.omega, g.dt, g.sample_dt = w, dt, sdt
    n = 4000
    dirs = rng.standard_normal((n, 3))
    dirs[:, 0] = np.abs(dirs[:, 0]) + 0.2
    dirs /= np.linalg.norm(dirs, axis=1)[:, None]
    points = (tx + dirs * np.exp(rng.uniform(math.log(near), math.log(far), n))[:, None]).astype(f32)
    delays, samples = evaluate(lib, g, points, elems, pos, amp)
    t, err = delays.T
    decided = err >= 0
    t64, ratio = tx_delay(points, tx, boresight, pos, amp, w, np.float64)
    tld, _ = tx_delay(points, tx, boresight, pos, amp, w, LD)
    assert (decided == (ratio > 0.01))[np.abs(ratio - 0.01) > 1e-5].all()
    assert (np.abs(t - t64)[decided] <= err[decided]).all()
    assert (np.abs(t.astype(LD) - tld)[decided] <= err[decided]).all()
    for i, e in enumerate(elems):
        clear, m, f, below, above = samples[:, i].T
        d = length(points - e)
        sure = clear == 1
        assert not sure[~decided].any()
        for real, total in ((np.float64, t64), (LD, tld)):
            s = (total + d.astype(real) + real(0.5) * real(dt)) / real(sdt)
            m0 = np.floor(s)
            w0 = (s - m0).astype(f32)
            assert (m[sure] == m0[sure]).all()
            assert ((below <= w0) & (w0 <= above))[sure].all()
            assert ((f == w0) | (below != above))[sure].all()
    if spacing <= 0.5:
        assert decided.mean() > 0.9


def test_amplitudes_and_positions_beyond_the_pairs_go_to_fp64(lib):
    g = abi.RadarGeometry()
    for a, (t, b) in enumerate(zip((50.0, 50.0, 50.0), (1.0, 0.0, 0.0))):
        g.tx[a], g.axes[6 + a] = t, b
    g.omega, g.dt, g.sample_dt = 0.4, 0.5, 3.0
    tx = np.full((2, 3), 50.0, f32)
    ahead, behind = np.array([[90.0, 50.0, 50.0]], f32), np.array([[10.0, 50.0, 50.0]], f32)
    for points, amp in ((ahead, [1e-30, 1e-30]), (ahead, [1e30, 1e30]), (ahead, [np.nan, 1.0]), (ahead, [np.inf, 1.0]),
                        (ahead, [1.0, -1.0]), (behind, [1.0, 1.0]), (ahead * f32(1e6), [1.0, 1.0]),
                        (np.array([[np.nan, 50.0, 50.0]], f32), [1.0, 1.0])):
        delays, samples = evaluate(lib, g, points, tx, tx, np.array(amp))
        assert delays[0, 1] < 0 and not samples[0, :, 0].any()
    delays, samples = evaluate(lib, g, ahead, tx, tx, np.array([1.0, 1.0]))
    assert delays[0, 0] == pytest.approx(40.0, rel=1e-14) and delays[0, 1] >= 0
    for sdt in (0.0, np.nan, np.inf, 1e-9):  # positions that no record has
        g.sample_dt = sdt
        _, samples = evaluate(lib, g, ahead, tx, tx, np.array([1.0, 1.0]))
        assert not samples[0, :, 0].any()
