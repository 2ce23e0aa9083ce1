"""The middle row of a face with an odd number of rows is its own mirror: its sum is its field and its difference
zero, so it takes no part of the other quadrature. Seen by interference. The far-field DFT gets two samples: a
single Bz cell in the middle row of the low x face, then two Ey cells on the z faces, all exact in FP32 (the step is
undone on the way in). At six steps a period the H sample at 3/2 steps and the E sample at three are a quarter period
apart, and both phases exact. Along z with |r| = rho the x face gives N_y = j F c and the z faces
(rho x L)_y = T, real: |j F c - T|^2 is the same for T and -T. What a wrong difference adds, the sine of
position zero (some 1e-6 after 31 complex products), is in phase with T and is not.
Tolerance 2^-22: the z faces' own quadrature cancels to 2^-24 of half of F and meets F twice times rho <= 3/2,
three roundings of the squares and their sum."""
import numpy as np
import pytest

from em_lab_gb300 import SimulationGrid, abi

pytestmark = pytest.mark.gpu
DT = 0.5


def diff(a, axis, step):
    """a(i + 1) - a(i) (step 1) or a(i) - a(i - 1) (step -1) along x, y, z = 0, 1, 2; zero beyond the array."""
    ax = 2 - axis
    pad = [(0, 0)] * 3
    pad[ax] = (0, 1) if step > 0 else (1, 0)
    return np.diff(np.pad(a, pad), axis=ax)


def curl(f, step):
    return [diff(f[(c + 2) % 3], (c + 1) % 3, step) - diff(f[(c + 1) % 3], (c + 2) % 3, step) for c in range(3)]


def write_for_step(g, E, B):
    """Fields from which one step of the vacuum makes E and B."""
    E0 = [e - DT * c for e, c in zip(E, curl(B, -1))]
    B0 = [b + DT * c for b, c in zip(B, curl(E0, 1))]
    g.write_components([a.astype(np.float32) for a in E0 + B0])
    g.step(1)
    for got, want in zip(g.read_components(), E + B):
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("rows", [61, 63, 127])
def test_the_middle_row_has_no_difference(rows):
    nx, ny, nz = 34, 40, rows + 19
    lo, hi = (10, 8, 9), (20, 29, 8 + rows)
    dirs = np.zeros((512, 4), np.float32)
    dirs[:, 2] = np.linspace(0.05, 1.5, 512)
    power = []
    for sign in (1.0, -1.0):
        zero = [np.zeros((nz, ny, nx)) for _ in range(3)]
        E, B = [z.copy() for z in zero], [z.copy() for z in zero]
        B[2][lo[2] + rows // 2, 18, lo[0]] = 1.0
        E[1][hi[2], 18, 15], E[1][lo[2], 18, 15] = 0.25 * sign, -0.25 * sign
        g = SimulationGrid(abi.GridConfig((nx, ny, nz), courant=DT, pml_thickness=4))
        g.step(1)
        assert g.ntff_dft_configure(lo, hi, [6 * DT]) == (lo, hi)
        g.ntff_dft_engine(abi.DFT_CUDA_CORES)
        write_for_step(g, zero, B)
        write_for_step(g, E, zero)
        x = g.ntff_dft_read()[0]
        assert not x[:, :3, 1].any() and np.abs(x[:, 3:, 0]).max() < 1e-16 and np.abs(x[:, 3:, 1]).max() == 0.25
        power.append(g.ntff_dft_evaluate_all(dirs)[0, :, 0].astype(np.float64))
        g.close()
    total = power[0] + power[1]
    assert (total > 0).all()
    assert (np.abs(power[0] - power[1]) / total).max() <= 2.0 ** -22
