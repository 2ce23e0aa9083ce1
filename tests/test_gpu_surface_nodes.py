"""Sampling of the far-field surface with x faces at every position within an aligned pair and quad of cells,
rows of a face shorter than, equal to and longer than a warp, and the smallest box: the accumulated phasors
are bit-identical to the oracle's and the DFT's sums (FP32 in a block, in another order) within 1e-4 of the
largest of a component, some hundred times the rounding of the 20 samples summed."""
import numpy as np
import pytest

import oracle
from em_lab_gb300 import SimulationGrid, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi", [((6, 7, 8), (11, 40, 13)), ((7, 6, 6), (20, 37, 33)), ((8, 8, 7), (41, 41, 25)),
                                   ((9, 20, 9), (34, 24, 13)), ((12, 11, 10), (16, 15, 14))])
def test_x_faces(lo, hi):
    size = (49, 48, 40)
    sc = configs.random_scene(size=size, pml=4, seed=11, sources=2)
    rng = np.random.default_rng(2)
    comps = [rng.standard_normal(size[::-1]).astype(np.float32) for _ in range(6)]
    res = []
    for t in (SimulationGrid(sc.grid), oracle.Oracle(sc.grid, "f32")):
        oracle.load_scene(t, sc)
        t.write_components(comps)
        box = t.ntff_configure(lo, hi, 12.0)
        t.ntff_dft_configure(lo, hi, [9.0, 15.0])
        t.step(20)
        res.append((box, t.ntff_phasors(), t.ntff_dft_read()))
    assert res[0][0] == (lo, hi) and np.array_equal(res[0][1], res[1][1])
    got, ref = res[0][2], res[1][2]
    assert np.abs(ref).max() > 0 and np.abs(got - ref).max() <= 1e-4 * np.abs(ref).max()
