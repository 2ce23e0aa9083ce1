"""The far-field pattern sums at the edges of their strips, row blocks and direction blocks: boxes whose
faces end in and at a strip of four columns or a block of 32 rows, one direction up to a few blocks
of 256. Tolerance: 2e-5 of the pattern's maximum (the float phases of the restatement, about 2e-6 at
the box's corners, in every term of both sums)."""
import numpy as np
import pytest

import oracle
from em_lab_gb300 import SimulationGrid, abi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [((6, 6, 6), (10, 11, 12)), ((5, 6, 5), (36, 13, 9)), ((5, 5, 5), (8, 37, 40)),
                                 ((7, 5, 6), (39, 36, 37))])
@pytest.mark.parametrize("n_dirs", [1, 127, 257, 600])
def test_pattern_edges_match_the_restatement(box, n_dirs):
    grid = abi.GridConfig((46, 44, 47), courant=0.5, pml_thickness=4)
    rng = np.random.default_rng(sum(box[1]) + n_dirs)
    comps = [rng.standard_normal((47, 44, 46)).astype(np.float32) for _ in range(6)]
    lo, hi = box[0], tuple(max(h, l + 4) for l, h in zip(*box))
    g, o = SimulationGrid(grid), oracle.Oracle(grid, "f32")
    for s in (g, o):
        s.write_components(comps)
        assert s.ntff_configure(lo, hi, 11.0, 4.0) == (tuple(lo), tuple(hi))
        s.step(6)
    dirs = configs.fibonacci_directions(n_dirs)
    got, want = g.ntff_evaluate(dirs), o.ntff_evaluate(dirs)
    assert np.abs(got[:, 0] - want[:, 0]).max() <= 2e-5 * want[:, 0].max()
    assert abs(got[0, 1] - want[0, 1]) <= 2e-5 * np.abs(want[0, 1]) + 1e-6 * want[:, 0].max()
    assert not got[1:, 1].any()


@pytest.mark.parametrize("rows_y,rows_z", [(62, 66), (63, 65), (64, 64), (65, 63)])
def test_mirrored_rows_across_a_row_block(rows_y, rows_z):
    """Faces whose rows and their mirrors just fit, fill and pass a block of 32, with and without a middle row."""
    grid = abi.GridConfig((24, 78, 80), courant=0.5, pml_thickness=4)
    rng = np.random.default_rng(rows_y)
    comps = [rng.standard_normal((80, 78, 24)).astype(np.float32) for _ in range(6)]
    lo, hi = (6, 5, 5), (17, 4 + rows_y, 4 + rows_z)
    g, o = SimulationGrid(grid), oracle.Oracle(grid, "f32")
    for s in (g, o):
        s.write_components(comps)
        assert s.ntff_configure(lo, hi, 13.0, 4.0) == (lo, hi)
        s.step(4)
    dirs = configs.fibonacci_directions(70)
    got, want = g.ntff_evaluate(dirs), o.ntff_evaluate(dirs)
    assert np.abs(got[:, 0] - want[:, 0]).max() <= 2e-5 * want[:, 0].max()
