"""The tensor-core pattern at the edges of its tiles: even and odd lattices (the folded middle row), faces
that end in and at a block of 32 columns or a chunk of 16 folded rows, a face of more than 320 rows (two
segments), and one direction up to just over a tile of 128. Against the FP32 sums; tolerance 1e-4 of the
pattern's maximum (operands of 16 significant bits: about 2^-17 of each product, at most twice that in the
square, with room for the largest of some thousand directions)."""
import numpy as np
import pytest

from em_lab_gb300 import SimulationGrid, abi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,box", [((46, 44, 47), [6, 6, 6, 10, 11, 12]), ((46, 44, 47), [5, 6, 5, 36, 13, 9]),
                                      ((46, 44, 76), [5, 5, 5, 37, 36, 68]), ((24, 24, 372), [7, 6, 10, 15, 15, 353])])
@pytest.mark.parametrize("n_dirs", [1, 128, 129, 700])
def test_tile_edges(size, box, n_dirs):
    g = SimulationGrid(abi.GridConfig(size, courant=0.5, pml_thickness=4))
    rng = np.random.default_rng(sum(box) + n_dirs)
    g.write_components([rng.standard_normal(size[::-1]).astype(np.float32) for _ in range(6)])
    g.ntff_dft_configure_boxes([box], [9.0, 14.5, 40.0])
    g.step(20)
    dirs = configs.fibonacci_directions(n_dirs)
    got, want = g.ntff_dft_pattern_gemm(0, dirs), g.ntff_dft_evaluate_all(dirs)
    for f in range(3):
        assert np.abs(got[f, :, 0] - want[f, :, 0]).max() <= 1e-4 * want[f, :, 0].max(), f
        assert got[f, 0, 1] == pytest.approx(want[f, 0, 1], rel=1e-4, abs=1e-6 * want[f, :, 0].max())
        assert not got[f, 1:, 1].any()
