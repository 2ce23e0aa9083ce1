"""The pair kernel at the edges of its tiles and chunks: rows that end in, at and after a 64-cell tile,
partial tile rows, grids of one to a few planes per chunk, and warps whose 64 cells mix vacuum,
materials, thin wires and absorber."""
import numpy as np
import pytest

import oracle
from em_lab_gb300 import SimulationGrid, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [32, 64, 128])
@pytest.mark.parametrize("size,pml", [((63, 21, 20), 6), ((64, 16, 41), 4), ((65, 23, 18), 5), ((129, 50, 17), 4),
                                      ((192, 33, 64), 12), ((16, 16, 150), 3)])
def test_tile_and_chunk_edges_bit_exact(rows, size, pml):
    sc = configs.random_scene(size=size, pml=pml, seed=sum(size), sources=2)
    rng = np.random.default_rng(7)
    comps = [rng.standard_normal(size[::-1]).astype(np.float32) for _ in range(6)]
    g, o = SimulationGrid(sc.grid), oracle.Oracle(sc.grid, "f32")
    for s in (g, o):
        oracle.load_scene(s, sc)
        s.write_components(comps)
    g.set_tiling(rows)
    g.step(21)
    g.synchronize(60000)
    o.step(21)
    for c, (a, b) in enumerate(zip(g.read_components(), o.read_components())):
        assert np.array_equal(a, b), (c, int((a != b).sum()))
