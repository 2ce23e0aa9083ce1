"""The convolutional absorber's passes at the edges of their tiles: both row widths (64 and 32 cells a tile),
odd rows, rows shorter than a tile, slabs that meet, and grids deep and wide enough for chunks of several planes."""
import numpy as np
import pytest

import oracle
from em_lab_gb300 import SimulationGrid, abi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,pml,steps", [((63, 19, 21), 5, 25), ((65, 23, 18), 4, 25), ((70, 21, 33), 6, 25), ((97, 30, 20), 3, 25),
                                            ((16, 16, 16), 3, 25), ((66, 130, 150), 7, 6), ((129, 140, 131), 9, 6)])
def test_tiles_and_chunks_bit_exact(size, pml, steps):
    sc = configs.random_scene(size=size, pml=pml, seed=sum(size), sources=2)
    rng = np.random.default_rng(5)
    comps = [rng.standard_normal(size[::-1]).astype(np.float32) for _ in range(6)]
    g, o = SimulationGrid(sc.grid), oracle.Oracle(sc.grid, "f32")
    for s in (g, o):
        s.set_cpml((2.0, 3.0, 0.1, 3.0))
        oracle.load_scene(s, sc)
        s.write_components(comps)
        s.step(steps)
    for c, (a, b) in enumerate(zip(g.read_components(), o.read_components())):
        assert np.array_equal(a, b), (c, int((a != b).sum()))


def test_32_bit_classes():
    size = (70, 45, 41)  # every cell a material of its own: more than 65536 edge classes
    rng = np.random.default_rng(6)
    cfg = abi.GridConfig(size, courant=0.5, pml_thickness=5)
    sigma = (10.0 ** rng.uniform(-3, 0, size[::-1])).astype(np.float32)
    eps = rng.uniform(1.0, 9.0, size[::-1]).astype(np.float32)
    comps = [rng.standard_normal(size[::-1]).astype(np.float32) for _ in range(6)]
    g, o = SimulationGrid(cfg), oracle.Oracle(cfg, "f32")
    for s in (g, o):
        s.set_cpml((2.0, 3.0, 0.1, 3.0))
        s.upload_materials(sigma, eps)
        s.write_components(comps)
        s.step(7)
    for c, (a, b) in enumerate(zip(g.read_components(), o.read_components())):
        assert np.array_equal(a, b), (c, int((a != b).sum()))
