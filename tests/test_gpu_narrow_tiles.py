"""The 32 x 16 tiles of the pair kernel (two rows a warp), which the automatic tiling takes where 64 x 8 tiles
would cover more cells: grids whose rows end in, at and after a tile, partial tile rows, one to a few planes
per chunk, 16- and 32-bit class indices, and stacks of scenes before and after a compaction that changes the choice."""
import numpy as np
import pytest

import oracle
from em_lab_gb300 import SimulationGrid, abi, configs
from em_lab_gb300.grid import SceneStack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,pml", [((65, 31, 20), 6), ((80, 16, 41), 4), ((96, 33, 18), 5), ((90, 47, 17), 4),
                                      ((160, 48, 64), 12), ((81, 30, 150), 3)])
def test_narrow_tiles_bit_exact(size, pml):
    sc = configs.random_scene(size=size, pml=pml, seed=sum(size), sources=2)
    rng = np.random.default_rng(7)
    comps = [rng.standard_normal(size[::-1]).astype(np.float32) for _ in range(6)]
    g, o = SimulationGrid(sc.grid), oracle.Oracle(sc.grid, "f32")
    for s in (g, o):
        oracle.load_scene(s, sc)
        s.write_components(comps)
        s.step(21)
    g.synchronize(60000)
    for c, (a, b) in enumerate(zip(g.read_components(), o.read_components())):
        assert np.array_equal(a, b), (c, int((a != b).sum()))


def test_narrow_tiles_with_32_bit_classes():
    size = (80, 45, 40)  # every cell a material of its own: more than 65536 edge classes
    rng = np.random.default_rng(3)
    cfg = abi.GridConfig(size, courant=0.5, pml_thickness=5)
    sigma = (10.0 ** rng.uniform(-3, 0, size[::-1])).astype(np.float32)
    eps = rng.uniform(1.0, 9.0, size[::-1]).astype(np.float32)
    comps = [rng.standard_normal(size[::-1]).astype(np.float32) for _ in range(6)]
    g, o = SimulationGrid(cfg), oracle.Oracle(cfg, "f32")
    for s in (g, o):
        s.upload_materials(sigma, eps)
        s.write_components(comps)
        s.step(5)
    for c, (a, b) in enumerate(zip(g.read_components(), o.read_components())):
        assert np.array_equal(a, b), (c, int((a != b).sum()))


def test_narrow_tiles_in_stacks():
    dims = [(80, 64, 18), (96, 33, 20), (48, 48, 19), (64, 56, 21)]
    scenes = [configs.random_scene(size=d, seed=40 + k, pml=4) for k, d in enumerate(dims)]
    st = SceneStack(scenes[0].grid, scene_dims=dims)
    for k, sc in enumerate(scenes):
        st.upload_scene_materials(k, sc.materials.sigma, sc.materials.epsilon_r, sc.edges, sc.wires)
    st.set_scene_sources([sc.sources for sc in scenes])
    st.step(15)
    alone = []
    for k, sc in enumerate(scenes):
        o = oracle.Oracle(sc.grid, "f32")
        oracle.load_scene(o, sc)
        o.step(15)
        alone.append(o)
    comps = st.read_components()
    for k, o in enumerate(alone):
        for a, b in zip(st.scene_components(k, comps), o.read_components()):
            assert np.array_equal(a, b), k
    st.compact([False, False, True, True])  # 64 x 8 tiles fit what is left
    st.step(9)
    comps = st.read_components()
    for k, o in enumerate(alone[2:]):
        o.step(9)
        for a, b in zip(st.scene_components(k, comps), o.read_components()):
            assert np.array_equal(a, b), k
