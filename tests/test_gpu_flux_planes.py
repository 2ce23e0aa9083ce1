"""Flux planes go to the GPU up to sixteen in a launch, and small read-backs through pinned scratch: a list of
planes (whole, clipped, empty and outside ones; fewer and more than a launch takes) gives the sums of its planes
measured one by one, by each of the three ways to ask for them, and probes beyond the scratch the ones within."""
import ctypes as C

import numpy as np
import pytest

import oracle
from em_lab_gb300 import SimulationGrid, abi, configs

pytestmark = pytest.mark.gpu


def _grid(size):
    sc = configs.random_scene(size=size, pml=4, seed=2, sources=1)
    g = SimulationGrid(sc.grid)
    oracle.load_scene(g, sc)
    rng = np.random.default_rng(4)
    g.write_components([rng.standard_normal(size[::-1]).astype(np.float32) for _ in range(6)])
    return g


@pytest.mark.parametrize("n", [1, 15, 16, 17, 40])
def test_planes_together_equal_planes_alone(n):
    size = (33, 47, 18)
    g = _grid(size)
    rng = np.random.default_rng(n)
    planes = []
    for i in range(n):
        axis = int(rng.integers(0, 3))
        lo, hi = rng.integers(-3, 12, 2), rng.integers(8, 60, 2)
        index = int(rng.integers(0, size[axis])) if i % 5 else [-1, size[axis]][i % 2]
        planes.append(abi.FluxPlane(axis, index, (C.c_int * 2)(*lo), (C.c_int * 2)(*(lo - 1 if i % 7 == 3 else hi))))
    alone = np.array([g.flux_planes([p])[0] for p in planes])
    assert n == 1 or alone.any()
    assert np.array_equal(g.flux_planes(planes), alone)
    assert np.array_equal(g.flux_planes_noalloc(planes), alone)
    g.analyzer_submit([], planes)
    assert np.array_equal(g.analyzer_collect()[1], alone)


def test_probes_beyond_the_scratch():
    g = _grid((24, 20, 18))
    rng = np.random.default_rng(9)
    origins = rng.integers(-2, 24, (1500, 3))  # 1.3 MB of samples; up to 1 MB goes through the scratch
    got = g.probe_gather(origins)
    assert np.array_equal(got[:40], g.probe_gather(origins[:40]))
    assert np.array_equal(got[-40:], g.probe_gather(origins[-40:]))
