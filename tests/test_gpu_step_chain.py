"""The kernels of a step launched as a chain (blocks start beside the kernel before) against the same
launches in full stream order, which a timed step takes: fields and every monitor agree bit for bit, with
and without sources (whose launch decides how the monitors behind it are chained), for each solver path."""
import numpy as np
import pytest

import oracle
from em_lab_gb300 import SimulationGrid, abi, configs
from em_lab_gb300.scene import SourceDesc

pytestmark = pytest.mark.gpu


def _run(timed, sources, path, size, steps=23):
    sc = configs.random_scene(size=size, pml=5, seed=3, sources=2)
    rng = np.random.default_rng(1)
    g = SimulationGrid(sc.grid)
    if path == "cpml":
        g.set_cpml((1.2, 3.0, 0.05, 3.0))
    oracle.load_scene(g, sc)
    desc = list(sc.sources) if sources else []
    if sources == "many":  # every interior cell
        desc.append(SourceDesc(center=tuple(v * 0.5 for v in size), half_extent=tuple(v * 0.5 for v in size),
                               amplitude=1e-3, wavelength=12.0))
    g.set_sources(desc)
    g.write_components([rng.standard_normal(size[::-1]).astype(np.float32) for _ in range(6)])
    if path == "split":
        g.set_kernel(abi.KERNEL_SPLIT)
    elif path != "cpml":
        g.set_tiling(path)
    g.ports_configure([sc.ports[0].to_c()], 12.0, 4.0, True, 64)
    g.ntff_configure((7, 7, 7), tuple(v - 8 for v in size), 12.0)
    g.ntff_dft_configure((7, 7, 7), tuple(v - 8 for v in size), [9.0, 15.0])
    g.lines_configure([[0, 2, 0, 0]], [[9, 9, 9, 2], [9, 9, 10, 2]], [1.0, 0.5], 12.0)
    g.set_timing(timed)
    g.step(steps)
    g.step(2)
    g.synchronize(60000)
    ph, now = g.lines_read()
    return [*g.read_components(), g.ports_phasors(), g.ports_series(), g.ntff_phasors(), g.ntff_dft_read(), ph, now]


@pytest.mark.parametrize("sources", [False, True, "many"])
@pytest.mark.parametrize("path,size", [(32, (64, 40, 36)), (64, (130, 61, 30)), (8, (40, 40, 40)), (16, (40, 33, 30)),
                                       ("split", (48, 40, 33)), ("cpml", (48, 40, 33))])
def test_chained_steps_match_stream_order(path, size, sources):
    for a, b in zip(_run(False, sources, path, size), _run(True, sources, path, size)):
        assert np.array_equal(a, b)
