"""The patterns' device scratch is kept while a far-field monitor is attached and goes back with the last of them;
patterns after a new configuration are what they were."""
import numpy as np
import pytest

from em_lab_gb300 import SimulationGrid, abi, configs

pytestmark = pytest.mark.gpu
SIZE, LO, HI = (90, 84, 80), (8, 8, 8), (80, 74, 70)


def test_scratch_goes_back_with_the_last_monitor():
    import torch
    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    g = SimulationGrid(abi.GridConfig(SIZE, courant=0.5, pml_thickness=4))
    rng = np.random.default_rng(1)
    fields = [rng.standard_normal(SIZE[::-1]).astype(np.float32) for _ in range(6)]
    wl, dirs = [float(9 + k) for k in range(32)], configs.fibonacci_directions(9000)

    def patterns():
        g.reset_fields()
        g.ntff_configure(LO, HI, 12.0, 4.0)
        g.ntff_dft_configure(LO, HI, wl)
        g.write_components(fields)
        g.step(3)
        return g.ntff_evaluate(dirs), g.ntff_dft_evaluate_all(dirs), g.ntff_dft_pattern_gemm(0, dirs)

    def off(dft, one):
        if dft:
            g.ntff_dft_configure(LO, HI, [])
        if one:
            g.ntff_configure(LO, HI, 0.0)

    patterns(), off(True, True)
    bare = free()
    first = patterns()
    g.synchronize(60000)
    held = free()
    for dft, one in ((True, False), (False, True)):  # one monitor stays: so does the scratch
        off(dft, one)
        assert bare - free() > 40 << 20
        if dft:
            g.ntff_dft_configure(LO, HI, wl)
    off(True, True)
    assert abs(bare - free()) < 8 << 20 < bare - held
    for a, b in zip(first, patterns()):
        np.testing.assert_array_equal(a[..., 0], b[..., 0])
    g.close()
