"""The tensor-core pattern kernel with its bounded waits made to run out: it ends, the host reports
EMLAB_ERR_TIMEOUT, and with the normal bound restored the same grid's pattern is what it was. With a few
polls allowed some lanes and roles still see their barriers complete while others give up; whichever way
that goes the call either fails or is right. Two items a CTA and more, faces with and without the folded
middle row, one face of two segments."""
import numpy as np
import pytest

from em_lab_gb300 import EmlabError, SimulationGrid, abi, configs, grid as gridmod

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,box", [((46, 44, 47), [5, 6, 5, 36, 13, 9]), ((24, 24, 372), [7, 6, 10, 15, 15, 353])])
@pytest.mark.parametrize("polls", [0, 1, 4, 64])
def test_waits_that_run_out_report_timeout(size, box, polls):
    g = SimulationGrid(abi.GridConfig(size, courant=0.5, pml_thickness=4))
    rng = np.random.default_rng(polls)
    g.write_components([rng.standard_normal(size[::-1]).astype(np.float32) for _ in range(6)])
    g.ntff_dft_configure_boxes([box], [9.0, 14.5, 40.0])
    g.step(20)
    dirs = configs.fibonacci_directions(128 * 160)
    want = g.ntff_dft_pattern_gemm(0, dirs)
    for _ in range(3):
        try:
            gridmod.debug_set_wait_limit(polls)
            got = g.ntff_dft_pattern_gemm(0, dirs)
        except EmlabError as e:
            assert e.code == abi.EMLAB_ERR_TIMEOUT
        else:
            assert polls > 0
            np.testing.assert_array_equal(got, want)
        finally:
            gridmod.debug_set_wait_limit(gridmod.WAIT_POLLS_DEFAULT)
        g.synchronize(60000)
        np.testing.assert_array_equal(g.ntff_dft_pattern_gemm(0, dirs), want)
    g.close()
