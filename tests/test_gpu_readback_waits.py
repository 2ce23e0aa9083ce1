"""Read-backs through the grid's pinned scratch when a wait runs out: the call whose wait ran out, and the ones after it
that find the scratch still in use, return EMLAB_ERR_TIMEOUT within the limit instead of waiting without one; once
the stream has caught up the results are right. The stream is kept busy by a bounded device sleep."""
import time

import numpy as np
import pytest

from em_lab_gb300 import EmlabError, SimulationGrid, abi, grid as gridmod

pytestmark = pytest.mark.gpu
SIZE = (40, 36, 34)


def test_calls_behind_a_busy_stream_time_out():
    import torch
    g = SimulationGrid(abi.GridConfig(SIZE, courant=0.5, pml_thickness=4))
    rng = np.random.default_rng(3)
    g.write_components([rng.standard_normal(SIZE[::-1]).astype(np.float32) for _ in range(6)])
    origins = [(5, 6, 7), (20, 20, 20)]
    planes = [abi.FluxPlane(2, 17, (8, 8), (30, 28))]
    probes, flux = g.probe_gather(origins), g.flux_planes(planes)
    with torch.cuda.stream(torch.cuda.ExternalStream(g.stream_handle())):
        torch.cuda._sleep(int(4e9))  # about two seconds of cycles: a bounded spin
    began = time.perf_counter()
    try:
        gridmod.debug_set_host_wait(50)
        for call in (lambda: g.probe_gather(origins), lambda: g.probe_gather(origins), lambda: g.flux_planes(planes)):
            with pytest.raises(EmlabError) as e:
                call()
            assert e.value.code == abi.EMLAB_ERR_TIMEOUT
    finally:
        gridmod.debug_set_host_wait(0)
    took = time.perf_counter() - began
    g.synchronize(60000)
    slept = time.perf_counter() - began
    assert took < 0.5 < slept  # three limits of 50 ms, not the stream's two seconds
    np.testing.assert_array_equal(g.probe_gather(origins), probes)
    np.testing.assert_array_equal(g.flux_planes(planes), flux)
    g.close()
