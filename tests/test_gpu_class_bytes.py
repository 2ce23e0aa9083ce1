"""The width of the class index that the solver pass reads, which the roofline counts: 2 bytes, and 4 with more
than 65536 classes."""
import numpy as np
import pytest

from em_lab_gb300 import SimulationGrid, abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("own,width", [(False, 2), (True, 4)])
def test_class_bytes(own, width):
    size = (70, 45, 41)
    rng = np.random.default_rng(1)
    eps = rng.uniform(1.0, 9.0, size[::-1]).astype(np.float32) if own else np.full(size[::-1], 2.0, np.float32)
    g = SimulationGrid(abi.GridConfig(size, courant=0.5, pml_thickness=5))
    assert g.class_bytes() == 2
    g.upload_materials(np.zeros(size[::-1], np.float32), eps)
    assert g.class_bytes() == width
    g.close()
