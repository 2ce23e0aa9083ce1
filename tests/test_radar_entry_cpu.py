"""emlab_radar_backproject with sizes that cannot be had returns an error code: nothing is read from the arrays, no
exception leaves the C entry (one would end the process, so the call runs in a process of its own)."""
import subprocess
import sys

import pytest

CALL = """
import ctypes as C
import numpy as np
from em_lab_gb300 import abi
from em_lab_gb300.grid import load_library
lib = load_library()
g = abi.RadarGeometry()
g.nr = g.nel = g.naz = 1
f, d = (C.c_float * 4)(), (C.c_double * 4)()
rc = lib.emlab_radar_backproject(C.byref(g), f, {M}, {C}, f, d, f, d, 1, d)
print(rc, abi.EMLAB_ERR_OOM)
"""


@pytest.mark.parametrize("M,C", [(2 ** 31 - 1, 2 ** 29), (2 ** 31 - 1, 2 ** 31 - 1), (2 ** 31 - 1, 2 ** 28)])
def test_sizes_that_cannot_be_had_are_an_error(M, C):
    from em_lab_gb300.grid import EmlabError, load_library
    try:
        load_library()
    except EmlabError as e:
        pytest.skip(str(e))
    p = subprocess.run([sys.executable, "-c", CALL.format(M=M, C=C)], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, p.stderr[-500:]
    rc, oom = map(int, p.stdout.split())
    assert rc == oom
