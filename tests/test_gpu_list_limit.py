"""A neighbour list longer than its index type is refused before anything is
touched (GPU)."""
import ctypes

import numpy as np
import pytest

from test_gpu_near import _engine, _scene

pytestmark = pytest.mark.gpu


def test_longest_list(gpu_lib):
    from rockable_gb300 import abi
    g = _engine(_scene("cubes", 0.5), 0, False)
    before = g.entries()
    assert abi.ERRORS[g.L.rk_upload_entries(g.h, ctypes.byref(abi.RkEntries(2 ** 31)))] == "RK_ERR_CAPACITY"
    after = g.entries()
    for k in before:
        assert np.array_equal(before[k], after[k]), k
    g.step(3)
    g.close()
