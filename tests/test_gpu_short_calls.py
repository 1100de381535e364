"""Calls of one and two steps (GPU): their launches, and the same bits as
longer calls."""
import numpy as np
import pytest

from helpers import bitwise_equal
from test_gpu_near import _engine, _scene

pytestmark = pytest.mark.gpu


def test_mixed_steps_on_the_whole_list_make_one_pass_over_the_bodies(gpu_lib):
    """Drift and body frames in one launch, the two narrow passes and the two
    resultant kernels."""
    g = _engine(_scene("avalanche", 0.5), 1, False)
    g.step(1)
    assert g.last_step_timing()[1] == 5
    g.close()


@pytest.mark.parametrize("form", [0, 1])
def test_short_calls_leave_the_same_bits(gpu_lib, form):
    sc = _scene("default", 3.0)
    runs = []
    for calls in ([1] * 24, [2] * 12, [3] * 8, [24], [5, 1, 2, 4, 2, 10]):
        g = _engine(sc, form, False)
        for k in calls:
            g.step(k)
        runs.append((g.bodies(), g.entries()))
        g.close()
    for b, e in runs[1:]:
        for k in b:
            assert bitwise_equal(b[k], runs[0][0][k]), k
        for k in ("fn", "ft", "mom"):
            assert bitwise_equal(e[k], runs[0][1][k]), k
        assert np.array_equal(e["active"], runs[0][1]["active"])
