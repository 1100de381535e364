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


@pytest.mark.parametrize("speed,lasting", [(0.05, True), (60.0, False)])
def test_mixed_steps_leave_near_sets_that_do_not_last(gpu_lib, speed, lasting):
    """Grains that use up their allowance in every step: after a few calls the
    steps run on the whole list (5 launches a step instead of 6), with the same
    bits; slow grains stay on their near set.  Sets are tried again later."""
    sc = _scene("default", speed)
    nd = sc["n_driven"]
    sc["bodies"]["vrot"][nd:] = 0.0
    sc["interVerlet"] = 20 * sc["dt"]
    a, b = _engine(sc, 1, False), _engine(sc, 1, False)
    launches = []
    for _ in range(12):
        if b.step(5)["nl_updates"] == 0:
            launches.append(b.last_step_timing()[1])
        for _ in range(5):
            a.step(1)
    near, whole = 4 * 6 + 5, 5 * 5
    assert len(launches) >= 6 and launches[0] == near
    assert launches[-1] == (near if lasting else whole), launches
    x, y = a.bodies(), b.bodies()
    for k in x:
        assert bitwise_equal(x[k], y[k]), k
    a.close()
    b.close()
