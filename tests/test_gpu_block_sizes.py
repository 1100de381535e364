"""rk_get_block_sizes reports what the steps launch (GPU)."""
import pytest

from test_gpu_near import _engine, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tuned", [False, True])
def test_reported_block_sizes_are_launched(gpu_lib, tuned):
    """A scene of 700 grains: FP64 resultants run in blocks of 128 threads
    (8 lanes per body) whatever the tuner found, the mixed form's first narrow
    pass in 128 unless it was tuned."""
    sc = _scene("avalanche", 0.05)
    for form in (0, 1):
        g = _engine(sc, form, False)
        if tuned:
            g.autotune(1)
        g.step(12)
        t = g.block_sizes()
        if form == 0:
            assert t["resultants"] == 128
        elif not tuned:
            assert t["narrow"] == 128
        assert all(v in (32, 64, 128, 256, 512) for v in t.values())
        g.close()
