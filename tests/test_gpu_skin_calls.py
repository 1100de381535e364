"""Learned skin (GPU): the decisions of its batches of steps, their cost in
host round trips, and the windows of its policy."""
import numpy as np
import pytest

from test_gpu_near import _scene

pytestmark = pytest.mark.gpu


def _engine(src, form=0):
    from rockable_gb300 import scenes
    from rockable_gb300.abi import GpuScene
    g = GpuScene(form=form)
    g.upload_shapes(src["shape_tables"])
    g.upload_bodies(src["bodies"], src["n_driven"])
    scenes.set_scene_params(g, src)
    if src.get("entries") is not None:
        g.upload_entries(src["entries"])
    return g


@pytest.mark.parametrize("form", [0, 1])
def test_batches_match_the_host_decided_path(gpu_lib, form):
    """With the skin and the interval pinned the refreshes depend on the state
    alone: batches decided on the device (as a graph, and launched one by one)
    and the path that decides on the host after every step, which profiled
    steps take, make the same refreshes and leave the same bits."""
    from rockable_gb300 import scenes
    scene = scenes.column_collapse(n=2000, nshapes=64, semi=(0.0025, 0.0075))
    gs = scenes.settle(scene, steps=1500)
    src = scenes.scene_from_gpu(scene, gs)
    gs.close()
    skin = 0.1 * scene["dVerlet"]
    out = {}
    for arm in ("host", "launched", "graph"):
        g = _engine(src, form)
        g.set_skin(use_mlp=False, skin_min=skin, skin_max=skin, interval_min=45, interval_max=45)
        g.set_graphs(arm == "graph")
        g.set_profiling(arm == "host")
        for n in (7, 100, 33, 160):
            g.step(n)
        out[arm] = (g.bodies(), g.skin_stats(), g.entries())
        g.close()
    b0, s0, e0 = out.pop("host")
    assert s0["rebuilds"] >= 3 and s0["partial"] + s0["forced"] >= 1
    for arm, (b, s, e) in out.items():
        for k in ("rebuilds", "forced", "scheduled", "partial", "partial_bodies"):
            assert s0[k] == s[k], (arm, k, s0[k], s[k])
        for k in b0:
            assert np.array_equal(b0[k], b[k]), (arm, k)
        for k in ("i", "j", "type", "isub", "jsub", "fn", "ft"):
            assert np.array_equal(e0[k], e[k]), (arm, k)


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("kind", ["free flight", "recorded"])
def test_steps_without_a_near_set_run_in_batches(gpu_lib, kind, form):
    """An empty list (grains in free flight) and recorded contact geometry
    have no near set: their steps share host round trips all the same."""
    from rockable_gb300 import scenes
    if kind == "free flight":
        src = scenes.drop_bodies(scenes.sphero_cube_box(4), range(6))
        src["bodies"]["pos"] *= 2.0
    else:
        src = _scene("avalanche", 0.0)
    src["gravity"] = (0.0, 0.0, 0.0)
    a, b = _engine(src, form), _engine(src, form)
    for g, graphs in ((a, True), (b, False)):
        g.set_skin(use_mlp=False, skin_min=src["dVerlet"], skin_max=src["dVerlet"], interval_min=4000,
                   interval_max=4000)
        g.set_record_geometry(kind == "recorded")
        g.set_graphs(graphs)
    assert (a.n_entries == 0) == (kind == "free flight")
    r0 = a.graph_stats()["replays"]
    for k in (128, 3, 1, 40):
        a.step(k)
        for _ in range(k):
            b.step(1)
    assert a.graph_stats()["replays"] - r0 <= 20
    x, y = a.bodies(), b.bodies()
    for k in x:
        assert np.array_equal(x[k], y[k]), k
    a.close()
    b.close()


def test_a_new_skin_does_not_pay_for_earlier_steps(gpu_lib):
    """Near sets that a context made before rk_set_skin are not charged to the
    policy's first window: the same state in a new context gets the same skin."""
    from rockable_gb300 import scenes
    sc = scenes.column_collapse(n=3000, nshapes=24, tries=2, law="Default")
    nd, n = sc["n_driven"], len(sc["bodies"]["mass"])
    sc["bodies"]["vel"][nd:] = np.random.default_rng(1).normal(0.0, 3.0, (n - nd, 3))
    sc["gravity"] = (0.0, 0.0, 0.0)
    sc["interVerlet"] = 40 * sc["dt"]
    a = _engine(sc)
    a.update_nl()
    a.step(1500)
    src = scenes.scene_from_gpu(sc, a)
    b = _engine(src)
    d = sc["dVerlet"]
    skins = []
    for g in (a, b):
        g.set_skin(use_mlp=False, skin_min=0.25 * d, skin_max=d, interval_min=20, interval_max=1000)
        while g.skin_stats()["rebuilds"] == 0:
            g.step(20)
        skins.append(g.skin_stats()["skin"] / d)
        g.close()
    assert skins[0] == skins[1], skins


@pytest.mark.parametrize("use_mlp,steps", [(False, 6000), (True, 14000)])
def test_windows_reach_interval_max(gpu_lib, use_mlp, steps):
    """Grains at rest: nothing uses up the skin, so the refreshes become as
    rare as the caller allows (with the network, once it has learnt)."""
    src = _scene("default", 0.0)
    src["bodies"]["pos"][src["n_driven"]:, 2] += 0.002  # (off the floor)
    src["gravity"] = (0.0, 0.0, 0.0)
    g = _engine(src)
    d = src["dVerlet"]
    g.set_skin(use_mlp=use_mlp, skin_min=0.1 * d, skin_max=d, interval_min=2, interval_max=2000)
    g.step(steps)
    st = g.skin_stats()
    assert st["interval"] == 2000, st
    g.close()
