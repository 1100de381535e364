"""Steps on the near set (GPU): K steps in one call (all but the last on the
near set) leave the same bits as K calls of one step (each on the whole
list), in both forms: slow and fast bodies (allowances that last for many
steps and for one), four-sided faces, each law, a wall under force control
with more than 1024 entries (summed by a block), bodies that the host moves
into contact and back between calls, and list updates in between.  (Bonds,
rupture and updates on demand: the frozen cases run through the same steps.)"""
import numpy as np
import pytest

from helpers import bitwise_equal

pytestmark = pytest.mark.gpu


def _scene(kind, speed):
    from rockable_gb300 import scenes
    rng = np.random.default_rng(11)
    if kind == "cubes":
        sc = scenes.sphero_cube_box(6)
        sc["bodies"]["pos"][6:] *= 0.7  # into touch (the walls stay)
    elif kind == "wall":
        sc = scenes.iso_compression(n=3000, nshapes=24, tries=2)
        sc["dVerlet"] *= 6.0
        sc["DVerlet"] *= 6.0
    else:
        sc = scenes.column_collapse(n=700, nshapes=24, tries=2, column=(0.16, 0.16, 1.5),
                                    law={"avalanche": "Avalanche", "default": "Default"}[kind])
    nd, n = sc["n_driven"], len(sc["bodies"]["mass"])
    size = 0.01 if kind != "cubes" else 0.001
    sc["bodies"]["vel"][nd:] = rng.normal(0, speed * size / 0.01, (n - nd, 3))
    sc["bodies"]["vrot"][nd:] = rng.normal(0, speed / 0.01, (n - nd, 3))
    sc["interVerlet"] = 40 * sc["dt"]
    return sc


def _engine(sc, form, graphs):
    from rockable_gb300 import scenes
    from rockable_gb300.abi import GpuScene
    g = GpuScene(form=form)
    g.upload_shapes(sc["shape_tables"])
    g.upload_bodies(sc["bodies"], sc["n_driven"])
    scenes.set_scene_params(g, sc)
    g.update_nl()
    g.set_graphs(graphs)
    return g


def _same(a, b, form):
    x, y = a.bodies(), b.bodies()
    for k in x:
        assert bitwise_equal(x[k], y[k]), k
    e, f = a.entries(), b.entries()
    for k in ["i", "j", "type", "isub", "jsub", "active"]:
        assert np.array_equal(e[k], f[k]), k
    # (the mixed form keeps an estimate of a separated entry's dn, of which only the sign is used)
    for k in ["fn", "ft", "mom"] + (["dn"] if form == 0 else []):
        assert bitwise_equal(e[k], f[k]), k
    return e


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("kind,speed", [("avalanche", 0.05), ("default", 3.0), ("cubes", 0.5), ("wall", 0.3)])
def test_near_set_steps_equal_whole_list_steps(gpu_lib, form, kind, speed):
    sc = _scene(kind, speed)
    a, b = _engine(sc, form, False), _engine(sc, form, True)
    if kind == "wall":
        e = a.entries()
        assert max(np.sum((e["i"] == w) | (e["j"] == w)) for w in (1, 3, 5)) > 1024
    nd = sc["n_driven"]
    shift = np.zeros((a.n, 3))
    shift[nd::2, 2] = 2e-5 if kind != "cubes" else 2e-6  # half of the grains into their neighbours
    seen = 0
    for k in [1, 2, 37, 60]:
        for _ in range(k):
            a.step(1)
        b.step(k)
        seen = max(seen, int(_same(a, b, form)["active"].sum()))
        # the host pushes grains together for one step, and puts them back
        back = a.bodies()["pos"]
        for g, steps in ((a, 1), (b, 1)):
            g.upload_kinematics(pos=np.ascontiguousarray(back + shift))
            g.step(steps)
        for g in (a, b):
            g.upload_kinematics(pos=np.ascontiguousarray(back))
    a.step(1)
    a.step(1)
    b.step(2)
    _same(a, b, form)
    assert seen > 20
    a.close()
    b.close()


def test_big_body_resultant_is_the_serial_sum(gpu_lib):
    """The block that sums a body of more than 1024 entries (whole list and
    near set) adds the contributions in the serial order, bit for bit: the
    components that start from zero of the servo walls' resultants."""
    sc = _scene("wall", 0.3)
    g = _engine(sc, 0, False)
    for steps in (1, 6):
        g.step(steps)
        e, f = g.entries(), g.contributions()
        b = g.bodies()
        for w, axis in ((1, 0), (3, 1)):
            idx = np.nonzero(((e["i"] == w) | (e["j"] == w)))[0]
            assert len(idx) > 1024
            F, M = np.zeros(3), np.zeros(3)
            for k in idx[e["active"][idx]]:
                own = e["i"][k] == w
                F = F + f[0][k] if own else F - f[0][k]
                M = M + (f[1][k] if own else f[2][k])
            for d in range(3):
                if d != axis:
                    assert bitwise_equal(F[d:d + 1], b["force"][w, d:d + 1]), (steps, w, d)
            assert bitwise_equal(M, b["moment"][w]), (steps, w)
    g.close()


@pytest.mark.parametrize("scale,longest", [(1.0, 0), (3.0, 64), (8.0, 128)])
def test_resultants_of_lists_of_several_rounds(gpu_lib, scale, longest):
    """Small scenes, whose lanes look at 64 positions of a whole list (32 of a
    near list) together: lists within one round and over several give every
    free body the serial sum of its contributions, bit for bit (the moment,
    which starts from zero), on the near set as on the whole list."""
    sc = _scene("avalanche", 0.5)
    sc["dVerlet"] *= scale
    sc["DVerlet"] *= scale
    a, b = _engine(sc, 0, False), _engine(sc, 0, False)
    shift = np.zeros((a.n, 3))
    shift[sc["n_driven"]::2, 2] = 2e-5
    for g in (a, b):
        g.upload_kinematics(pos=np.ascontiguousarray(g.bodies()["pos"] + shift))
    for _ in range(12):
        a.step(1)
    b.step(12)
    e = _same(a, b, 0)
    f, bodies = b.contributions(), b.bodies()
    lengths = np.bincount(np.concatenate([e["i"], e["j"]]), minlength=a.n)[sc["n_driven"]:]
    assert lengths.max() > longest and e["active"].sum() > 20
    M = np.zeros((a.n, 3))
    for k in np.nonzero(e["active"])[0]:
        M[e["i"][k]] = M[e["i"][k]] + f[1][k]
        M[e["j"][k]] = M[e["j"][k]] + f[2][k]
    assert bitwise_equal(M[sc["n_driven"]:], bodies["moment"][sc["n_driven"]:])
    a.close()
    b.close()
