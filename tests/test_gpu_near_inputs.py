"""Steps on the near set (GPU) over inputs that its tests and tables have to
follow: K steps in one call leave the same bits as K calls of one step, which
run on the whole list."""
import numpy as np
import pytest

from helpers import bitwise_equal
from test_gpu_near import _engine, _same, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1])
def test_new_shape_tables_reach_the_near_set(gpu_lib, form):
    """New shape tables under bodies and a list that stay: the elements that
    an entry's indices name are other ones (edges and faces in another order)."""
    sc = _scene("avalanche", 0.5)
    a, b = _engine(sc, form, False), _engine(sc, form, False)
    t = {k: np.array(v) for k, v in sc["shape_tables"].items()}
    assert np.all(np.diff(t["face_vofs"])[t["face_ofs"][1]:] == 3)  # (the floor's face stays)
    edges, faces = t["edges"].reshape(-1, 2), t["face_verts"]
    for k in range(1, len(t["radius"])):
        e, f = slice(*t["edge_ofs"][k:k + 2]), slice(*t["face_vofs"][t["face_ofs"][k:k + 2]])
        edges[e] = edges[e][::-1].copy()
        faces[f] = faces[f].reshape(-1, 3)[::-1].ravel().copy()
    t["edges"] = edges.ravel()
    for g in (a, b):
        g.step(3)
        g.upload_shapes(t)
    for _ in range(24):
        a.step(1)
    b.step(24)
    assert _same(a, b, form)["active"].sum() > 20
    a.close()
    b.close()


def _tips(count, length, rng):
    """Long rods (driven, all centred at the origin) with a sphere at the tip of each."""
    from rockable_gb300 import scenes
    r, rho = 0.005, 2700.0
    rod = {"name": "ROD", "radius": r, "vertices": np.array([[0.0, 0.0, 0.0], [length, 0.0, 0.0]]),
           "edges": np.array([[0, 1]]), "faces": [], "obb_center": np.array([0.5 * length, 0.0, 0.0]),
           "obb_extent": np.array([0.5 * length + r, r, r])}
    ball = {"name": "BALL", "radius": r, "vertices": np.zeros((1, 3)), "edges": np.zeros((0, 2), int), "faces": [],
            "obb_center": np.zeros(3), "obb_extent": np.full(3, r)}
    Q = scenes.random_quaternions(rng, count)
    w, x, y, z = Q.T
    axis = np.stack([1.0 - 2.0 * (y * y + z * z), 2.0 * (x * y + w * z), 2.0 * (x * z - w * y)], 1)
    overlap = rng.uniform(2e-8, 4e-6, count)
    zero = np.zeros((2 * count, 3))
    bodies = {"pos": np.concatenate([np.zeros((count, 3)), axis * (length + 2.0 * r - overlap)[:, None]]),
              "vel": zero, "acc": zero, "vrot": zero, "arot": zero, "Q": np.concatenate([Q, Q]),
              "homothety": np.ones(2 * count), "mass": np.full(2 * count, 4.0 / 3.0 * np.pi * r ** 3 * rho),
              "inertia": np.full((2 * count, 3), 0.4 * 4.0 / 3.0 * np.pi * r ** 5 * rho),
              "shape": np.repeat([0, 1], count), "group": np.repeat([1, 0], count), "cluster": np.zeros(2 * count)}
    return {"shape_tables": scenes.flatten_shapes([rod, ball]), "bodies": bodies, "n_driven": count, "law": "Default",
            "ngroup": 2, "table": scenes.law_table(1e6, 1e6, 0.25, 0.4), "dt": 1e-6, "gravity": (0.0, 0.0, 0.0),
            "DVerlet": 2e-3, "dVerlet": 1e-3, "interVerlet": 1.0}


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("length", [0.5, 30.0, 200.0])
def test_contacts_far_from_their_bodys_centre(gpu_lib, form, length):
    """Overlaps that are small against the rounding of a float vertex offset
    of a large body: the near set's float distance must not pass them by."""
    sc = _tips(64, length, np.random.default_rng(3))
    a, b = _engine(sc, form, False), _engine(sc, form, False)
    for _ in range(12):
        a.step(1)
    b.step(12)
    assert _same(a, b, form)["active"].sum() == 64
    a.close()
    b.close()


@pytest.mark.parametrize("form", [0, 1])
def test_bonds_without_interfaces(gpu_lib, form):
    """Entries uploaded with a bond in a scene without interfaces count as
    active while apart, which restarts their history from zero: balls that
    bounce on a rod's tip, dragged sideways, in flights of 20 steps."""
    from rockable_gb300 import scenes
    n = 4
    sc = _tips(n, 0.6, np.random.default_rng(5))
    sc["dVerlet"], sc["DVerlet"] = 0.3, 0.6  # (near sets that last for several bounces)
    sc["table"] = scenes.law_table(1e6, 1e6, 1.0, 10.0)
    d = sc["bodies"]["pos"][n:] / np.linalg.norm(sc["bodies"]["pos"][n:], axis=1)[:, None]
    side = np.cross(d, np.eye(3)[np.argmin(np.abs(d), axis=1)])
    sc["bodies"]["pos"][n:] = d * (0.61 - 1e-9)
    vel = np.zeros((2 * n, 3))
    vel[n:] = 10.0 * d + side
    sc["bodies"]["vel"] = vel
    a, b = _engine(sc, form, False), _engine(sc, form, False)
    e = a.entries()
    tips = e["type"] == 0
    assert tips.sum() == n
    e["bond"][tips] = 0
    for g in (a, b):
        g.upload_entries(e)
        g.set_body_force("AttractingPoint", (0.0, 0.0, 0.0, 1e6))
    for k in (100, 600, 800):
        for _ in range(k):
            ra = a.step(1)
        rb = b.step(k)
        assert ra["n_active"] == rb["n_active"] == n
        _same(a, b, form)
    a.close()
    b.close()


@pytest.mark.parametrize("form", [0, 1])
def test_near_set_steps_of_a_large_scene(gpu_lib, form):
    """More than 19 456 bodies (one thread per body in the resultants and in
    the drift), not a multiple of a block, with walls of more than 1024
    entries whose resultants a block sums."""
    from rockable_gb300 import scenes
    sc = scenes.iso_compression(n=20011, nshapes=24, tries=1)
    sc["dVerlet"] *= 3.0
    sc["DVerlet"] *= 3.0
    nd, n = sc["n_driven"], len(sc["bodies"]["mass"])
    rng = np.random.default_rng(11)
    sc["bodies"]["vel"][nd:] = rng.normal(0, 0.3, (n - nd, 3))
    sc["bodies"]["vrot"][nd:] = rng.normal(0, 30.0, (n - nd, 3))
    sc["interVerlet"] = 20 * sc["dt"]
    a, b = _engine(sc, form, False), _engine(sc, form, True)
    e = a.entries()
    assert max(np.sum((e["i"] == w) | (e["j"] == w)) for w in (1, 3, 5)) > 1024
    shift = np.zeros((n, 3))
    shift[nd::2, 2] = 2e-5  # half of the grains into their neighbours
    for g in (a, b):
        g.upload_kinematics(pos=np.ascontiguousarray(g.bodies()["pos"] + shift))
    for _ in range(33):
        a.step(1)
    b.step(33)
    assert _same(a, b, form)["active"].sum() > 1000
    a.close()
    b.close()
