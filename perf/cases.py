"""The work that a user of this framework has it do, as cases that can be timed.

A case builds a granular scene (packed sphero-polyhedra that touch and carry load, as in a running
simulation), holds it in an engine context, and runs one pass of what a program does with it:

  run       the host hands its particles over, the engine advances them some DEM steps, and the host
            takes them back (the coupling through rk_upload/download_kinematics_packed and rk_step)
  advance   a simulation that owns its state on the device runs on for some steps
  relist    the host moved the particles (a restart, a preprocessing command): neighbour list and
            forces are computed anew
  snapshot  the text of a conf file of the current state
  diagnose  the data extractors and the statistics of the current state

The scenes are the workloads of the repository's benchmark and tests at sizes from a few hundred
grains to its largest scene: a column that collapses (Avalanche law), a box of cubes and a slope
(Default law), isotropic compression between six servo walls, blocks of bonded grains that fall
(StickedLinks law, list updates on demand), and an ensemble of slopes in one context.
"""
import functools
import math

import numpy as np
import torch

from rockable_gb300 import abi, scenes

GRAINS_PER_TILE = 1000
INFLATE = 2e-6  # grains packed in touch are scaled by 1 + this: overlaps of about 3e-8 m, forces of the grains' weight
FLOOR_R = 0.005
FIELDS = (("pos", 3), ("vel", 3), ("acc", 3), ("Q", 4), ("vrot", 3), ("arot", 3))


# ------------------------------------------------------------------ shapes
@functools.lru_cache(maxsize=None)
def _library(kind):
    """The grain shapes a scene's shape file holds (the same file for every run)."""
    rng = np.random.default_rng(20261203)
    if kind == "cube":
        return [scenes.sphero_cube_box(2)["shapes"][1]]
    lo, hi, count = {"column": (0.005, 0.015, 192), "slope": (0.0025, 0.0075, 128), "iso": (0.004, 0.006, 192),
                     "block": (0.005, 0.010, 128)}[kind]
    return [scenes.hull_shape(rng, "%s%04d" % (kind, k), semi_lo=lo, semi_hi=hi) for k in range(count)]


@functools.lru_cache(maxsize=None)
def _at_rest(kind):
    """The orientation in which each shape of a library lies on a face."""
    lib = _library(kind)
    return scenes.stable_face_quaternions(np.random.default_rng(1), lib, np.arange(len(lib)))


def _yaw(q, a):
    """Quaternions q (rows) turned by the angle a (one, or one a row) about the vertical."""
    c, s = np.cos(0.5 * a), np.sin(0.5 * a)
    w, x, y, z = q.T
    return np.stack([c * w - s * z, c * x - s * y, c * y + s * x, c * z + s * w], 1)


def _tile(rng, kind, m, homothety=None):
    """m grains packed in a square footprint: positions, orientations, shapes, scales, side, height."""
    lib = _library(kind)
    so = rng.integers(0, len(lib), m)
    h = np.ones(m) if homothety is None else rng.uniform(homothety[0], homothety[1], m)
    if homothety is not None:
        h = h / np.array([2.0 * lib[k]["bound"] for k in so])  # homothety: a range of grain diameters
    q = _yaw(_at_rest(kind)[so], rng.uniform(0.0, 2.0 * math.pi, m))
    vol = np.array([lib[k]["volume"] for k in so]) * h ** 3
    side = max((vol.sum() / 0.5) ** (1.0 / 3.0), 2.2 * max(lib[k]["bound"] * s for k, s in zip(so, h)))
    pos, st = scenes.pack(lib, so, q, vol, (-0.5 * side, -0.5 * side, 0.0), (0.5 * side, 0.5 * side, 8.0 * side),
                          scale=h, seed=int(rng.integers(1, 1 << 30)), tries=4, cache=False)
    return pos, q, so, h, side, st["top"]


def _pile(rng, kind, n, homothety=None, aspect=1.0):
    """n grains: one packed tile set side by side and stacked, each copy turned by a multiple of 90
    degrees.  aspect: height over width.  Also returns the extents and each grain's copy."""
    m = min(n, GRAINS_PER_TILE)
    pos, q, so, h, side, top = _tile(rng, kind, m, homothety)
    order = np.argsort(pos[:, 2], kind="stable")  # a copy that is cut loses its top
    pos, q, so, h = pos[order], q[order], so[order], h[order]
    copies = -(-n // m)
    width = max(1, round((copies / aspect) ** (1.0 / 3.0)))
    nx = min(width, copies)
    ny = min(width, -(-copies // nx))
    layer = nx * ny
    P, Q, S, H, T = [], [], [], [], []
    left = n
    for c in range(copies):
        k = min(m, left)
        left -= k
        turn = int(rng.integers(0, 4))
        a, b = round(math.cos(0.5 * math.pi * turn)), round(math.sin(0.5 * math.pi * turn))
        p = pos[:k] @ np.array([[a, b, 0], [-b, a, 0], [0, 0, 1]], np.float64)
        at = c % layer
        p = p + np.array([(at % nx - 0.5 * (nx - 1)) * side, (at // nx - 0.5 * (ny - 1)) * side, (c // layer) * top])
        P.append(p)
        Q.append(_yaw(q[:k], 0.5 * math.pi * turn))
        S.append(so[:k])
        H.append(h[:k])
        T.append(np.full(k, c))
    ext = (nx * side, ny * side, -(-copies // layer) * top)
    return np.concatenate(P), np.concatenate(Q), np.concatenate(S), np.concatenate(H) * (1.0 + INFLATE), ext, \
        np.concatenate(T)


# ------------------------------------------------------------------ scenes
def _scene(rng, lib, walls, pile, law, dt, speed, kn=1e6, numbers=None):
    """Walls (driven bodies of group 1: shape, position, quaternion) first, then the grains (group 0)."""
    pos, q, so, h, _, copy = pile
    wall_shapes = []
    for w in walls:
        if not any(w[0] is s for s in wall_shapes):
            wall_shapes.append(w[0])
    shapes = wall_shapes + lib
    nd, n = len(walls), len(walls) + len(pos)
    shape = np.array([next(k for k, s in enumerate(wall_shapes) if s is w[0]) for w in walls] +
                     list(so + len(wall_shapes)), np.int32)
    hom = np.concatenate([np.ones(nd), h])
    P = np.concatenate([np.array([w[1] for w in walls], np.float64).reshape(-1, 3), pos])
    Q = np.concatenate([np.array([w[2] for w in walls], np.float64).reshape(-1, 4), q])
    Q = Q / np.linalg.norm(Q, axis=1)[:, None]
    mass = hom ** 3 * np.array([s["volume"] for s in shapes])[shape] * 2700.0
    inertia = np.array([s["I/m"] for s in shapes])[shape] * (hom ** 2 * mass)[:, None]
    bound = np.array([s["bound"] for s in shapes])[shape] * hom
    bmax = float(bound[nd:].max())
    vel, vrot = np.zeros((n, 3)), np.zeros((n, 3))
    vel[nd:] = rng.normal(0.0, speed, (n - nd, 3))
    vrot[nd:] = rng.normal(0.0, speed, (n - nd, 3)) / bound[nd:, None]
    body = {"pos": P, "vel": vel, "acc": np.zeros((n, 3)), "Q": Q, "vrot": vrot, "arot": np.zeros((n, 3)),
            "homothety": hom, "mass": mass, "inertia": inertia, "shape": shape,
            "group": np.concatenate([np.ones(nd), np.zeros(n - nd)]).astype(np.int32),
            "cluster": np.concatenate([np.zeros(nd), copy + 1]).astype(np.int32)}
    return {"name": law, "shapes": shapes, "n_driven": nd,
            "bodies": body, "law": law, "ngroup": 2, "dt": dt, "gravity": (0.0, 0.0, -9.81),
            "table": scenes.law_table(kn=kn, kt=kn, en2=0.25, mu=0.4) if numbers is None else numbers,
            "DVerlet": 0.2 * bmax, "dVerlet": 0.1 * bmax, "interVerlet": 100 * dt, "params": {}}


UPRIGHT = (1.0, 0.0, 0.0, 0.0)
S2 = math.sqrt(0.5)


def _grain_scene(rng, case):
    kind, n = case["scene"], case["n"]
    floor = scenes.plate_shape("FLOOR", 1.5, FLOOR_R)
    ground = [(floor, (0.0, 0.0, -FLOOR_R), UPRIGHT)]
    if kind == "column":  # the collapse of a column, about twice as high as wide
        lib = _library("column")
        return _scene(rng, lib, ground, _pile(rng, "column", n, aspect=2.0), "Avalanche", 1e-6, 0.05)
    if kind == "box":  # a heap of cubes (four-sided faces)
        lib = _library("cube")
        return _scene(rng, lib, ground, _pile(rng, "cube", n), "Default", 1e-6, 0.05)
    if kind == "slope":  # a pile on a plate inclined by 25 to 45 degrees
        lib = _library("slope")
        sc = _scene(rng, lib, ground, _pile(rng, "slope", n, aspect=0.5), "Default", 1e-6, 0.1)
        return scenes.tilt(sc, math.radians(float(rng.uniform(25.0, 45.0))))
    if kind == "iso":  # six walls around a dense box, three of them pushed at 100 kPa by the servo
        lib = _library("iso")
        pile = _pile(rng, "iso", n, homothety=(0.01, 0.03))
        X, Y, Z = pile[4]
        plate = scenes.plate_shape("WALL", 0.5 * max(X, Y, Z) + 0.02, FLOOR_R)
        x, y, z, c = 0.5 * X + FLOOR_R, 0.5 * Y + FLOOR_R, Z + FLOOR_R, 0.5 * Z
        walls = [(plate, (-x, 0, c), (S2, 0, S2, 0)), (plate, (x, 0, c), (S2, 0, S2, 0)),
                 (plate, (0, -y, c), (S2, S2, 0, 0)), (plate, (0, y, c), (S2, S2, 0, 0)),
                 (plate, (0, 0, -FLOOR_R), UPRIGHT), (plate, (0, 0, z), UPRIGHT)]
        sc = _scene(rng, lib, walls, pile, "Default", 5e-7, 0.01)
        sc["gravity"] = (0.0, 0.0, 0.0)
        sc["controls"] = {"type": [0, 6, 1, 7, 2, 8], "body": list(range(6)), "value": [0.0] * 6,
                          "vec": [[0.0] * 3] * 6}
        sc["servo"] = {"kind": 1, "icontr": 0, "walls": list(range(6)), "pressure": 1e5}
        return sc
    if kind == "blocks":  # blocks of bonded grains falling on a slope at 10 m/s
        lib = _library("block")
        sc = _scene(rng, lib, ground, _pile(rng, "block", n, aspect=0.3), "StickedLinks", 1e-6, 0.02, kn=1e7)
        sc["bodies"]["pos"][1:, 2] += 0.002
        sc["bodies"]["vel"][1:, 2] -= 10.0
        sc["bonded"] = True
        return scenes.tilt(sc, math.radians(30.0))
    raise ValueError(kind)


def _build_scene(case, seed):
    rng = np.random.default_rng([seed, case["n"]])
    if case["scene"] != "ensemble":
        sc = _grain_scene(rng, case)
        sc["shape_tables"] = scenes.flatten_shapes(sc["shapes"])
        return sc
    # independent slopes of different sizes in one context
    k = case["scenes"]
    share = np.random.default_rng([k, case["n"]]).uniform(0.3, 1.7, k)
    sizes = np.maximum(100, (case["n"] * share / share.sum()).astype(int))
    parts = [_grain_scene(rng, {"scene": "slope", "n": int(s)}) for s in sizes]
    d = min(p["dVerlet"] for p in parts)
    tables = scenes.flatten_shapes(parts[0]["shapes"])
    for p in parts:
        p.update(shapes=parts[0]["shapes"], shape_tables=tables, dVerlet=d, DVerlet=2.0 * d)
    return scenes.batch(parts)


# ------------------------------------------------------------------ states
def _bond(g, sc):
    """Bonds between vertices of one block's grains that lie within 0.3 mm, at rest at their distance."""
    g.accelerations()  # the list's distances
    e = g.entries()
    cl = sc["bodies"]["cluster"]
    near = (e["type"] == 0) & (e["dn"] < 3e-4) & (e["i"] >= sc["n_driven"]) & (cl[e["i"]] == cl[e["j"]])
    pair = e["i"].astype(np.int64) << 32 | e["j"].astype(np.int64)
    own, first, idx = np.unique(pair[near], return_index=True, return_inverse=True)
    at = np.nonzero(near)[0]
    e["bond"][:] = -1
    e["bond"][at] = idx
    i, j = (own >> 32).astype(np.int32), (own & 0xffffffff).astype(np.int32)
    par = np.tile(np.array([1e5, 1e5, 0.0, 1e3, 1e3, 1e10, 2.0, 0.0]), (len(own), 1))
    g.upload_interfaces(i, j, np.maximum(e["dn"][at[first]], 0.0), par, np.ones(len(own), np.int32))
    g.upload_entries(e)


def prepare(case, seed):
    sc = _build_scene(case, seed)
    b = sc["bodies"]
    mixed = case["form"] != "fp64"
    g = abi.GpuScene(device=0, form=abi.RK_FORM_MIXED if mixed else abi.RK_FORM_FP64)
    g.upload_shapes(sc["shape_tables"])
    g.upload_bodies(b, sc["n_driven"])
    if sc.get("scene_of") is not None:
        g.set_scenes(sc["scene_of"])
    if sc.get("bonded"):
        # list updates on demand: Rockable's guard on the bodies' displacement
        g.set_params(t=0.0, dt=sc["dt"], gravity=sc["gravity"], DVerlet=sc["DVerlet"], dVerlet=sc["dVerlet"],
                     interVerlet=sc["interVerlet"], interVerletC=0.0, law=abi.RK_LAW[sc["law"]], ngroup=2,
                     table=sc["table"], params_in_interfaces=1, dynamic_update_nl=1, disp_update_nl=5e-5,
                     angle_update_nl=math.radians(5.0))
    else:
        scenes.set_scene_params(g, sc)
    if case["form"] == "skin":
        d = sc["dVerlet"]
        g.set_skin(use_mlp=True, skin_min=0.1 * d, skin_max=4.0 * d, dverlet_ratio=2.0, interval_min=2,
                   interval_max=300, seed=3, exact_contacts=True)
    else:
        g.update_nl()
    if sc.get("bonded"):
        _bond(g, sc)
    g.set_graphs(case["graphs"])
    n = len(b["mass"])
    pinned = [torch.zeros(19 * n, dtype=torch.float64, pin_memory=True).numpy() for _ in range(3)]
    host = np.concatenate([np.ascontiguousarray(b[k]).ravel() for k, _ in FIELDS])
    pinned[0][:] = host
    pinned[1][:] = host  # the particles somewhat later (relist)
    pinned[1][:3 * n] += 5e-4 * host[3 * n:6 * n]
    st = {"case": dict(case), "g": g, "n": n, "bufs": pinned, "turn": 0, "mixed": mixed,
          "forces": {k: np.zeros((n, 3)) for k in ("force", "moment")}}
    if case["task"] in ("snapshot", "diagnose"):  # forces and contact geometry of the state that is put out
        g.set_shape_names([s["name"] for s in sc["shapes"]])
        g.set_record_geometry(True)
        g.accelerations()
        g.set_record_geometry(False)
        st["cluster"] = int(b["cluster"][-1])
        st["pages"] = [np.zeros(n * size, np.uint8) for size in (520, 2400)]
    return st


def _kinematics(st, buf):
    """The downloaded fields.  The mixed form computes accelerations, and the changes of the
    velocities, in float32; a program keeps them as such."""
    out, at = {}, 0
    for name, w in FIELDS:
        v = buf[at:at + w * st["n"]].reshape(st["n"], w)
        at += w * st["n"]
        out[name] = v.astype(np.float32) if st["mixed"] and name not in ("pos", "Q") else v
    return out


def run(st):
    case, g = st["case"], st["g"]
    task = case["task"]
    if task == "run":
        g.upload_kinematics_packed(st["bufs"][0])
        rep = g.step(case["steps"])
        out = _kinematics(st, g.download_kinematics_packed(st["bufs"][2]))
        if not st["mixed"]:
            out["counts"] = np.array([rep["n_entries"], rep["n_active"], rep["n_broken"]])
            if st["n"] <= 4000:  # a small scene's resultants too
                f = g.bodies(out=st["forces"])
                out.update(force=f["force"], moment=f["moment"])
        return out
    if task == "advance":
        g.step(case["steps"])
        return _kinematics(st, g.download_kinematics_packed(st["bufs"][2]))
    if task == "relist":
        st["turn"] ^= 1
        g.upload_kinematics_packed(st["bufs"][st["turn"]])
        g.update_nl()
        g.accelerations()
        s = g.bodies()
        return {"force": s["force"], "moment": s["moment"], "acc": s["acc"], "arot": s["arot"],
                "entries": g.n_entries}
    if task == "snapshot":
        bodies, contacts, count = g.format_conf(16)
        for text, page in ((bodies, st["pages"][0]), (contacts, st["pages"][1])):  # the file's buffers
            page[:len(text)] = np.frombuffer(text.encode(), np.uint8)
            page[len(text):] = 0
        return {"bodies": st["pages"][0], "contacts": st["pages"][1], "count": count > 0}
    if task == "diagnose":
        lo, hi = g.cluster_aabb(st["cluster"])
        s = g.stats()
        return {"speed": g.mean_velocity(), "dn": {k: v for k, v in g.dn_stat().items()}, "lo": lo, "hi": hi,
                "last": g.body(st["n"] - 1), "pair": g.duo_balance(0, st["n"] - 1),
                "e_trans": s["e_trans"], "e_rot": s["e_rot"], "contacts": s["n_active"]}
    raise ValueError(task)


def work(case):
    """One pass reads and writes the particles (152 bytes each), reads the contacts' history once and
    writes it once (a few contacts a grain, 88 bytes each), and computes each step's motion and contacts."""
    n, k = case["n"], case["steps"]
    if case["task"] == "snapshot":
        return {"bytes": n * (152 + 500) + 2 * n * (176 + 420), "flops": n * 20 * 40 + 2 * n * 17 * 40}
    if case["task"] == "diagnose":
        return {"bytes": n * (104 + 15 * 24) + 2 * n * 24, "flops": n * 200}
    if case["task"] == "relist":
        return {"bytes": 304 * n + 2 * 88 * 2 * n, "flops": n * 400 + 2 * n * 600}
    return {"bytes": 304 * n + 2 * 88 * 2 * n, "flops": k * (n * 400 + 2 * n * 300)}


def exact(case, seed):
    """The sums and boxes of `diagnose` in numpy.  The results of DEM steps have no closed form (None)."""
    if case["task"] != "diagnose":
        return None
    sc = _build_scene(case, seed)
    b, shapes = sc["bodies"], sc["shapes"]
    vel, q = b["vel"], b["Q"]
    conj = q * np.array([1.0, -1.0, -1.0, -1.0])
    w = _rotate(conj, b["vrot"])
    lo, hi = np.full(3, np.inf), np.full(3, -np.inf)
    for k in np.nonzero(b["cluster"] == b["cluster"][-1])[0]:
        s, h = shapes[b["shape"][k]], b["homothety"][k]
        v = _rotate(np.broadcast_to(q[k], (len(s["vertices"]), 4)), h * s["vertices"]) + b["pos"][k]
        lo, hi = np.minimum(lo, v.min(0) - h * s["radius"]), np.maximum(hi, v.max(0) + h * s["radius"])
    last = {k: b[k][-1] if k in ("pos", "vel", "Q", "vrot") else None for k in
            ("pos", "vel", "acc", "Q", "vrot", "arot", "force", "moment")}
    return {"speed": float(np.linalg.norm(vel, axis=1).mean()), "dn": None, "lo": lo, "hi": hi, "last": last,
            "pair": None, "e_trans": float(0.5 * (b["mass"] * (vel ** 2).sum(1)).sum()),
            "e_rot": float(0.5 * (b["inertia"] * w ** 2).sum()), "contacts": None}


def _rotate(q, v):
    u = q[:, 1:]
    t = 2.0 * np.cross(u, v)
    return v + q[:, :1] * t + np.cross(u, t)


def _case(name, task, scene, n, form, steps, graphs=True, **more):
    c = {"task": task, "scene": scene, "n": n, "form": form, "steps": steps, "graphs": graphs, **more}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a host loop that looks at the particles after every step: the smallest call, default options
        _case("box_512_call", "run", "box", 512, "fp64", 1, graphs=False),
        # one slope of a parameter study, the usual block of 100 steps between list updates
        _case("slope_1700", "run", "slope", 1700, "fp64", 100),
        _case("slope_4300_mixed", "run", "slope", 4300, "mixed", 100),
        # the collapse of a column of 50 000 grains: reference arithmetic, mixed, mixed with the learned skin
        _case("column_50k", "run", "column", 50000, "fp64", 100),
        _case("column_50k_mixed", "run", "column", 50000, "mixed", 100),
        _case("column_50k_skin", "advance", "column", 50000, "skin", 100),
        # isotropic compression between servo walls, the largest scene (half a list interval)
        _case("iso_200k", "run", "iso", 200000, "fp64", 50),
        # bonded blocks in fall: breakable interfaces and list updates on demand
        _case("blocks_6k", "run", "blocks", 6000, "fp64", 40),
        # many slopes in one context
        _case("ensemble_24", "run", "ensemble", 24011, "fp64", 50, scenes=24),
        # list and forces of particles that the host moved
        _case("relist_50k", "relist", "column", 50000, "fp64", 0),
        # output between the steps: the conf text, and the extractors
        _case("snapshot_20k", "snapshot", "column", 20000, "fp64", 0),
        _case("diagnose_20k", "diagnose", "column", 20000, "fp64", 0, graphs=False),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | 1

    pick = rng.random()
    if pick < 0.10:
        return _case(None, "run", "box", size(300, 4000), "fp64", rng.choice([1, 2, 5]), graphs=False)
    if pick < 0.35:
        return _case(None, "run", "slope", size(200, 20000), rng.choice(["fp64", "mixed"]), rng.choice([20, 50, 100]),
                     graphs=rng.random() < 0.7)
    if pick < 0.60:
        form = rng.choice(["fp64", "mixed", "skin"])
        return _case(None, "advance" if form == "skin" else "run", "column", size(1000, 60000), form,
                     rng.choice([20, 50, 100]))
    if pick < 0.70:
        return _case(None, "run", "iso", size(2000, 80000), rng.choice(["fp64", "mixed"]), rng.choice([20, 50]))
    if pick < 0.78:
        return _case(None, "run", "blocks", size(500, 10000), "fp64", rng.choice([10, 20, 40]))
    if pick < 0.84:
        k = rng.randint(4, 32)
        return _case(None, "run", "ensemble", size(200 * k, 600 * k), "fp64", rng.choice([20, 50]), scenes=k)
    if pick < 0.92:
        return _case(None, "relist", rng.choice(["column", "slope"]), size(1000, 60000), "fp64", 0)
    if pick < 0.96:
        return _case(None, "snapshot", rng.choice(["column", "slope"]), size(500, 40000), "fp64", 0)
    return _case(None, "diagnose", "slope", size(500, 40000), "fp64", 0, graphs=False)
