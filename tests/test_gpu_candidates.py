"""Candidate sub-contacts of the list build (GPU): the neighbour list of
bodies of the smallest and the largest vertex counts (4 to 64: one and two
vertices a lane), of four-sided faces and of a plate, from touching to far
overlapping and to just beyond the NEAR distance, equals the oracle's list
key for key; so does the list after the bodies moved (old entries tested or
kept)."""
import numpy as np
import pytest

from helpers import bitwise_equal, gpu_from_oracle, key_tuples

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spacing", [0.7, 1.0, 1.25])
@pytest.mark.parametrize("verts", [(4, 4), (31, 33), (60, 64), (0, 0)])
def test_candidates_match_oracle(gpu_lib, oracle_lib, tmp_path, verts, spacing):
    from rockable_gb300 import scenes
    rng = np.random.default_rng(7)
    if verts[0]:
        lib = [scenes.hull_shape(rng, "H%d" % k, kmin=verts[0], kmax=verts[1]) for k in range(6)]
    else:
        lib = [scenes.sphero_cube_box(2)["shapes"][1]]
    shapes = [scenes.plate_shape("FLOOR", 0.3, 0.005)] + lib
    d = 2.0 * max(s["bound"] for s in lib)
    side = 4
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (g - 0.5 * (side - 1)) * d * spacing * 0.75 + rng.normal(0, 0.05 * d, (len(g), 3))
    pos[:, 2] += 0.55 * d - pos[:, 2].min()
    Q = scenes.random_quaternions(rng, len(pos))
    sc = scenes._assemble(shapes, [np.array([0, 0, -0.005])], [np.array([1.0, 0, 0, 0])], pos, Q,
                          rng.integers(1, len(shapes), len(pos)), 2700.0, "Default", 1e6, 1e6, 0.25, 0.4, 1e-6,
                          gravity=(0.0, 0.0, -9.81), DVerlet=0.2 * d, dVerlet=0.1 * d, interVerlet=1e-4, name="cand")
    o = oracle_lib.Oracle(scenes.write_conf(sc, str(tmp_path)))
    gp = gpu_from_oracle(o)
    o.update_nl()
    gp.update_nl()
    oe, ge = o.entries(), gp.entries()
    assert spacing > 0.8 or len(ge["i"]) > 0
    assert key_tuples(oe) == key_tuples(ge)
    # a few steps of the violent overlaps move the bodies; then the next list
    o.run(3)
    gp.step(3)
    o.update_nl()
    gp.update_nl()
    oe, ge = o.entries(), gp.entries()
    assert key_tuples(oe) == key_tuples(ge)
    for k in ["dn", "fn", "ft", "mom", "damp"]:
        assert bitwise_equal(oe[k], ge[k]), k
