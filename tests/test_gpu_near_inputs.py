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
