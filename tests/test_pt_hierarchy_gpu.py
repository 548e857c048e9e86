"""GPU parity of the path tracer where its hierarchy is unusual: a scene that is one leaf, many triangles in one
place (no split separates them), a long thin row of triangles (deep splits).  Bit-exact against the CPU oracle, ray
counts included."""
import numpy as np
import pytest

from neonengine_b200 import pt_synth
from oracle import pt

pytestmark = pytest.mark.gpu


def _scene(offsets, sizes):
    """Quads facing the camera (two triangles each) at the offsets; material 0 is the one light."""
    vs, idx = [], []
    for i, (o, s) in enumerate(zip(offsets, sizes)):
        v = np.zeros(4, pt_synth.VERTEX_DTYPE)
        v["pos"][:, :3] = np.asarray(o, np.float32) + np.float32(s) * np.array([(-1, -1, 0), (1, -1, 0), (1, 1, 0), (-1, 1, 0)], np.float32)
        v["pos"][:, 3] = 1.0
        v["normal"][:, 2] = -1.0
        v["material"] = 0 if i == 0 else 1
        vs.append(v)
        idx += [4 * i + k for k in ((0, 1, 2, 0, 2, 3) if i % 2 else (0, 2, 1, 0, 3, 2))]
    mats = np.zeros(2, pt_synth.MATERIAL_DTYPE)
    mats["albedo"] = 0.8
    mats["misc"][:, 0] = 0.6
    mats[0]["emission"] = 5.0
    mats[0]["position"] = (*offsets[0], 0.1)
    return pt_synth.PtScene(np.concatenate(vs), np.array(idx, np.uint32), mats, 1)


CASES = {
    "one leaf": ([(0, 0, 1.0)], [0.8]),
    "one place": ([(0, 0, 1.0)] * 40, [0.7] * 40),
    "row": ([(0, -0.6, 0.5)] + [(0.9 ** i - 0.4, 0, 1.0 + 0.001 * i) for i in range(300)], [0.1] + [0.05 * 0.97 ** i for i in range(300)]),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_unusual_hierarchies(name):
    from neonengine_b200.path_tracer import PathTracer
    sc = _scene(*CASES[name])
    w, h = 61, 47
    ip, iv = pt_synth.camera(w, h, position=(0.0, 0.0, -1.0))
    t = PathTracer(sc, w, h, device=0)
    want, rays = pt.render(sc, ip, iv, 3.0, w, h)
    np.testing.assert_array_equal(t.render_host(ip, iv, 3.0), want)
    assert t.rays() == rays and t.status() == 0
    assert t.bvh_info()[1] < 48
    t.close()
