"""GPU parity of the denoiser's tiled filter: images smaller than a tile, at its edges and one pixel beyond, and
iteration counts whose steps reach every tiled variant (1, 2, 4, 8) and the untiled one (16, 32); G-buffers with
infinities and NaN in places.  Bit-exact against the restatement, images and state."""
import numpy as np
import pytest

from neonengine_b200 import svgf_synth
from oracle import svgf
from test_svgf_gpu import _denoiser, _run_frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (31, 15), (32, 16), (33, 17), (64, 8), (7, 70)])
@pytest.mark.parametrize("iterations", [3, 4, 6])
def test_tile_edges_and_steps(w, h, iterations):
    _run_frames(w, h, iterations, 3, device_path=True)


def test_values_that_are_not_finite():
    w, h = 70, 40
    dn, st = _denoiser(w, h), svgf.State.zeros(w, h)
    rng = np.random.default_rng(2)
    for i in range(3):
        g, image = svgf_synth.make_frame(w, h, i)
        for a, v in ((g[0], np.nan), (g[0], np.inf), (g[1], np.nan), (g[1], 3.0)):  # depths, normals (one of them far from unit)
            a[rng.integers(0, h, 6), rng.integers(0, w, 6), 2] = v
        want = image.copy()
        svgf.frame(g, want, st, 3, serial=False)
        dn.render_host(g, image)
        np.testing.assert_array_equal(image, want)
        a, b, m, pp = dn.read_state()
        np.testing.assert_array_equal(a, st.colour_a)
        np.testing.assert_array_equal(b, st.colour_b)
        np.testing.assert_array_equal(m, st.data)  # a NaN equals a NaN here, whatever its bits
    dn.close()
