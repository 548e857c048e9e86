"""GPU checks of the denoiser's state between frames: history loaded from device and from pageable host memory, the
moments read straight after a frame on the NULL stream, frames that the caller captures and replays between others.
Bit-exact against the restatement."""
import ctypes

import numpy as np
import pytest

from neonengine_b200 import svgf_synth
from oracle import svgf
from test_svgf_gpu import _check_state, _denoiser

pytestmark = pytest.mark.gpu


def _state(w, h, seed=5):
    rng = np.random.default_rng(seed)
    return svgf.State(rng.random((h, w, 4)).astype(np.float16).view(np.uint16), rng.random((h, w, 4)).astype(np.float16).view(np.uint16),
                      rng.random((h, w, 4)).astype(np.float32) * np.array([6, 1, 1, 0.05], np.float32), 1)


def _read(dn, name, like):
    got = np.empty_like(like)
    dn._check(dn._lib.neon_svgf_read(dn._h, name.encode(), ctypes.c_void_p(got.ctypes.data), got.nbytes), "neon_svgf_read")
    return got


@pytest.mark.parametrize("on_device", [True, False])
def test_large_history_arrives(on_device):
    import torch
    w, h = 1920, 1080
    dn, st = _denoiser(w, h), _state(w, h)
    for turn in range(3):
        images = [st.colour_a, st.colour_b, np.roll(st.data, turn, axis=1)]
        held = [torch.from_numpy(a.view(np.int16) if a.dtype == np.uint16 else a).cuda() for a in images] if on_device else images
        ptrs = [ctypes.c_void_p(a.data_ptr() if on_device else a.ctypes.data) for a in held]
        dn._check(dn._lib.neon_svgf_set_history(dn._h, *ptrs, 1, int(on_device)), "neon_svgf_set_history")
        np.testing.assert_array_equal(_read(dn, "moments", st.data), images[2])
        np.testing.assert_array_equal(_read(dn, "colour_b", st.colour_b), images[1])
    dn.close()


def test_frame_from_device_history():
    import torch
    w, h = 200, 120
    dn, st = _denoiser(w, h), _state(w, h)
    held = [torch.from_numpy(a.view(np.int16) if a.dtype == np.uint16 else a).cuda() for a in (st.colour_a, st.colour_b, st.data)]
    dn._check(dn._lib.neon_svgf_set_history(dn._h, *(ctypes.c_void_p(a.data_ptr()) for a in held), 1, 1), "neon_svgf_set_history")
    g, image = svgf_synth.make_frame(w, h, 3)
    dg, dimg = [torch.from_numpy(a).cuda() for a in g], torch.from_numpy(image).cuda()
    dn.render(dg, dimg, stream=torch.cuda.Stream())  # a stream that the NULL stream does not order
    svgf.frame(g, image, st, 3, serial=False)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(dimg.cpu().numpy(), image)
    _check_state(dn, st)
    dn.close()


def test_moments_straight_after_a_frame():
    import torch
    w, h = 1920, 1080
    dn = _denoiser(w, h)
    frames = [svgf_synth.make_frame(w, h, i) for i in range(2)]
    dg = [[torch.from_numpy(a).cuda() for a in g] for g, _ in frames]
    dimg = [torch.from_numpy(image).cuda() for _, image in frames]
    torch.cuda.synchronize()
    for g, image in zip(dg, dimg):
        dn.render(g, image)  # the NULL stream; nothing waits for it before the read
    got = _read(dn, "moments", np.empty((h, w, 4), np.float32))
    np.testing.assert_array_equal(_read(dn, "moments", got), got)
    st = svgf.State.zeros(w, h)
    for g, image in frames:
        svgf.frame(g, image, st, 3, serial=False)
    np.testing.assert_array_equal(got, st.data)
    dn.close()


@pytest.mark.parametrize("before", [0, 1])
@pytest.mark.parametrize("captured", [1, 2])
def test_captured_frames_go_on_with_the_history(before, captured):
    import torch
    w, h = 96, 64
    dn, st = _denoiser(w, h), svgf.State.zeros(w, h)
    g, image = svgf_synth.make_frame(w, h, 1)
    dg, fresh = [torch.from_numpy(a).cuda() for a in g], torch.from_numpy(image).cuda()
    dimg = fresh.clone()

    def eager():
        dimg.copy_(fresh)
        dn.render(dg, dimg)
        check(1, st.ping_pong)

    def check(frames, ping_pong):
        st.ping_pong = ping_pong
        for _ in range(frames):
            want = image.copy()
            svgf.frame(g, want, st, 3, serial=False)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(dimg.cpu().numpy(), want)
        np.testing.assert_array_equal(_read(dn, "moments", st.data), st.data)
        np.testing.assert_array_equal(_read(dn, "colour_a", st.colour_a), st.colour_a)
        np.testing.assert_array_equal(_read(dn, "colour_b", st.colour_b), st.colour_b)

    for _ in range(before):
        eager()
    flag = st.ping_pong
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side):
        for _ in range(captured):
            dimg.copy_(fresh)
            dn.render(dg, dimg, stream=side)
    st.ping_pong = (flag + captured) & 1  # what the captured calls left the handle's own flag at
    for replays in (1, 2, 3):
        for _ in range(replays):
            own = st.ping_pong
            graph.replay()
            check(captured, flag)
            st.ping_pong = own
        eager()
    history = _state(w, h)
    torch.cuda.synchronize()
    dn.set_history(history.colour_a, history.colour_b, history.data, flag)
    st = history
    graph.replay()
    check(captured, flag)
    dn.close()
