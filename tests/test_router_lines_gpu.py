"""GPU checks of which router a pass takes: the one-CTA-per-token router up to 384 tokens where the tensor-core router
does not serve the expert count, up to 224 where it does.  Only the first leaves the token maxima that tiles of 32
tokens need: after the others they are one more launch."""
import pytest

from neonengine_b200 import synth
from test_moe_gpu import make_layer, run_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("experts,line", [(16, 384), (64, 384), (32, 224), (128, 224)])
def test_router_line(experts, line):
    shape = synth.MoeShape(hidden=704, inter=64, n_experts=experts, top_k=4)
    W = synth.make_weights(shape, 3)
    layer = make_layer(shape, W, max_tokens=385)
    layer.set_option("tile_tokens", 32)

    def launches(x, wide_max):
        layer.set_option("router_wide_max", wide_max)
        before = layer.launch_count
        run_device(layer, x)
        return layer.launch_count - before

    for T in (224, 225, 300, 384, 385):
        x = synth.make_hidden(T, W, T)
        wide, other = launches(x, 385), launches(x, 0)
        assert other == wide + 1
        assert launches(x, -1) == (wide if T <= line else other)
    layer.close()


@pytest.mark.parametrize("experts,waves", [(32, 32), (128, 16), (128, 32)])
def test_large_router_tiles(experts, waves):
    """Passes of more than 16 and 32 tokens per SM take 32 and 64 tokens a CTA: the last tile holds one token."""
    import numpy as np
    import torch
    from test_moe_gpu import check_against_oracle
    T = waves * torch.cuda.get_device_properties(0).multi_processor_count + 1
    shape = synth.MoeShape(hidden=320, inter=64, n_experts=experts, top_k=4)
    W = synth.make_weights(shape, 4)
    layer = make_layer(shape, W, max_tokens=T)
    x = synth.make_hidden(T, W, 6)
    check_against_oracle(layer, W, x, tokens=np.unique(np.r_[0, np.arange(0, T, 97), T - 2, T - 1]).astype(np.int32), what="router tiles")
    layer.close()
