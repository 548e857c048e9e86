"""GPU parity of the streamed pass of one token (csrc/decode_stream.cuh): depths whose chunks do not divide evenly
over its warps (fewer chunks than warps among them), a last weight tile that is half padding, every expert count that
changes the router's split, scale bytes over a wide range, a token whose logits are the bias alone, against the CPU
oracle and against the one-launch and the grouped-GEMM path."""
import numpy as np
import pytest

import oracle
from helpers import assert_close, errors
from neonengine_b200 import synth
from test_moe_gpu import check_against_oracle, make_layer, run_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,inter,experts,top_k", [(64, 64, 8, 2), (192, 320, 32, 4), (576, 192, 128, 4), (704, 448, 256, 3), (320, 576, 4, 4), (2880, 64, 8, 8)])
@pytest.mark.parametrize("seed", [1, 2])
def test_against_the_oracle(hidden, inter, experts, top_k, seed):
    shape = synth.MoeShape(hidden=hidden, inter=inter, n_experts=experts, top_k=top_k)
    W = synth.make_weights(shape, 11)
    lb = synth.zipf_logit_bias(experts) if seed == 2 and experts > top_k else None
    x = synth.make_hidden(1, W, 20 + seed, logit_bias=lb)
    layer = make_layer(shape, W, max_tokens=8)
    layer.set_option("use_graphs", 0)
    before = layer.launch_count
    out, (max_abs, mean_rel) = check_against_oracle(layer, W, x, logit_bias=lb, what="stream")
    assert layer.launch_count - before == 3
    # f32 sums of at most 2880 exact products (their rounding adds up like its square root, 54 * 2^-24) and 22-bit activations
    assert mean_rel < 4e-6, (max_abs, mean_rel)
    np.testing.assert_array_equal(run_device(layer, x, lb)[0], out)  # two runs, the same bits
    for option in ("decode_stream", "decode_fused"):
        layer.set_option(option, 0)
        before = layer.launch_count
        assert_close(out, run_device(layer, x, lb)[0], "stream vs " + option + " 0")
        launches = layer.launch_count - before
        # the one-launch kernel (which takes no more experts than there are SMs), the general path: not the stream again
        assert launches == 1 if option == "decode_stream" and experts <= 128 else launches >= 6
    layer.close()


def test_scales_over_a_wide_range_and_a_zero_token():
    shape = synth.MoeShape(hidden=192, inter=128, n_experts=8, top_k=2)
    W = synth.make_weights(shape, 3)
    rng = np.random.default_rng(0)
    W.gate_up_scales[:] = rng.integers(2, 132, W.gate_up_scales.shape)
    W.down_scales[:] = rng.integers(2, 132, W.down_scales.shape)
    layer = make_layer(shape, W, max_tokens=1)
    for x in (synth.make_hidden(1, W, 5), np.zeros((1, 192), np.uint16)):
        out, idx, w = run_device(layer, x)
        assert errors(out, oracle.experts(x, idx, w, W))[1] < 4e-6 and np.isfinite(out).all()
    layer.close()


@pytest.mark.parametrize("limit,alpha", [(0.02, 1.702), (0.05, 1.702), (0.3, 0.1), (7.0, 0.01), (0.5, 1e-4), (50.0, 1.702)])
def test_swiglu_bounds(limit, alpha):
    """The gate's negative lobe is 0.278 / alpha deep, with gates far enough out to meet it."""
    shape = synth.MoeShape(hidden=192, inter=128, n_experts=8, top_k=2, swiglu_limit=limit, swiglu_alpha=alpha)
    W = synth.make_weights(shape, 7)
    x = synth.make_hidden(1, W, 8)
    # gates of a few times 1.28 / alpha, where the lobe is deepest
    W.gate_up_scales[:] = np.clip(W.gate_up_scales.astype(int) + int(np.round(np.log2(4.0 / alpha))), 1, 250)
    layer = make_layer(shape, W, max_tokens=1)
    layer.set_option("use_graphs", 0)
    before = layer.launch_count
    out, idx, w = run_device(layer, x)
    assert layer.launch_count - before == 3
    ref = oracle.experts(x, idx, w, W)
    assert np.isfinite(out).all() and errors(out, ref)[1] < 4e-6
    layer.close()


@pytest.mark.parametrize("alpha", [0.0, -1.0])
def test_gates_without_a_bound_keep_off_the_stream(alpha):
    shape = synth.MoeShape(hidden=192, inter=128, n_experts=8, top_k=2, swiglu_alpha=alpha)
    W = synth.make_weights(shape, 7)
    layer = make_layer(shape, W, max_tokens=1)
    layer.set_option("use_graphs", 0)
    before = layer.launch_count
    out, idx, w = run_device(layer, synth.make_hidden(1, W, 8))
    assert layer.launch_count - before == 1 and np.isfinite(out).all()
    layer.close()


@pytest.fixture(scope="module")
def small_layer():
    shape = synth.MoeShape(hidden=192, inter=320, n_experts=8, top_k=2)
    W = synth.make_weights(shape, 9)
    layer = make_layer(shape, W, max_tokens=8)
    layer.set_option("use_graphs", 0)
    yield layer, synth.make_hidden(1, W, 10)
    layer.close()


def _with(layer, x, **options):
    """Output and number of launches of a pass with the options set, which go back to their defaults."""
    defaults = {"decode_fused": 1, "decode_fused_tokens": 1, "decode_stream": 1, "decode_sliced": 0}
    for k, v in options.items():
        layer.set_option(k, v)
    before = layer.launch_count
    out = run_device(layer, x)[0]
    for k in options:
        layer.set_option(k, defaults[k])
    return out, layer.launch_count - before


def test_no_tokens_for_the_one_launch_kernel_means_the_general_path(small_layer):
    layer, x = small_layer
    general, launches = _with(layer, x, decode_fused=0)
    out, n = _with(layer, x, decode_fused_tokens=0)
    assert n == launches > 3
    np.testing.assert_array_equal(out, general)


def test_the_sliced_variant_is_taken_when_asked_for(small_layer):
    layer, x = small_layer
    sliced, n = _with(layer, x, decode_sliced=1)
    want, m = _with(layer, x, decode_sliced=1, decode_fused_tokens=8)
    one_launch, k = _with(layer, x, decode_stream=0)
    assert n == m == k == 1
    np.testing.assert_array_equal(sliced, want)
    assert (sliced != one_launch).any()  # another order of the sums: not the one-launch kernel under another name
