"""GPU parity of the prefill operand rows (split_rows_kernel and quant_rows_mxfp4_kernel, csrc/gmm_sm100.cuh): depths
that end in half a chunk, chunk groups that are not full, a single chunk, every top_k up to 8, token tiles with
one row and with 128, blocks of zeros, against the CPU oracle."""
import numpy as np
import pytest

import oracle
from helpers import errors
from neonengine_b200 import synth
from test_moe_gpu import check_against_oracle, make_layer, run_device

pytestmark = pytest.mark.gpu

SHAPES = [(64, 64, 4, 1), (192, 320, 8, 2), (576, 704, 4, 4), (704, 192, 8, 8), (2880, 64, 3, 3)]


@pytest.mark.parametrize("hidden,inter,experts,top_k", SHAPES)
@pytest.mark.parametrize("T", [512, 777])
def test_terms_against_the_oracle(hidden, inter, experts, top_k, T):
    shape = synth.MoeShape(hidden=hidden, inter=inter, n_experts=experts, top_k=top_k)
    W = synth.make_weights(shape, 5)
    layer = make_layer(shape, W, max_tokens=T)
    layer.set_option("use_graphs", 0)
    x = synth.make_hidden(T, W, T)
    x[3, :32] = 0      # a block whose scale has no exponent to take
    x[5] = 0
    toks = np.unique(np.r_[3, 5, np.arange(0, T, 41), T - 1]).astype(np.int32)
    out, (_, mean_rel) = check_against_oracle(layer, W, x, tokens=toks, what="split")
    # each e4m3 term leaves at most 2^-4 of what it was given: two terms in front, three in the middle
    assert mean_rel < 2.0**-8 + 2.0**-12, mean_rel
    np.testing.assert_array_equal(run_device(layer, x)[0], out)
    layer.close()


@pytest.mark.parametrize("hidden,inter,experts,top_k", SHAPES)
def test_mxfp4_rows_against_the_quantising_oracle(hidden, inter, experts, top_k):
    shape = synth.MoeShape(hidden=hidden, inter=inter, n_experts=experts, top_k=top_k)
    W = synth.make_weights(shape, 6)
    T = 777
    layer = make_layer(shape, W, max_tokens=T)
    layer.set_option("mxf4_prefill", 1)
    x = synth.make_hidden(T, W, 9)
    x[3, :32] = 0
    toks = np.unique(np.r_[3, np.arange(0, T, 41), T - 1]).astype(np.int32)
    out, idx, w = run_device(layer, x)
    ref = oracle.experts(x, idx, w, W, tokens=toks, quant_act=True)
    # the same 4-bit codes: what is left is f32 accumulation, and a code step where a SwiGLU value lies on a boundary
    assert errors(out[toks], ref)[1] < 5e-3
    assert (np.abs(out[toks] - ref) > 2e-2).mean() <= 1e-3
    assert layer.status() == 0
    layer.close()
