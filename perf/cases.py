"""The work that users of this library have it do, as measurable cases: the MoE layer from one token to a
prefill batch (with its wide-expert shape and its 4-bit-activation option), the decoder step, and the engine's
own three systems (water step, denoiser, path tracer).

`listed()` holds fixed cases, `draw(rng)` makes more of the same ranges; `prepare(case, seed)` builds what a
program holds before the call, `run(state)` is one pass through the public entry points, `work(case)` and
`tolerance(case)` say what one pass cannot do without and how far two correct implementations may differ.
Shapes and value distributions are those of bench.py and neonengine_b200/*synth.py; the tensors are drawn on the
GPU so that a state is made in well under a second."""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from neonengine_b200 import pt_synth, water_synth
from neonengine_b200.decoder_synth import AttentionWeights, DecoderShape
from neonengine_b200.decoder_system import DecoderSystem
from neonengine_b200.moe_layer_system import MoeLayerSystem
from neonengine_b200.path_tracer import PathTracer
from neonengine_b200.svgf_denoiser import SvgfDenoiser
from neonengine_b200.synth import MoeShape, MoeWeights, zipf_logit_bias
from neonengine_b200.water_physics import WaterPhysics

DEV = "cuda:0"


def _moe(name, tokens, experts=32, zipf=False, mxf4=False):
    return {"name": name, "kind": "moe", "tokens": tokens, "experts": experts, "zipf": zipf, "mxf4": mxf4}


def listed():
    return [
        # one user's next token: four experts' weights stream by, latency is everything
        _moe("moe decode 1", 1),
        # a handful of sequences (or drafted tokens of one), a size no tile was made for
        _moe("moe decode 5", 5),
        # a serving batch with the skewed expert loads of real routers
        _moe("moe decode 64 skewed", 64, zipf=True),
        # a prompt chunk or a busy server's mixed batch: ragged, between decode and prefill
        _moe("moe chunk 300", 300),
        # prompt processing
        _moe("moe prefill 4096", 4096),
        # the same with the 4-bit activations a user may choose
        _moe("moe prefill 4096 mxf4", 4096, mxf4=True),
        # the wide-expert layer's largest pass
        _moe("moe 128 experts 8192", 8192, experts=128),
        # one conversation through the whole stack, in the middle of its context
        {"name": "decoder batch 1", "kind": "decoder", "batch": 1, "position": 1500, "layers": 24},
        # a full batch at the end of its context
        {"name": "decoder batch 8", "kind": "decoder", "batch": 8, "position": 4095, "layers": 24},
        # the engine's water demo, one simulation step of a running simulation
        {"name": "water 8000", "kind": "water", "side": 20, "substeps": 4, "iterations": 50},
        # denoising one video frame
        {"name": "denoise 1080p", "kind": "denoise", "width": 1920, "height": 1080, "iterations": 3},
        # one frame of the path tracer in the engine's window
        {"name": "path trace 800x600", "kind": "trace", "width": 800, "height": 600, "lights": 50},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["moe"] * 6 + ["moe128", "decoder", "decoder", "water", "denoise", "trace"])
    if kind == "moe":
        mxf4 = rng.random() < 0.15
        c = _moe("", _log_int(rng, 256 if mxf4 else 1, 6000), zipf=rng.random() < 0.4, mxf4=mxf4)
    elif kind == "moe128":
        c = _moe("", _log_int(rng, 1, 6000), experts=128, zipf=rng.random() < 0.4)
    elif kind == "decoder":
        c = {"kind": "decoder", "batch": rng.randint(1, 8), "position": _log_int(rng, 30, 4095), "layers": rng.randint(6, 24)}
    elif kind == "water":
        c = {"kind": "water", "side": rng.randint(10, 28), "substeps": rng.choice([2, 4]), "iterations": rng.randint(20, 60)}
    elif kind == "denoise":
        c = {"kind": "denoise", "width": rng.randint(320, 1920), "height": rng.randint(200, 1080), "iterations": rng.choice([2, 3, 3, 3, 4])}
    else:
        c = {"kind": "trace", "width": rng.randint(160, 800), "height": rng.randint(120, 600), "lights": rng.randint(6, 50)}
    c.pop("name", None)
    return c


# ---- the MoE layer ----------------------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _normal(g, dims, std, mean=0.0):
    return (torch.randn(dims, generator=g, device=DEV) * std + mean).to(torch.bfloat16)


def _bytes(g, dims):
    """Uniform bytes: two e2m1 codes each, all sixteen codes alike."""
    n = math.prod(dims)
    words = torch.randint(-2**63, 2**63 - 1, ((n + 7) // 8,), generator=g, device=DEV, dtype=torch.int64)
    return words.view(torch.uint8)[:n].view(dims)


def _scales(g, dims, largest=-4):
    """E8M0 bytes with the seven exponents up to the largest."""
    return torch.randint(121 + largest, 128 + largest, dims, generator=g, device=DEV, dtype=torch.uint8)


def _moe_weights(g, s, down_largest=-4):
    E, H, I = s.n_experts, s.hidden, s.inter
    return MoeWeights(s, _normal(g, (E, H), 0.02), _normal(g, (E,), 0.02),
                      _bytes(g, (E, 2 * I, H // 2)), _scales(g, (E, 2 * I, H // 32)), _normal(g, (E, 2 * I), 0.02),
                      _bytes(g, (E, H, I // 2)), _scales(g, (E, H, I // 32), down_largest), _normal(g, (E, H), 0.02))


def _hidden(g, tokens, w, bias):
    """N(0, 1) rows whose k + 1 largest router logits lie 1e-4 apart (redrawn until they do, as the package's own
    generator does): below that, which expert comes first is a matter of summation order."""
    k = w.shape.top_k
    x = _normal(g, (tokens, w.shape.hidden), 1.0)
    for _ in range(32):
        logits = x.double() @ w.router_w.double().T + w.router_b.double() + (0.0 if bias is None else bias.double())
        top = logits.topk(k + 1, dim=1).values
        close = ((top[:, :-1] - top[:, 1:]).min(dim=1).values < 1e-4).nonzero().flatten()
        if not len(close):
            return x
        x[close] = _normal(g, (len(close), w.shape.hidden), 1.0)
    raise RuntimeError("could not separate the router logits")


def _prepare_moe(case, seed):
    g = _generator(seed)
    shape = MoeShape(n_experts=case["experts"])
    w = _moe_weights(g, shape)
    bias = torch.from_numpy(zipf_logit_bias(case["experts"])).to(DEV) if case["zipf"] else None
    layer = MoeLayerSystem(shape, None, max_tokens=case["tokens"])
    tensors = (w.router_w, w.router_b, w.gate_up_blocks, w.gate_up_scales, w.gate_up_bias, w.down_blocks, w.down_scales, w.down_bias)
    torch.cuda.synchronize()
    rc = layer._lib.neon_moe_set_weights(layer._h, *(ctypes.c_void_p(t.data_ptr()) for t in tensors), 1)  # weights on the device
    if rc:
        raise RuntimeError("neon_moe_set_weights failed (%d)" % rc)
    if case["mxf4"]:
        layer.set_option("mxf4_prefill", 1)
    hidden = _hidden(g, case["tokens"], w, bias)
    out = torch.empty((case["tokens"], shape.hidden), dtype=torch.float32, device=DEV)
    return {"kind": "moe", "layer": layer, "hidden": hidden, "bias": bias, "out": out}


def _touched(case):
    """Experts that a batch can be expected to touch."""
    E, n = case["experts"], case["tokens"]
    p = np.arange(1, E + 1) ** -1.1 if case["zipf"] else np.ones(E)
    p = p / p.sum()
    return float((1 - (1 - np.minimum(1.0, MoeShape().top_k * p)) ** n).sum())


def _moe_work(case):
    s = MoeShape(n_experts=case["experts"])
    n = case["tokens"]
    return {"bytes": _touched(case) * s.expert_bytes + s.router_bytes + n * s.hidden * 6,
            "flops": n * s.top_k * s.flops_per_pair + 2 * n * s.hidden * s.n_experts}


# ---- the decoder ------------------------------------------------------------------------------------------------
# As in a trained network, the residual stream is of the embedding's order and every MoE layer adds a percent to it:
# the embedding is N(0, 1) and the down products' block scales are 2**-11 of the single layer's.  (With layers that
# outweigh the stream, one expert swapped for its near equal in some layer would move the logits by half.)
def _prepare_decoder(case, seed):
    g = _generator(seed)
    s = DecoderShape(n_layers=case["layers"])
    B, pos, H = case["batch"], case["position"], s.hidden
    dec = DecoderSystem(s, B, 4096)
    dec.set_embeddings(_normal(g, (s.vocab, H), 1.0), _normal(g, (s.vocab, H), 0.02), _normal(g, (H,), 0.1, 1.0))
    for layer in range(s.n_layers):
        dec.set_attention(layer, AttentionWeights(
            ln1=_normal(g, (H,), 0.1, 1.0), wqkv=_normal(g, (s.qkv_rows, H), 0.02), bqkv=_normal(g, (s.qkv_rows,), 0.02),
            sinks=_normal(g, (s.n_q_heads,), 1.0), wo=_normal(g, (H, s.q_dim), 0.02), bo=_normal(g, (H,), 0.02),
            ln2=_normal(g, (H,), 0.1, 1.0)))
        dec.set_moe(layer, _moe_weights(g, s.moe, down_largest=-15))
        dec.load_kv(layer, *(_normal(g, (B, pos, s.n_kv_heads, s.head_dim), 1.0) for _ in range(2)))
    tokens = torch.randint(0, s.vocab, (B,), generator=g, device=DEV, dtype=torch.int32)
    return {"kind": "decoder", "dec": dec, "tokens": tokens,
            "positions": torch.full((B,), pos, device=DEV, dtype=torch.int32),
            "logits": torch.empty((B, s.vocab), device=DEV), "next": torch.empty((B,), device=DEV, dtype=torch.int32)}


def _decoder_work(case):
    s = DecoderShape()
    B, ctx, L = case["batch"], case["position"] + 1, case["layers"]
    dense = L * (s.qkv_rows * s.hidden + s.hidden * s.q_dim) + s.vocab * s.hidden
    seen = [min(ctx, s.window) if layer % 2 == 0 else ctx for layer in range(L)]
    kv = B * sum(seen) * 2 * s.n_kv_heads * s.head_dim
    moe = _moe_work({"experts": s.moe.n_experts, "tokens": B, "zipf": False})
    return {"bytes": 2 * dense + 2 * kv + L * moe["bytes"] + B * s.vocab * 4,
            "flops": 2 * B * dense + 4 * B * sum(seen) * s.q_dim + L * moe["flops"]}


# ---- the engine's own systems -----------------------------------------------------------------------------------
class _DeviceArray:
    """The library's own particle buffer, as torch can look at it; it keeps the simulation that owns it."""

    def __init__(self, owner, address, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (address, False), "version": 3}


def _prepare_water(case, seed):
    cfg = water_synth.WaterConfig(particles_per_side=case["side"], collision_substeps=case["substeps"],
                                  jacobi_iterations=case["iterations"])
    # the engine's spawn: a lattice inside the box, jittered
    n, f = cfg.particles_per_side, np.float32
    rng = np.random.default_rng(seed)
    lo, hi = (np.array(b, f) * f(0.9) for b in (cfg.box_min, cfg.box_max))
    lo, hi = lo + f(cfg.cell_size), hi - f(cfg.cell_size)
    z, y, x = np.meshgrid(*(np.arange(n),) * 3, indexing="ij")
    at = np.stack([x, y, z], -1).reshape(-1, 3).astype(f) / f(n - 1)
    pos = np.ones((n**3, 4), f)
    pos[:, :3] = lo + at * (hi - lo) + (rng.random((n**3, 3), dtype=f) - f(0.5)) * f(0.396)
    sim = WaterPhysics(cfg, pos)
    sim.run_simulation(400)  # under way: the water has fallen and sloshes
    views = [torch.as_tensor(_DeviceArray(sim, p, (n**3, 4)), device=DEV) for p in sim.device_pointers()]
    return {"kind": "water", "sim": sim, "views": views, "stream": torch.cuda.current_stream()}


def _frame(case, index, g):
    """One G-buffer and noisy image: floor, back wall and two spheres, the camera sliding sideways (the scene of
    neonengine_b200/svgf_synth.py, drawn on the GPU)."""
    w, h, f, pan = case["width"], case["height"], 1.2, 0.01
    ys, xs = torch.meshgrid((0.5 - (torch.arange(h, device=DEV, dtype=torch.float64) + 0.5) / h) / f,
                            ((torch.arange(w, device=DEV, dtype=torch.float64) + 0.5) / w - 0.5) * (w / h) / f, indexing="ij")
    d = torch.stack([xs, ys, -torch.ones_like(xs)], -1)
    d = d / d.norm(dim=-1, keepdim=True)
    o = torch.tensor([pan * index, 0.0, 0.0], device=DEV, dtype=torch.float64)
    best = torch.full((h, w), float("inf"), device=DEV, dtype=torch.float64)
    normal = torch.zeros((h, w, 4), device=DEV, dtype=torch.float64)

    def take(t, n, ident, ok):
        hit = ok & (t > 1e-3) & (t < best)
        best[hit] = t[hit]
        normal[..., :3] = torch.where(hit[..., None], n, normal[..., :3])
        normal[..., 3] = torch.where(hit, float(ident), normal[..., 3])

    vec = lambda *v: torch.tensor(v, device=DEV, dtype=torch.float64)  # noqa: E731
    t = -1.0 / d[..., 1]
    take(t, vec(0.0, 1.0, 0.0), 1, torch.isfinite(t) & (t * d[..., 2] > -7.0))
    t = -7.0 / d[..., 2]
    take(t, vec(0.0, 0.0, 1.0), 2, t * d[..., 1] < 1.2)
    for ident, c, r in ((3, vec(-0.8, -0.4, -4.0), 0.6), (4, vec(1.1, -0.55, -3.2), 0.45)):
        oc = o - c
        b = (d * oc).sum(-1)
        disc = b * b - ((oc * oc).sum() - r * r)
        t = -b - disc.clamp_min(0.0).sqrt()
        take(t, (o + t[..., None] * d - c) / r, ident, disc > 0)
    hit = normal[..., 3] > 0
    cam = torch.where(hit[..., None], best.nan_to_num(posinf=0.0)[..., None] * d, 0.0)
    position = torch.cat([cam, hit[..., None].double()], -1)
    bary = torch.zeros_like(position)
    bary[..., :3] = torch.where(hit[..., None], 0.5 + 0.3 * torch.sin(0.5 * (cam + o) + vec(0.0, 1.0, 2.0)), 0.0)
    depth = torch.where(hit, -cam[..., 2], 1.0)
    motion = torch.zeros_like(position)
    u, v = (torch.arange(w, device=DEV) + 0.5) / w, (torch.arange(h, device=DEV) + 0.5) / h
    motion[..., 0] = torch.where(hit, u - (0.5 + (cam[..., 0] + pan) / depth * f * (h / w)), 0.0)
    motion[..., 1] = torch.where(hit, v[:, None] - (0.5 - cam[..., 1] / depth * f), 0.0)
    light = vec(0.4, 0.8, 0.45)
    albedo = torch.tensor([[0, 0, 0], [0.7, 0.7, 0.65], [0.3, 0.5, 0.8], [0.9, 0.3, 0.2], [0.3, 0.8, 0.3]], device=DEV, dtype=torch.float64)
    shade = (normal[..., :3] @ (light / light.norm())).clamp_min(0.1)[..., None] * albedo[normal[..., 3].long()]
    radiance = torch.where(hit[..., None], shade, vec(0.35, 0.55, 0.9))
    radiance = radiance + 0.15 * torch.randn((h, w, 3), generator=g, device=DEV) * hit[..., None]
    image = torch.full((h, w, 4), 255, device=DEV, dtype=torch.uint8)
    image[..., :3] = (radiance.clamp(0.0, 1.0) * 255.0).round().to(torch.uint8)
    return [a.float().contiguous() for a in (position, normal, bary, motion)], image


def _prepare_denoise(case, seed):
    g = _generator(seed)
    dn = SvgfDenoiser(case["width"], case["height"], case["iterations"])
    index = 1 + seed % 40
    for i in (index, index + 1):  # two frames of history
        gbuffer, image = _frame(case, i, g)
        dn.render(gbuffer, image)
    gbuffer, image = _frame(case, index + 2, g)
    return {"kind": "denoise", "dn": dn, "gbuffer": gbuffer, "traced": image, "image": image.clone(),
            "stream": torch.cuda.current_stream()}


def _prepare_trace(case, seed):
    scene = pt_synth.cornell_box(seed, n_lights=case["lights"])
    rng = np.random.default_rng(seed)
    at = (0.0444 + 0.05 * rng.standard_normal(), -0.7041 + 0.05 * rng.standard_normal(), -1.1978)
    camera = pt_synth.camera(case["width"], case["height"], position=at)
    image = torch.empty((case["height"], case["width"], 4), dtype=torch.uint8, device=DEV)
    return {"kind": "trace", "tracer": PathTracer(scene, case["width"], case["height"]), "camera": camera, "frame": seed % 1000, "image": image}


# ---- one interface over all kinds -------------------------------------------------------------------------------
def prepare(case, seed):
    make = {"moe": _prepare_moe, "decoder": _prepare_decoder, "water": _prepare_water, "denoise": _prepare_denoise, "trace": _prepare_trace}
    return make[case["kind"]](case, seed)


def run(state):
    kind = state["kind"]
    if kind == "moe":
        return state["layer"].run(state["hidden"], logit_bias=state["bias"], out=state["out"])
    if kind == "decoder":
        state["dec"].step(state["tokens"], state["positions"], logits=state["logits"], next_tokens=state["next"])
        return state["logits"]  # the next tokens are their argmax, and a matter of ties where logits differ in their last bits
    if kind == "water":
        state["sim"].run_simulation(1, stream=state["stream"])
        return state["views"]
    if kind == "denoise":
        state["image"].copy_(state["traced"])  # the path tracer's frame arrives; the denoiser works in place
        state["dn"].render(state["gbuffer"], state["image"], stream=state["stream"])
        return state["image"]
    state["frame"] += 1  # every frame is a new sample of the scene
    return state["tracer"].render(*state["camera"], float(state["frame"]), image=state["image"])


def work(case):
    kind = case["kind"]
    if kind == "moe":
        return _moe_work(case)
    if kind == "decoder":
        return _decoder_work(case)
    if kind == "water":
        cfg = water_synth.WaterConfig(particles_per_side=case["side"])
        return {"bytes": cfg.n_particles * 64, "flops": cfg.n_cells * case["iterations"] * 12}
    pixels = case["width"] * case["height"]
    if kind == "denoise":  # G-buffer and image in, history colour and moments in and out, image out; 25 taps of about 40 operations
        return {"bytes": pixels * (64 + 4 + 2 * (8 + 16) + 4), "flops": pixels * case["iterations"] * 25 * 40}
    triangles = 12 * 4 + case["lights"] * 224
    return {"bytes": pixels * 4 + triangles * 3 * 64, "flops": 0}


def tolerance(case):
    if case["kind"] == "moe":
        # against 64-bit sums: 1e-6 with the four-term activations of small passes, 1.5e-5 with the three-term ones of
        # large passes; with 4-bit activations 4e-7, and a value at a rounding tie moves its row by a percent
        if case["mxf4"]:
            return {"rel": 1e-4, "max": 2e-2}
        return {"rel": 5e-6 if case["tokens"] <= 224 else 6e-5}
    if case["kind"] == "decoder":
        # bf16 activations between the layers: 0.4 % from their rounding, a percent where a near tie routes the other way
        return {"rel": 2e-2, "max": 0.3}
    return "exact"  # bit for bit what the engine's shaders compute
