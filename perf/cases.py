"""Performance cases of the quantized DiT hot path: the work a user of this framework has it do,
through its public entry points.

A case is a dict of plain values; its ``kind`` says which entry point it calls:

* ``linear``        ``ops.w8a8_linear``: one int8-convrot Linear of a block (quantise + INT8 GEMM).
* ``quantize``      ``ops.quantize_int8_rows``: activation codes for a Linear whose input is a concatenation.
* ``norm_quantize`` ``ops.rms_norm_modulate_quant`` / ``ops.layer_norm_modulate_quant``.
* ``pack``          ``ops.quantize_weight_rows``: packing one bf16 checkpoint matrix.
* ``attention``     ``ops.attention``: bf16 q / k / v through the INT8 lowering, GQA and key mask.
* ``video_block``   ``VideoBlock.forward``: the whole video DiT block on device-resident tensors.
* ``mmdit_plugin``  ``PreparedExecution.run``: the MMDiT double-stream block as a DiffIR program behind
                    the backend plugin, host arrays in and out.
* ``video_plugin``  the same for the video block, with page-locked host arrays.

Widths are those of the benchmark configurations (hidden 3072, 24 heads of 128, MLP 12288, FFN
8192); token counts span one row to the 33272 tokens of the video benchmark.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from diffusion_compiler_b200 import blocks, ops, plugin
from diffusion_compiler_b200.sequence_shard import GatherBuffers, ShardPlan, VideoBlock

HIDDEN, HEADS, DIM, MLP, FFN, ROTARY = 3072, 24, 128, 12288, 8192, 96
VIDEO_TOKENS = 21 * 30 * 52 + 512
H256 = 2  # Int8RowQuantization: unsigned 256-wide ConvRot, the default of the rewrite

# The linears of the two blocks: (K, N, bias, gelu)
LINEARS = [
    (HIDDEN, 3 * HIDDEN, True, False),   # fused QKV of the MMDiT block
    (HIDDEN, HIDDEN, True, False),       # its output projection
    (HIDDEN, MLP, True, True),           # MLP up, GELU in the epilogue
    (MLP, HIDDEN, True, False),          # MLP down
    (HIDDEN, HIDDEN, False, False),      # q / k / v / o of the video block
    (HIDDEN, 2 * FFN, False, False),     # fc1 (SwiGLU)
    (FFN, HIDDEN, False, False),         # fc2
]


def listed():
    return [
        # a conditioning vector at batch 2 (CFG): the smallest call there is, two kernels
        {"name": "linear_vector", "kind": "linear", "rows": 2, "k": HIDDEN, "n": HIDDEN, "bias": True, "gelu": False},
        # the text stream of one image: 512 tokens through MLP up
        {"name": "linear_text", "kind": "linear", "rows": 512, "k": HIDDEN, "n": MLP, "bias": True, "gelu": True},
        # one rank's slice of the video block on eight GPUs: fc2 on a ragged row count
        {"name": "linear_slice", "kind": "linear", "rows": 4159, "k": FFN, "n": HIDDEN, "bias": False, "gelu": False},
        # both streams of a 1024 x 1024 image at batch 2 (CFG) through the fused QKV projection
        {"name": "linear_image", "kind": "linear", "rows": 9216, "k": HIDDEN, "n": 3 * HIDDEN, "bias": True,
         "gelu": False},
        # the second linear of a single-stream block reads attention and MLP outputs side by side
        {"name": "quantize_concat", "kind": "quantize", "rows": 4608, "widths": "3072,12288", "variant": H256,
         "residual": False},
        # norm + modulate + quantise in front of the projections, a quarter of the video's tokens
        {"name": "norm_rms_video", "kind": "norm_quantize", "rows": 8318, "layer": False, "per_modulation": 1},
        # offline packing of one MLP matrix with the packer's scale search and input equalisation
        {"name": "pack_mlp", "kind": "pack", "n": MLP, "k": HIDDEN, "variant": H256, "mse": True, "equalise": True},
        # a small image with 77 text tokens, some of them padding: GQA and a key mask
        {"name": "attention_small", "kind": "attention", "batch": 1, "tokens": 1101, "kv_heads": 8, "masked": 51},
        # joint attention of a 1024 x 1024 image at batch 2
        {"name": "attention_image", "kind": "attention", "batch": 2, "tokens": 4608, "kv_heads": HEADS, "masked": 0},
        # the video benchmark's block, tensors resident on the device
        {"name": "block_video", "kind": "video_block", "tokens": VIDEO_TOKENS},
        # a 256 x 256 image through the backend plugin: ordinary host arrays, one call per block
        {"name": "plugin_mmdit_small", "kind": "mmdit_plugin", "batch": 1, "side": 16, "text": 77},
        # a shorter clip (9 latent frames) through the backend plugin: page-locked host arrays
        {"name": "plugin_video", "kind": "video_plugin", "tokens": 9 * 30 * 52 + 512},
    ]


def _spread(rng, low, high):
    """A size spread over the logarithm of [low, high]; odd sizes are as likely as even ones."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "quantize", "norm_quantize", "pack", "attention", "attention",
                       "video_block", "mmdit_plugin", "video_plugin"])
    if kind == "linear":
        k, n, bias, gelu = rng.choice(LINEARS)
        return {"kind": kind, "rows": _spread(rng, 1, VIDEO_TOKENS), "k": k, "n": n, "bias": bias, "gelu": gelu}
    if kind == "quantize":
        variant = rng.choice([2, 2, 3, 4, 5, 6, 7])
        widths = rng.choice(["4096", "12288", "8192"] if variant in (4, 7) else
                            ["3072", "8192", "12288", "3072,12288", "3072,8192"])
        return {"kind": kind, "rows": _spread(rng, 16, 16384), "widths": widths, "variant": variant,
                "residual": rng.random() < 0.2}
    if kind == "norm_quantize":
        layer = rng.random() < 0.5
        shared = rng.choice([1, 2]) if layer else 1  # modulation rows: one per batch entry, or one per token
        rows = _spread(rng, 16, 16384)
        return {"kind": kind, "rows": rows * shared, "layer": layer, "per_modulation": rows if layer else 1}
    if kind == "pack":
        k, n, _, _ = rng.choice(LINEARS)
        return {"kind": kind, "n": n, "k": k, "variant": rng.choice([2, 2, 3, 5, 6]), "mse": rng.random() < 0.5,
                "equalise": rng.random() < 0.5}
    if kind == "attention":
        tokens = _spread(rng, 64, 12288)
        masked = rng.randrange(1, max(2, min(128, tokens // 2))) if rng.random() < 0.4 else 0
        return {"kind": kind, "batch": rng.choice([1, 2]), "tokens": tokens, "kv_heads": rng.choice([HEADS, HEADS, 8]),
                "masked": masked}
    if kind == "video_block":
        return {"kind": kind, "tokens": _spread(rng, 512, VIDEO_TOKENS)}
    if kind == "mmdit_plugin":
        return {"kind": kind, "batch": rng.choice([1, 2]), "side": rng.randrange(8, 65), "text": rng.choice([77, 256, 512])}
    return {"kind": kind, "tokens": _spread(rng, 1024, 16384)}


# ---- inputs: seeded, made on the device --------------------------------------------------------
def _normal(g, shape, std=1.0):
    return (torch.randn(shape, generator=g, device="cuda", dtype=torch.float32) * std).to(torch.bfloat16)


def _activations(g, rows, width):
    """N(0,1) with 32 channels sixteen times as large, the outliers ConvRot is there for."""
    x = torch.randn((rows, width), generator=g, device="cuda", dtype=torch.float32)
    x[:, torch.randperm(width, generator=g, device="cuda")[:32]] *= 16.0
    return x.to(torch.bfloat16)


def _packed_linear(g, n, k):
    """Weights N(0, 0.02) packed by the weight-side transform: (codes, column scales)."""
    return ops.quantize_int8_rows([_normal(g, (n, k), 0.02)], H256)


def _bits(t):
    """The uint16 bit patterns of a bf16 tensor as a host array (ordinary memory)."""
    return t.contiguous().view(torch.int16).cpu().numpy().view(np.uint16)


def _pinned_bits(t):
    host = torch.empty(t.shape, dtype=torch.int16, pin_memory=True)
    host.copy_(t.contiguous().view(torch.int16))
    return host.numpy().view(np.uint16)


def _modulations(g, rows):
    """Six modulation tensors, every row the same vector: a conditioning vector through a random map."""
    cond = torch.randn(64, generator=g, device="cuda")
    maps = torch.randn((6, HIDDEN, 64), generator=g, device="cuda") * 0.02
    return [v.to(torch.bfloat16)[None, :].expand(rows, HIDDEN).contiguous() for v in maps @ cond]


def _video_linears(g):
    shapes = {"q": (HIDDEN, HIDDEN), "k": (HIDDEN, HIDDEN), "v": (HIDDEN, HIDDEN), "o": (HIDDEN, HIDDEN),
              "fc1": (2 * FFN, HIDDEN), "fc2": (HIDDEN, FFN)}
    return {name: tuple(t.cpu().numpy() for t in _packed_linear(g, n, k)) for name, (n, k) in shapes.items()}


def _video_constants(tokens):
    """Norm weights and the 3-axis rotary tables of a clip of 30 x 52 latents per frame, then its text."""
    at = np.arange(tokens)
    text = min(512, tokens // 4)
    latent = tokens - text
    positions = np.stack([at // 1560, (at // 52) % 30, at % 52], axis=1).astype(np.float32)
    positions[latent:] = 0
    positions[latent:, 0] = np.arange(text)
    cos, sin = blocks.rope_tables_3axis(positions, ROTARY)
    ones = lambda n: blocks.f32_to_bf16(np.ones(n, np.float32))  # noqa: E731
    return {"norm1": ones(HIDDEN), "norm2": ones(HIDDEN), "q_norm": ones(DIM), "k_norm": ones(DIM), "cos": cos,
            "sin": sin}


# ---- prepare / run per kind --------------------------------------------------------------------
def _prepare_linear(case, g):
    x = _activations(g, case["rows"], case["k"])
    w8, scales = _packed_linear(g, case["n"], case["k"])
    return {"x": x, "w8": w8, "scales": scales, "bias": _normal(g, (case["n"],), 0.01) if case["bias"] else None,
            "gelu": case["gelu"]}


def _run_linear(s):
    return ops.w8a8_linear(s["x"], s["w8"], s["scales"], bias=s["bias"], gelu=s["gelu"])


def _prepare_quantize(case, g):
    parts = [_activations(g, case["rows"], int(w)) for w in case["widths"].split(",")]
    return {"parts": parts, "variant": case["variant"], "residual": case["residual"]}


def _run_quantize(s):
    return ops.quantize_int8_rows(s["parts"], s["variant"], residual=s["residual"])


def _prepare_norm_quantize(case, g):
    x = _activations(g, case["rows"], HIDDEN)
    weight = (1.0 + 0.1 * torch.randn(HIDDEN, generator=g, device="cuda")).to(torch.bfloat16)
    mod_rows = case["rows"] // case["per_modulation"]
    s = {"layer": case["layer"], "x": x, "weight": weight, "scale": _normal(g, (mod_rows, HIDDEN), 0.1),
         "shift": _normal(g, (mod_rows, HIDDEN), 0.1)}
    if case["layer"]:
        s["bias"] = _normal(g, (HIDDEN,), 0.1)
    return s


def _run_norm_quantize(s):
    if s["layer"]:
        return ops.layer_norm_modulate_quant(s["x"], s["weight"], s["bias"], s["scale"], s["shift"], 1e-6)
    return ops.rms_norm_modulate_quant(s["x"], s["weight"], s["scale"], s["shift"])


def _prepare_pack(case, g):
    gains = torch.exp(0.5 * torch.randn(case["k"], generator=g, device="cuda"))  # uneven input channels
    w = (torch.randn((case["n"], case["k"]), generator=g, device="cuda") * 0.02 * gains).to(torch.bfloat16)
    return {"w": w, "variant": case["variant"], "mse": case["mse"],
            "eq": ops.weight_equalization(w) if case["equalise"] else None}


def _run_pack(s):
    return ops.quantize_weight_rows(s["w"], s["variant"], mse_scale=s["mse"], input_scale=s["eq"])


def _prepare_attention(case, g):
    B, S, KV = case["batch"], case["tokens"], case["kv_heads"]

    def normed(heads):  # what QK-norm leaves: every head row with unit mean square
        t = torch.randn((B, S, heads, DIM), generator=g, device="cuda")
        return (t * torch.rsqrt(t.square().mean(-1, keepdim=True) + 1e-6)).to(torch.bfloat16)

    valid = None
    if case["masked"]:
        valid = torch.ones((B, S), dtype=torch.uint8, device="cuda")
        valid[:, : case["masked"]] = 0  # padded text comes first in the joint sequence
    return {"q": normed(HEADS), "k": normed(KV), "v": _normal(g, (B, S, KV, DIM)), "valid": valid}


def _run_attention(s):
    return ops.attention(s["q"], s["k"], s["v"], key_valid=s["valid"])


def _prepare_video_block(case, g):
    S = case["tokens"]
    tensors = dict(_video_constants(S), linears=_video_linears(g))
    block = VideoBlock(tensors, HIDDEN, HEADS, DIM, FFN, ROTARY, torch.device("cuda"))
    plan = ShardPlan.make(S, 1)
    return {"block": block, "plan": plan, "gb": GatherBuffers(plan, 0, HEADS, DIM, torch.device("cuda")),
            "x": _normal(g, (S, HIDDEN)), "mods": _modulations(g, S)}


def _run_video_block(s):
    return s["block"].forward(s["x"], s["mods"], s["plan"], 0, gb=s["gb"])


def _prepare_mmdit_plugin(case, g):
    B, side, text = case["batch"], case["side"], case["text"]
    program, ids = blocks.mmdit_double_stream_program(B, side * side, text, HIDDEN, HEADS, DIM, MLP)
    consts = {}
    for w, cs, b, n, k in ids["linears"].values():
        codes, scales = _packed_linear(g, n, k)
        consts[w], consts[cs] = codes.cpu().numpy(), scales.cpu().numpy()
        consts[b] = _bits(_normal(g, (n,), 0.01))
    for t in ids["qk_scales"].values():
        consts[t] = blocks.f32_to_bf16(np.ones(DIM, np.float32))
    consts[ids["pair_axes"]], consts[ids["pair_indices"]], consts[ids["axis_dims"]] = blocks.rope_pair_maps(
        ids["axes_dims"])
    inputs = {ids["image"]: _bits(_normal(g, (B, side * side, HIDDEN))),
              ids["text"]: _bits(_normal(g, (B, text, HIDDEN))),
              ids["positions"]: blocks.image_positions_2axis(B, text, (side, side))}
    for key in ("image_mod", "text_mod"):
        vec = torch.stack([m[0] for m in _modulations(g, 1)])
        inputs[ids[key]] = _bits(vec[None].expand(B, 6, HIDDEN))
    executor = plugin.PluginExecutor(0)
    return {"executor": executor, "prepared": executor.prepare(program, consts), "inputs": inputs,
            "outputs": (ids["image_out"], ids["text_out"])}


def _run_mmdit_plugin(s):
    out, _ = s["prepared"].run(s["inputs"])
    return [torch.from_numpy(out[t].view(np.int16)).view(torch.bfloat16) for t in s["outputs"]]


def _prepare_video_plugin(case, g):
    S = case["tokens"]
    program, ids = blocks.video_block_program(S, HIDDEN, HEADS, DIM, FFN, ROTARY)
    consts = {ids[name]: a for name, a in _video_constants(S).items()}
    for name, (codes, scales) in _video_linears(g).items():
        w, cs = ids["linears"][name][:2]
        consts[w], consts[cs] = codes, scales
    inputs = {ids["x"]: _pinned_bits(_normal(g, (S, HIDDEN)))}
    for t, m in zip(ids["mods"], _modulations(g, S)):
        inputs[t] = _pinned_bits(m)
    out = torch.empty((S, HIDDEN), dtype=torch.bfloat16, pin_memory=True)
    executor = plugin.PluginExecutor(0)
    return {"executor": executor, "prepared": executor.prepare(program, consts), "inputs": inputs, "out": out,
            "outputs": {ids["out"]: out.view(torch.int16).numpy().view(np.uint16)}}


def _run_video_plugin(s):
    s["prepared"].run(s["inputs"], outputs=s["outputs"])
    return s["out"]


_PREPARE = {"linear": _prepare_linear, "quantize": _prepare_quantize, "norm_quantize": _prepare_norm_quantize,
            "pack": _prepare_pack, "attention": _prepare_attention, "video_block": _prepare_video_block,
            "mmdit_plugin": _prepare_mmdit_plugin, "video_plugin": _prepare_video_plugin}
_RUN = {"linear": _run_linear, "quantize": _run_quantize, "norm_quantize": _run_norm_quantize, "pack": _run_pack,
        "attention": _run_attention, "video_block": _run_video_block, "mmdit_plugin": _run_mmdit_plugin,
        "video_plugin": _run_video_plugin}


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    state = _PREPARE[case["kind"]](case, g)
    state["kind"] = case["kind"]
    return state


def run(state):
    return _RUN[state["kind"]](state)


# ---- what a pass cannot do without -------------------------------------------------------------
def _linear_work(rows, k, n, bias):
    return 2.0 * rows * k + n * k + 4.0 * n + (2.0 * n if bias else 0.0) + 2.0 * rows * n, 2.0 * rows * k * n


def _attention_work(batch, tokens, kv_heads):
    return (2.0 * batch * tokens * DIM * (2 * HEADS + 2 * kv_heads), 4.0 * batch * HEADS * tokens * tokens * DIM)


def _video_work(tokens):
    """Inputs, weights and output once; the six linears and the attention."""
    weights = 4.0 * HIDDEN * HIDDEN + 3.0 * FFN * HIDDEN
    read = 2.0 * 7 * tokens * HIDDEN + 2.0 * 2 * tokens * ROTARY + weights
    return read + 2.0 * tokens * HIDDEN, 2.0 * tokens * weights + _attention_work(1, tokens, HEADS)[1]


def work(case):
    kind = case["kind"]
    if kind == "linear":
        size, flops = _linear_work(case["rows"], case["k"], case["n"], case["bias"])
    elif kind == "quantize":
        k, rows = sum(int(w) for w in case["widths"].split(",")), case["rows"]
        stages = 6 if case["variant"] in (4, 7) else 4
        codes = (k + 4.0) * rows * (2 if case["residual"] else 1)
        size, flops = 2.0 * rows * k + codes, 2.5 * stages * rows * k
    elif kind == "norm_quantize":
        rows = case["rows"]
        mods = 2.0 * 2.0 * HIDDEN * (rows // case["per_modulation"])
        size, flops = 3.0 * rows * HIDDEN + 4.0 * rows + mods + 2.0 * HIDDEN, 16.0 * rows * HIDDEN
    elif kind == "pack":
        size, flops = 3.0 * case["n"] * case["k"] + 4.0 * case["n"], 10.0 * case["n"] * case["k"]
    elif kind == "attention":
        size, flops = _attention_work(case["batch"], case["tokens"], case["kv_heads"])
    elif kind == "mmdit_plugin":
        B, image, text = case["batch"], case["side"] ** 2, case["text"]
        rows, per_token = B * (image + text), 4.0 * HIDDEN * HIDDEN + 2.0 * HIDDEN * MLP
        size = 2.0 * per_token + 2.0 * 2.0 * rows * HIDDEN + 8.0 * rows + 2.0 * 12 * B * HIDDEN
        flops = 2.0 * rows * per_token + _attention_work(B, image + text, HEADS)[1]
    else:
        size, flops = _video_work(case["tokens"])
    return {"bytes": size, "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind in ("quantize", "norm_quantize", "pack"):
        return "exact"  # codes and scales have the reference's bits
    if kind == "linear":
        return {"rel": 2e-3}  # exact INT32 sums, one bf16 rounding (three with bias and GELU)
    if kind == "attention":
        return {"rel": 5e-3}  # bf16 softmax weights and output, fp32 sums in any order
    # W8A8 linears behind the attention re-quantise: a difference d comes out as about sqrt(d * step)
    return {"rel": 1e-2}
