"""GPU: whole DiT blocks. (1) the video block and the MMDiT double-stream block as DiffIR programs
through the plugin against the reference CPU executor running the SAME program (its Attention is
exact, ours is the INT8 lowering, so the bar is the north star's bf16 tolerance, not bit-exact);
(2) the token-sharded video block, four ranks emulated one after another on one GPU, against the
unsharded block."""
import numpy as np
import pytest

import oracle_bridge as ob
from diffusion_compiler_b200 import blocks
from helpers import bf16_normal, cosine, rel_l2

pytestmark = pytest.mark.gpu


def _cpu_quantize(w_bits):
    return ob.orc().quantize_int8_rows([w_bits], 2)


@pytest.mark.skipif(not ob.ref_available(), reason="reference build (oracle/_ref) not present")
def test_video_block_through_plugin_matches_reference_executor():
    from diffusion_compiler_b200 import plugin
    rng = np.random.default_rng(4)
    S, hidden, heads, dim, ffn, rotary = 400, 512, 4, 128, 1024, 96
    p, ids, consts, inputs = blocks.synth_video_block(rng, S, hidden, heads, dim, ffn, rotary, _cpu_quantize)
    want, _ = ob.ref().run(p, {**consts, **inputs})
    ex = plugin.PluginExecutor(0)
    got, tel = ex.prepare(p, consts).run(inputs)
    a, b = ob.bf16_to_f32(got[ids["out"]]), ob.bf16_to_f32(want[ids["out"]])
    assert np.isfinite(a).all()
    assert rel_l2(a, b) <= 2e-3 and cosine(a, b) >= 0.9999, (rel_l2(a, b), cosine(a, b))
    ex.close()


def test_video_block_replayed_from_cuda_graphs_keeps_the_bits():
    """The block's kernels replayed from four CUDA graphs (captured on the first call for fixed
    tensors) give the bits of the kernel-by-kernel run, also after the inputs change in place."""
    import torch
    from diffusion_compiler_b200 import ops
    from diffusion_compiler_b200.sequence_shard import GatherBuffers, ShardPlan, VideoBlock
    rng = np.random.default_rng(8)
    S, hidden, heads, dim, ffn, rotary = 437, 512, 4, 128, 1024, 96
    p, ids, consts, inputs = blocks.synth_video_block(rng, S, hidden, heads, dim, ffn, rotary, _cpu_quantize)
    tensors = {"norm1": consts[ids["norm1"]], "norm2": consts[ids["norm2"]], "q_norm": consts[ids["q_norm"]],
               "k_norm": consts[ids["k_norm"]], "cos": consts[ids["cos"]], "sin": consts[ids["sin"]],
               "linears": {n: (consts[w], consts[cs]) for n, (w, cs, b, N, K) in ids["linears"].items()}}
    block = VideoBlock(tensors, hidden, heads, dim, ffn, rotary, "cuda")
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.int16)).cuda().view(torch.bfloat16)
    x = dev(inputs[ids["x"]])
    mods = [dev(inputs[m]) for m in ids["mods"]]
    plan = ShardPlan.make(S, 1)
    gb = GatherBuffers(plan, 0, heads, dim, "cuda")
    for trial in range(2):
        want = block.forward(x, mods, plan, 0, gb=gb).clone()
        got = block.forward(x, mods, plan, 0, gb=gb, graphs=True).clone()
        torch.cuda.synchronize()
        assert torch.equal(want.view(torch.int16), got.view(torch.int16))
        x.mul_(0.5)  # same storage, new values: the second trial replays the graphs of the first
    ops.poll_status()


@pytest.mark.parametrize("tokens", [2000, 4100, 8301])  # the last step as a whole, in two and in four blocks of rows
def test_video_block_with_page_locked_arrays_keeps_the_bits(tokens):
    """With page-locked arrays on both sides the gate of the last step comes in, and the output leaves, a block of rows at a
    time; with ordinary arrays, or only one side page-locked, as a whole. The same bits, for every input."""
    import torch
    from diffusion_compiler_b200 import plugin
    rng = np.random.default_rng(tokens)
    p, ids, consts, inputs = blocks.synth_video_block(rng, tokens, 1024, 8, 128, 256, 96, _cpu_quantize)
    ex = plugin.PluginExecutor(0)
    prepared = ex.prepare(p, consts)

    def locked(a):
        host = torch.empty(a.shape, dtype=torch.int16, pin_memory=True)
        host.numpy()[...] = a.view(np.int16)
        return host.numpy().view(np.uint16)

    for trial in range(3):
        want, _ = prepared.run(inputs)
        gate, want = inputs[ids["mods"][5]], want[ids["out"]]
        pinned = {t: locked(a) if a.dtype == np.uint16 else a for t, a in inputs.items()}
        for given, out in ((pinned, locked(np.full_like(want, 0x4000 + trial))), (pinned, np.zeros_like(want)), (inputs, locked(np.zeros_like(want)))):
            prepared.run(given, outputs={ids["out"]: out})
            assert np.array_equal(out, want)
        inputs = dict(inputs)
        inputs[ids["mods"][5]] = np.ascontiguousarray(gate[::-1])
        inputs[ids["x"]] = np.ascontiguousarray(inputs[ids["x"]][::-1])
    ex.close()


@pytest.mark.parametrize("case", ["shifted", "earlier output"])
def test_outputs_may_lie_on_the_last_gates_host_array(case):
    """Page-locked arrays that an Output has in common with the last step's gate: that Input is complete on the device before an Output
    that needs it, or an earlier one whose Inputs stand behind it in the program, overwrites it."""
    import torch
    from diffusion_compiler_b200 import diffir as ir
    from diffusion_compiler_b200 import plugin
    rows, width = 8192, 2048  # 32 MB: eight blocks of rows
    p = ir.Program()
    bf = ir.DType.BF16
    gate, first, a, b = (p.add_tensor(bf, [rows, width], ir.Role.Input) for _ in range(4))
    early, out = (p.add_tensor(bf, [rows, width], ir.Role.Output) for _ in range(2))
    p.add_op(ir.Opcode.ResidualGate, [a, b, first], [early])
    p.add_op(ir.Opcode.ResidualGate, [a, b, gate], [out])
    rng = np.random.default_rng(3)
    given = {t: bf16_normal(rng, (rows, width)) for t in (gate, first, a, b)}
    ex = plugin.PluginExecutor(0)
    prepared = ex.prepare(p, {})
    want, _ = prepared.run(given)
    host = torch.zeros((2, rows, width), dtype=torch.int16, pin_memory=True).numpy().view(np.uint16)
    flat = host.reshape(-1, width)
    locked = lambda x: np.ascontiguousarray(torch.from_numpy(x.view(np.int16)).pin_memory().numpy()).view(np.uint16)  # noqa: E731
    for _ in range(3):
        flat[:rows] = given[gate]
        bound = {t: locked(v) for t, v in given.items()}
        bound[gate] = flat[:rows]
        other = torch.zeros((rows, width), dtype=torch.int16, pin_memory=True).numpy().view(np.uint16)
        outputs = {early: other, out: flat[rows * 3 // 4:rows * 7 // 4]} if case == "shifted" else {early: flat[:rows], out: other}
        got, _ = prepared.run(bound, outputs=outputs)
        for t in (early, out):
            assert np.array_equal(got[t], want[t]), t
    ex.close()


def test_plugin_rope_fusions_keep_the_bits(monkeypatch):
    """The planner reads last-axis slices in place from QkNormPartialRope and lets that op write
    the attention kernel's INT8 q / k directly (through a Concat along tokens too). Same arithmetic,
    so the block output must not change by a bit against the unfused plan."""
    from diffusion_compiler_b200 import plugin
    rng = np.random.default_rng(6)
    p, ids, consts, inputs = blocks.synth_mmdit_block(rng, batch=2, grid=(8, 8), text_tokens=24, hidden=512, heads=4,
                                                     mlp=1024, quantize=_cpu_quantize)
    results = []
    for fusion in ("1", "0"):
        monkeypatch.setenv("DIFB200_ROPE_FUSION", fusion)
        ex = plugin.PluginExecutor(0)
        got, _ = ex.prepare(p, consts).run(inputs)
        ex.close()
        results.append(got)
    for key in ("image_out", "text_out"):
        assert np.array_equal(results[0][ids[key]], results[1][ids[key]])


def test_plugin_norm_quant_fusion_saves_the_normalised_tensor_and_stays_in_the_bar(monkeypatch):
    """RmsNormModulate -> QuantizeInt8Rows runs as one kernel in the plugin: the normalised tensors
    are not resident any more, and the block output stays well inside the path's bf16 bar against
    the plan with separate kernels (the row statistic is summed in another order, so single codes
    may move by one)."""
    from diffusion_compiler_b200 import plugin
    rng = np.random.default_rng(12)
    S, hidden, heads, dim, ffn, rotary = 400, 512, 4, 128, 1024, 96
    p, ids, consts, inputs = blocks.synth_video_block(rng, S, hidden, heads, dim, ffn, rotary, _cpu_quantize)
    results, resident = [], []
    monkeypatch.setenv("DIFB200_BUFFER_REUSE", "0")  # residency per tensor, so that the saved tensors show
    for fusion in ("1", "0"):
        monkeypatch.setenv("DIFB200_NORM_FUSION", fusion)
        ex = plugin.PluginExecutor(0)
        prepared = ex.prepare(p, consts)
        got, _ = prepared.run(inputs)
        resident.append(int(prepared.compile_telemetry.resident_bytes))
        ex.close()
        results.append(ob.bf16_to_f32(got[ids["out"]]))
    assert resident[1] - resident[0] >= 2 * S * hidden * 2  # two [S, hidden] bf16 tensors fewer
    assert rel_l2(results[0], results[1]) <= 5e-4 and cosine(results[0], results[1]) >= 0.99999


def test_plugin_buffer_reuse_keeps_the_bits_and_saves_memory(monkeypatch):
    """Internal tensors whose lifetimes do not overlap share device memory (the plugin's default):
    the same bits as with one allocation per tensor and fewer resident bytes,
    also when the same executable runs several passes."""
    from diffusion_compiler_b200 import plugin
    rng = np.random.default_rng(16)
    p, ids, consts, inputs = blocks.synth_mmdit_block(rng, batch=2, grid=(8, 8), text_tokens=24, hidden=512, heads=4,
                                                     mlp=1024, quantize=_cpu_quantize)
    results, resident = [], []
    for reuse in ("1", "0"):
        monkeypatch.setenv("DIFB200_BUFFER_REUSE", reuse)
        ex = plugin.PluginExecutor(0)
        prepared = ex.prepare(p, consts)
        got, _ = prepared.run(inputs, warmups=1, iterations=2)
        again, _ = prepared.run(inputs)
        resident.append(int(prepared.compile_telemetry.resident_bytes))
        ex.close()
        for key in ("image_out", "text_out"):
            assert np.array_equal(got[ids[key]], again[ids[key]])
        results.append(got)
    for key in ("image_out", "text_out"):
        assert np.array_equal(results[0][ids[key]], results[1][ids[key]])
    assert resident[0] < resident[1], resident


@pytest.mark.skipif(not ob.ref_available(), reason="reference build (oracle/_ref) not present")
def test_mmdit_double_stream_block_through_plugin_matches_reference_executor():
    from diffusion_compiler_b200 import plugin
    rng = np.random.default_rng(5)
    p, ids, consts, inputs = blocks.synth_mmdit_block(rng, batch=2, grid=(8, 8), text_tokens=24, hidden=512, heads=4,
                                                     mlp=1024, quantize=_cpu_quantize)
    want, _ = ob.ref().run(p, {**consts, **inputs})
    ex = plugin.PluginExecutor(0)
    got, _ = ex.prepare(p, consts).run(inputs)
    for key in ("image_out", "text_out"):
        a, b = ob.bf16_to_f32(got[ids[key]]), ob.bf16_to_f32(want[ids[key]])
        assert np.isfinite(a).all()
        assert rel_l2(a, b) <= 2e-3 and cosine(a, b) >= 0.9999, (key, rel_l2(a, b), cosine(a, b))
    ex.close()


def test_mmdit_block_at_batch_one_has_the_bits_of_batch_two():
    """At batch 1 the slices of the modulations and of the joint sequence are parts of their inputs' buffers, at batch 2 copies: the
    same image twice gives the same bits, also after other inputs."""
    from diffusion_compiler_b200 import plugin
    results = []
    for batch in (1, 2):
        rng = np.random.default_rng(15)
        p, ids, consts, inputs = blocks.synth_mmdit_block(rng, batch=batch, grid=(8, 6), text_tokens=19, hidden=512, heads=4, mlp=1024,
                                                         quantize=_cpu_quantize)
        if batch == 1:
            first_consts, first = consts, [inputs, {t: np.ascontiguousarray(a[..., ::-1]) if a.dtype == np.uint16 else a for t, a in inputs.items()}]
        names = ids
        ex = plugin.PluginExecutor(0)
        prepared = ex.prepare(p, {t: first_consts[t] for t in consts})
        for given in first:
            twice = {t: a if a.shape == tuple(inputs[t].shape) else np.concatenate([a] * 2, axis=0) for t, a in given.items()}
            got, _ = prepared.run(twice)
            results.append([got[names[key]] for key in ("image_out", "text_out")])
        ex.close()
    for one, two in zip(results[:2], results[2:]):
        for a, b in zip(one, two):
            assert np.array_equal(a[0], b[0]) and np.array_equal(a[0], b[1])
    assert not np.array_equal(results[0][0], results[1][0])


@pytest.mark.parametrize("case", ["kept", "output"])
def test_slices_that_share_a_buffer_take_no_more_memory(case, monkeypatch):
    """A few rows of a large internal tensor that are read long after it ("kept") or leave the program ("output"): sharing its buffer would
    hold all of it, a copy does not. Slices beside them that cost nothing still share. DIFB200_ROPE_FUSION=0 copies every Slice."""
    from diffusion_compiler_b200 import diffir as ir
    from diffusion_compiler_b200 import plugin
    rows, width, few = 4096, 1024, 16
    p = ir.Program()
    bf = ir.DType.BF16
    attrs = lambda start: [ir.Attribute.u64(ir.AttrKey.Axis, 0), ir.Attribute.u64(ir.AttrKey.Start, start)]  # noqa: E731
    x = p.add_tensor(bf, [rows, width], ir.Role.Input)
    large = [p.add_tensor(bf, [rows, width]) for _ in range(5)]
    part = p.add_tensor(bf, [few, width], ir.Role.Output if case == "output" else ir.Role.Internal)
    other, last = p.add_tensor(bf, [few, width]), p.add_tensor(bf, [few, width])
    out = p.add_tensor(bf, [few, width], ir.Role.Output)
    gelu = lambda a, b: p.add_op(ir.Opcode.Gelu, [a], [b], [ir.Attribute.u64(ir.AttrKey.Approximation, 1)])  # noqa: E731
    gelu(x, large[0])
    p.add_op(ir.Opcode.Slice, [large[0]], [part], attrs(3))
    p.add_op(ir.Opcode.Slice, [x], [other], attrs(5))  # of an Input, whose buffer stays anyway
    for a, b in zip(large, large[1:]):
        gelu(a, b)
    p.add_op(ir.Opcode.Slice, [large[-1]], [last], attrs(7))
    p.add_op(ir.Opcode.ResidualGate, [last, other, other if case == "output" else part], [out])
    given = {x: bf16_normal(np.random.default_rng(1), (rows, width))}
    results = {}
    monkeypatch.setenv("DIFB200_PROFILE", "1")
    for shared in (True, False):
        monkeypatch.setenv("DIFB200_ROPE_FUSION", "1" if shared else "0")
        ex = plugin.PluginExecutor(0)
        prepared = ex.prepare(p, {})
        got, _ = prepared.run(given, warmups=1)
        copies = prepared.profile().get(int(ir.Opcode.Slice), (0.0, 0))[1]
        results[shared] = prepared.compile_telemetry.resident_bytes, copies, got
        ex.close()
    assert results[True][0] <= results[False][0]
    assert (results[True][1], results[False][1]) == (1, 3)  # two share
    for t in results[True][2]:
        assert np.array_equal(results[True][2][t], results[False][2][t])


@pytest.mark.parametrize("S,world", [(512, 4), (437, 4)])
def test_token_sharded_video_block_matches_unsharded(S, world):
    """Ranks are emulated sequentially on one GPU: every rank runs its row-local part, the gather
    is done by copying slices between the per-rank buffers, then every rank attends and finishes.
    Without padding (S divisible) the key order and tiling are those of the unsharded run, so the
    outputs are bit-identical; with padding the fp32 accumulation order shifts (tolerance)."""
    import torch
    from diffusion_compiler_b200 import ops
    from diffusion_compiler_b200.sequence_shard import GatherBuffers, ShardPlan, VideoBlock
    rng = np.random.default_rng(6)
    hidden, heads, dim, ffn, rotary = 512, 4, 128, 1024, 96
    p, ids, consts, inputs = blocks.synth_video_block(rng, S, hidden, heads, dim, ffn, rotary, _cpu_quantize)
    tensors = {"norm1": consts[ids["norm1"]], "norm2": consts[ids["norm2"]], "q_norm": consts[ids["q_norm"]],
               "k_norm": consts[ids["k_norm"]], "cos": consts[ids["cos"]], "sin": consts[ids["sin"]],
               "linears": {n: (consts[w], consts[cs]) for n, (w, cs, b, N, K) in ids["linears"].items()}}
    block = VideoBlock(tensors, hidden, heads, dim, ffn, rotary, "cuda")
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.int16)).cuda().view(torch.bfloat16)
    x = dev(inputs[ids["x"]])
    mods = [dev(inputs[m]) for m in ids["mods"]]
    full = block.forward(x, mods, ShardPlan.make(S, 1), 0)
    plan = ShardPlan.make(S, world)
    gbs = [GatherBuffers(plan, r, heads, dim, "cuda") for r in range(world)]
    qs = []
    for r in range(world):
        lo, hi = plan.bounds(r)
        qs.append(block.pre_attention(x[lo:hi].contiguous(), [m[lo:hi].contiguous() for m in mods], plan, r, gbs[r]))
    for r in range(world):  # the all-gather: every rank receives every other rank's slice
        for src in range(world):
            for name in ("k8", "ks", "v"):
                getattr(gbs[r], name)[src * plan.slice_len:(src + 1) * plan.slice_len] = \
                    gbs[src].local(getattr(gbs[src], name))
    outs = []
    for r in range(world):
        lo, hi = plan.bounds(r)
        attn = block.attend(qs[r][0], qs[r][1], plan, gbs[r])
        outs.append(block.post_attention(x[lo:hi].contiguous(), attn, [m[lo:hi].contiguous() for m in mods]))
    sharded = torch.cat(outs, dim=0)
    torch.cuda.synchronize()
    ops.poll_status()
    if S % world == 0:
        assert torch.equal(sharded.view(torch.int16), full.view(torch.int16))
    else:
        a, b = sharded.float().cpu().numpy(), full.float().cpu().numpy()
        assert rel_l2(a, b) <= 1e-3 and cosine(a, b) >= 0.99999
