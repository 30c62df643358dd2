"""The Direct codes (QuantizeInt8Rows variant 1) that QkNormPartialRope and the attention's operand kernel make without a
division, against the oracle's quotients: rows whose quotients lie exactly in the middle between two integers, rows
with infinity and NaN, and the rotation kernel at the edges of its rows per warp, with every part of its addressing."""
import ctypes as C

import numpy as np
import pytest

import oracle_bridge as ob
from helpers import bf16_normal, from_torch_bf16, to_torch_bf16

pytestmark = pytest.mark.gpu


def _rope(x, w, cos, sin, rotary, interleaved, eps):
    """QkNormPartialRope in fp32 with the reference's order and roundings (cpu_executor.cpp:1741-1837): x [T,H,128] and
    w [128] as fp32 values, tables [T,width]."""
    f = np.float32
    total = np.zeros(x.shape[:2], f)
    for d in range(128):
        total = total + x[..., d] * x[..., d]
    inv = f(1) / np.sqrt(total / f(128) + f(eps))
    bf = lambda a: ob.bf16_to_f32(ob.f32_to_bf16(np.ascontiguousarray(a, f)))  # noqa: E731
    n = x * inv[..., None]
    n = bf(bf(n) * w) if interleaved else n * w
    c, s, half = cos[:, None, :], sin[:, None, :], rotary // 2
    out = n.copy()
    if interleaved:
        even, odd = n[..., 0:rotary:2], n[..., 1:rotary:2]
        out[..., 0:rotary:2], out[..., 1:rotary:2] = even * c - odd * s, even * s + odd * c
    else:
        a, b = n[..., :half], n[..., half:rotary]
        wide = cos.shape[1] == rotary
        c2, s2 = (c[..., half:], s[..., half:]) if wide else (c, s)
        out[..., :half], out[..., half:rotary] = a * c[..., :half] - b * s[..., :half], b * c2 + a * s2
    return ob.f32_to_bf16(np.ascontiguousarray(out, f))


@pytest.mark.parametrize("tokens,heads", [(1, 1), (3, 3), (11, 3), (2401, 24)])  # 1, 9, 33 rows: 8 per warp; the last: 32
@pytest.mark.parametrize("interleaved,rotary,wide", [(False, 96, True), (False, 128, False), (False, 64, True),
                                                     (True, 128, False), (True, 64, False), (True, 96, False)])
def test_rope_codes_and_output(tokens, heads, interleaved, rotary, wide):
    import torch
    from diffusion_compiler_b200 import _lib
    rng = np.random.default_rng(tokens + rotary)
    x, w = bf16_normal(rng, (tokens, heads, 128)), ob.f32_to_bf16((1 + 0.1 * rng.standard_normal(128)).astype(np.float32))
    width = rotary if wide else rotary // 2
    angle = rng.uniform(0, 6.28, (tokens, width)).astype(np.float32)
    cos, sin = np.cos(angle), np.sin(angle)
    want = _rope(ob.bf16_to_f32(x), ob.bf16_to_f32(w), cos, sin, rotary, interleaved, 1e-5)
    want_codes, want_scales = ob.orc().quantize_int8_rows([want.reshape(-1, 128)], 1)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    dx, dw, dc, ds = to_torch_bf16(x), to_torch_bf16(w), t(cos), t(sin)
    out = torch.zeros((tokens, heads, 128), dtype=torch.bfloat16, device="cuda")
    codes = torch.zeros((tokens, heads, 128), dtype=torch.int8, device="cuda")
    scales = torch.zeros(tokens * heads, dtype=torch.float32, device="cuda")
    p = lambda a: C.c_void_p(a.data_ptr())  # noqa: E731
    _lib.check(_lib.lib().difb200_qk_norm_rope_quant(p(dx), p(dw), p(dc), p(ds), p(out), p(codes), p(scales), 1, tokens,
                                                     heads, rotary, width, tokens, tokens, 0, 1e-5, int(interleaved), None))
    torch.cuda.synchronize()
    assert np.array_equal(from_torch_bf16(out), want)
    assert np.array_equal(codes.cpu().numpy().reshape(-1, 128), want_codes)
    assert np.array_equal(scales.cpu().numpy().view(np.uint32), want_scales.view(np.uint32))


def _rope_quant(x, w, cos, sin, rotary, interleaved, sequence, table_sequence, start):
    """difb200_qk_norm_rope_quant on device tensors: (output bits, codes, scales) as host arrays."""
    import torch
    from diffusion_compiler_b200 import _lib
    tokens, heads = x.shape[0], x.shape[1]
    out = torch.zeros((tokens, heads, 128), dtype=torch.bfloat16, device="cuda")
    codes = torch.full((tokens, heads, 128), 99, dtype=torch.int8, device="cuda")
    scales = torch.zeros(tokens * heads, dtype=torch.float32, device="cuda")
    p = lambda a: C.c_void_p(a.data_ptr())  # noqa: E731
    _lib.check(_lib.lib().difb200_qk_norm_rope_quant(
        p(x), p(w), p(cos), p(sin), p(out), p(codes), p(scales), 1 if cos.dtype == torch.float32 else 2, tokens, heads, rotary,
        cos.shape[-1], sequence, table_sequence, start, 1e-5, int(interleaved), None))
    torch.cuda.synchronize()
    return from_torch_bf16(out), codes.cpu().numpy().reshape(-1, 128), scales.cpu().numpy()


@pytest.mark.parametrize("sequence,heads", [(37, 5), (1201, 24)])  # 370 rows: 8 per warp; 57648: 32; neither fills the last
@pytest.mark.parametrize("interleaved,rotary", [(False, 96), (True, 128)])
@pytest.mark.parametrize("bf16_table", [False, True])
def test_rope_of_two_sequences_with_longer_tables(sequence, heads, interleaved, rotary, bf16_table):
    """Two sequences whose tables are longer than they are and start at a later row, with fp32 and bf16 tables."""
    import torch
    rng = np.random.default_rng(sequence + rotary)
    table, start = sequence + 13, 9
    x = bf16_normal(rng, (2 * sequence, heads, 128))
    w = ob.f32_to_bf16((1 + 0.1 * rng.standard_normal(128)).astype(np.float32))
    angle = rng.uniform(0, 6.28, (2, table, rotary // 2 if interleaved else rotary)).astype(np.float32)
    cos, sin = np.cos(angle), np.sin(angle)
    if bf16_table:
        dc, ds = to_torch_bf16(ob.f32_to_bf16(cos)), to_torch_bf16(ob.f32_to_bf16(sin))
        cos, sin = ob.bf16_to_f32(ob.f32_to_bf16(cos)), ob.bf16_to_f32(ob.f32_to_bf16(sin))
    else:
        dc, ds = torch.from_numpy(cos).cuda(), torch.from_numpy(sin).cuda()
    rows = lambda a: np.ascontiguousarray(a[:, start:start + sequence]).reshape(2 * sequence, -1)  # noqa: E731
    want = _rope(ob.bf16_to_f32(x), ob.bf16_to_f32(w), rows(cos), rows(sin), rotary, interleaved, 1e-5)
    want_codes, want_scales = ob.orc().quantize_int8_rows([want.reshape(-1, 128)], 1)
    out, codes, scales = _rope_quant(to_torch_bf16(x), to_torch_bf16(w), dc, ds, rotary, interleaved, sequence, table, start)
    assert np.array_equal(out, want)
    assert np.array_equal(codes, want_codes)
    assert np.array_equal(scales.view(np.uint32), want_scales.view(np.uint32))


@pytest.mark.parametrize("fusion", ["1", "0"])
def test_rope_reads_a_slice_of_a_wider_tensor(monkeypatch, fusion):
    """QkNormPartialRope on the middle third of a packed tensor [2, 37, 3 * 5 * 128], read in place and through a copy."""
    from diffusion_compiler_b200 import diffir, plugin
    from diffusion_compiler_b200.diffir import AttrKey, Attribute, DType, Opcode, Role
    monkeypatch.setenv("DIFB200_ROPE_FUSION", fusion)
    rng = np.random.default_rng(8)
    T, H, table, start = 37, 5, 50, 9
    x, w = bf16_normal(rng, (2, T, 3 * H * 128)), ob.f32_to_bf16((1 + 0.1 * rng.standard_normal(128)).astype(np.float32))
    angle = rng.uniform(0, 6.28, (2, table, 64)).astype(np.float32)
    cos, sin = np.cos(angle), np.sin(angle)
    p = diffir.Program()
    tx = p.add_tensor(DType.BF16, [2, T, 3 * H * 128], Role.Input)
    tw = p.add_tensor(DType.BF16, [128], Role.Constant)
    tc, ts = (p.add_tensor(DType.F32, [2, table, 64], Role.Input) for _ in range(2))
    flat, shaped = p.add_tensor(DType.BF16, [2, T, H * 128]), p.add_tensor(DType.BF16, [2, T, H, 128])
    to = p.add_tensor(DType.BF16, [2, T, H, 128], Role.Output)
    p.add_op(Opcode.Slice, [tx], [flat], [Attribute.u64(AttrKey.Axis, 2), Attribute.u64(AttrKey.Start, H * 128)])
    p.add_op(Opcode.Reshape, [flat], [shaped])
    p.add_op(Opcode.QkNormPartialRope, [shaped, tw, tc, ts], [to],
             [Attribute.f64(AttrKey.Epsilon, 1e-5), Attribute.u64(AttrKey.Implementation, 2),
              Attribute.u64(AttrKey.BlockSize, 128), Attribute.u64(AttrKey.RotaryDim, 128),
              Attribute.u64(AttrKey.Start, start), Attribute.u64(AttrKey.RotaryLayout, 1)])
    ex = plugin.PluginExecutor(0)
    got, _ = ex.prepare(p, {tw: w}).run({tx: x, tc: cos, ts: sin})
    ex.close()
    part = ob.bf16_to_f32(np.ascontiguousarray(x[:, :, H * 128:2 * H * 128])).reshape(2 * T, H, 128)
    rows = lambda a: np.ascontiguousarray(a[:, start:start + T]).reshape(2 * T, -1)  # noqa: E731
    want = _rope(part, ob.bf16_to_f32(w), rows(cos), rows(sin), 128, True, 1e-5)
    assert np.array_equal(got[to].reshape(want.shape), want)


@pytest.mark.parametrize("tokens", [11, 2401])  # 8 and 32 rows per warp
@pytest.mark.parametrize("interleaved,rotary", [(False, 96), (True, 128)])
def test_rope_keeps_nan_and_infinity(tokens, interleaved, rotary):
    """A NaN makes its row NaN, an infinity makes NaN of itself and of its partner in the rotation and zeros of the rest (its
    norm is infinite), a NaN in a table those two elements: as on a CPU, so that a broken activation shows. Codes are zero
    where the value is NaN, and the scale is that of the other elements."""
    import torch
    rng = np.random.default_rng(tokens)
    heads = 24
    x = bf16_normal(rng, (tokens, heads, 128))
    for row, (at, bits) in {1: (5, 0x7fc0), 3: (100, 0xffc0), 4: (2, 0x7f80), 6: (97, 0xff80), 8: (0, 0x7f81)}.items():
        x[row, 2, at] = bits
        x[tokens - 1 - row, heads - 1, at] = bits
    w = ob.f32_to_bf16((1 + 0.1 * rng.standard_normal(128)).astype(np.float32))
    angle = rng.uniform(0, 6.28, (tokens, rotary // 2 if interleaved else rotary)).astype(np.float32)
    cos, sin = np.cos(angle), np.sin(angle)
    cos[7, 3] = np.nan
    with np.errstate(invalid="ignore"):
        want = _rope(ob.bf16_to_f32(x), ob.bf16_to_f32(w), cos, sin, rotary, interleaved, 1e-5)
    t = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    out, codes, scales = _rope_quant(to_torch_bf16(x), to_torch_bf16(w), t(cos), t(sin), rotary, interleaved, tokens, tokens, 0)
    nan = np.isnan(ob.bf16_to_f32(want))
    assert 6 * 128 <= nan.sum() < want.size // 2
    assert np.array_equal(np.isnan(ob.bf16_to_f32(out)), nan)
    assert np.array_equal(out[~nan], want[~nan])
    others = want.copy()
    others[nan] = 0
    want_codes, want_scales = ob.orc().quantize_int8_rows([others.reshape(-1, 128)], 1)
    assert np.array_equal(codes, want_codes)
    assert np.array_equal(scales.view(np.uint32), want_scales.view(np.uint32))


def test_operand_codes_of_ties():
    """ops.attention (its operand kernel) against ops.attention_int8 on the oracle's codes. A row of which 127 is the
    largest has the scale 1, and its values k + 1/2 are ties. A query with infinity has an infinite
    scale and is left out."""
    import torch
    from diffusion_compiler_b200 import ops
    rng = np.random.default_rng(4)
    S, H, KV = 150, 3, 1
    q = ob.bf16_to_f32(bf16_normal(rng, (1, S, H, 128)))
    k, v = bf16_normal(rng, (1, S, KV, 128)), bf16_normal(rng, (1, S, KV, 128))
    ties = np.round(rng.uniform(-126, 126, (40, H, 128))) + 0.5
    ties[:, :, 17] = np.where(rng.random((40, H)) < 0.5, 127, -127)
    q[0, :40] = ties * np.exp2(rng.integers(-12, -6, (40, H, 1)))
    q[0, 41, 1, 9], q[0, 42, 2, :] = np.inf, 0
    q = ob.f32_to_bf16(q.astype(np.float32))
    kf = ob.bf16_to_f32(k)
    kf[0, 3:9] = (np.round(rng.uniform(-126, 126, (6, KV, 128))) + 0.5) * 2.0 ** -6
    kf[0, 3:9, 0, 64] = 127 * 2.0 ** -6
    k = ob.f32_to_bf16(kf.astype(np.float32))
    q8, qs = ob.orc().quantize_int8_rows([q.reshape(-1, 128)], 1)
    k8, ks = ob.orc().quantize_int8_rows([k.reshape(-1, 128)], 1)
    t = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    want = ops.attention_int8(t(q8.reshape(1, S, H, 128)), t(qs), t(k8.reshape(1, S, KV, 128)), t(ks), to_torch_bf16(v))
    got = ops.attention(to_torch_bf16(q), to_torch_bf16(k), to_torch_bf16(v))
    torch.cuda.synchronize()
    ops.poll_status()
    finite = np.isfinite(qs.reshape(S, H))
    assert finite.sum() >= S * H - 1
    a, b = from_torch_bf16(got)[0][finite], from_torch_bf16(want)[0][finite]
    assert np.array_equal(a, b)
