"""The forms of the 256-wide ConvRot quantiser at the edges of their dispatch: one block of 1024 columns per warp
(packing: or three), partial blocks, several warps per row, rows that only start on 16 bytes, and the
norm prologue. Codes and scales are whole numbers and exact fp32 values: every bit must agree."""
import numpy as np
import pytest

import oracle_bridge as ob
from helpers import activations, bf16_normal, to_torch_bf16

pytestmark = pytest.mark.gpu


def _bits_equal(want, got):
    got = got.cpu().numpy().reshape(want.shape)
    return np.array_equal(want.view(np.uint8), got.view(np.uint8))


@pytest.mark.parametrize("impl,rows,widths,clip,residual", [
    (2, 1200, [3072], 1.0, False),        # several rows per CTA, more than are resident at once
    (3, 1190, [3072], 0.97, False),       # the same with sign masks and clipped codes
    (2, 1301, [2816], 1.0, False),        # the row's last block holds three of four groups
    (2, 800, [3072, 12288], 1.0, False),  # fifteen warps per row, two inputs
    (2, 3, [3072, 12288], 1.0, False),    # the same width with few rows
    (2, 330, [10496], 1.0, False),        # eleven blocks, the last of one group
    (2, 500, [8192], 1.0, False),         # eight blocks: a CTA each
    (5, 130, [8192], 1.0, False),         # fp32 division
    (6, 40, [256], 1.0, True),            # the narrowest row, residual pair
    (2, 7, [16384], 1.0, True),           # the widest row, residual pair
    (4, 5, [16384], 1.0, False),          # 4096-wide rotation at its widest
])
def test_forms_bit_exact(impl, rows, widths, clip, residual):
    import torch
    from diffusion_compiler_b200 import ops
    rng = np.random.default_rng(rows + sum(widths))
    x = activations(rng, rows, sum(widths))
    x[rows // 2] = 0
    cuts = np.cumsum([0] + widths)
    parts = [np.ascontiguousarray(x[:, cuts[i]:cuts[i + 1]]) for i in range(len(widths))]
    want = ob.orc().quantize_int8_rows(parts, impl, clip, residual)
    for shift in (0, 8):  # 8 elements: parts that start on 16 bytes and not on 32
        tensors = []
        for p in parts:
            room = torch.empty(p.size + shift, dtype=torch.bfloat16, device="cuda")[shift:].view(p.shape)
            tensors.append(room.copy_(to_torch_bf16(p)))
        got = ops.quantize_int8_rows(tensors, impl, clip, residual=residual)
        for name, w, g in zip(("codes", "scales", "rcodes", "rscales"), want, got):
            assert _bits_equal(w, g), (name, shift)


@pytest.mark.parametrize("rows,K", [(444, 8192), (445, 6400), (445, 8192), (740, 7168), (740, 6144), (741, 8192)])
@pytest.mark.parametrize("impl", [2, 3, 5, 6])
def test_rows_of_a_cta_each_around_the_second_round(impl, rows, K):
    """Rows of 7 and 8 blocks, from as many as three CTAs per SM hold (444 on 148 SMs) to five for each SM, and 6 blocks."""
    from diffusion_compiler_b200 import ops
    x = activations(np.random.default_rng(rows + K + impl), rows, K)
    x[1] = 0
    want = ob.orc().quantize_int8_rows([x], impl, 1.0, False)
    got = ops.quantize_int8_rows([to_torch_bf16(x)], impl)
    assert _bits_equal(want[0], got[0]) and _bits_equal(want[1], got[1])


@pytest.mark.parametrize("N,K,impl", [(1300, 3072, 2), (450, 8192, 3), (9, 8192, 2), (20, 10496, 5)])
def test_packing_forms_bit_exact(N, K, impl):
    import torch
    from diffusion_compiler_b200 import ops
    rng = np.random.default_rng(N)
    w = ob.f32_to_bf16((rng.standard_normal((N, K)) * 0.02).astype(np.float32))
    w[N // 2] = 0
    eq = ob.orc().weight_equalization(w)
    for vector in (None, eq):
        want_codes, want_scales = ob.orc().quantize_weight_rows(w, impl, mse=True, equalise=vector)
        codes, scales = ops.quantize_weight_rows(to_torch_bf16(w), impl, mse_scale=True,
                                                 input_scale=None if vector is None else to_torch_bf16(vector))
        assert _bits_equal(want_scales, scales) and _bits_equal(want_codes, codes)


@pytest.mark.parametrize("rows,K", [(5, 3072), (1201, 3072), (33, 2816), (17, 12288), (70, 256)])
@pytest.mark.parametrize("impl", [2, 3, 5])
def test_norm_prologue_equals_the_two_ops(rows, K, impl):
    """RmsNormModulate / LayerNormModulate in front of the quantiser give the bits of the separate ops
    (the contraction of a product and a sum, or a lost rounding, shows as codes off by one)."""
    import ctypes as C

    import torch
    from diffusion_compiler_b200 import _lib, ops
    rng = np.random.default_rng(rows * 7 + K)
    t = lambda *shape, std=1.0: to_torch_bf16(bf16_normal(rng, shape, std))  # noqa: E731
    x, w, b, s, h = t(rows, K), t(K), t(K, std=0.1), t(rows, K, std=0.3), t(rows, K, std=0.3)
    p = lambda v: C.c_void_p(v.data_ptr())  # noqa: E731
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    normed = torch.empty_like(x)
    _lib.check(_lib.lib().difb200_rms_norm_modulate(p(x), p(w), p(s), p(h), p(normed), 2, rows, K, 1e-5, stream))
    want = ops.quantize_int8_rows([normed], impl)
    got = ops.rms_norm_modulate_quant(x, w, s, h, 1e-5, impl)
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])
    _lib.check(_lib.lib().difb200_layer_norm_modulate(p(x), p(w), p(b), p(s), p(h), p(normed), 2, rows, K, rows, 1e-6,
                                                      stream))
    want = ops.quantize_int8_rows([normed], impl)
    got = ops.layer_norm_modulate_quant(x, w, b, s, h, 1e-6, impl)
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])


@pytest.mark.parametrize("impl,mse", [(2, True), (2, False), (3, True), (5, False), (6, True)])
def test_equalised_packing_of_weights_that_are_not_finite(impl, mse):
    """Division by an equalisation entry keeps infinities and NaNs: a vector of ones (or of twos with doubled weights)
    gives the bits of packing without one, scale of the row included."""
    import torch
    from diffusion_compiler_b200 import ops
    rng = np.random.default_rng(impl)
    w = to_torch_bf16(bf16_normal(rng, (8, 2816), 0.02))
    w[1, 5], w[2, 300], w[2, 2700], w[3, 7], w[4] = float("inf"), float("-inf"), float("inf"), float("nan"), 0.0
    w[5, 9] = 3.0e38 / 2  # finite, and its double too
    want = ops.quantize_weight_rows(w, impl, mse_scale=mse)
    assert not torch.isfinite(want[1][1]) and torch.isfinite(want[1][5])
    for by in (1.0, 2.0):
        vector = torch.full((2816,), by, dtype=torch.bfloat16, device="cuda")
        got = ops.quantize_weight_rows(w * by, impl, mse_scale=mse, input_scale=vector)
        assert torch.equal(got[0], want[0]), by
        assert torch.equal(got[1].view(torch.int32), want[1].view(torch.int32)), by


@pytest.mark.parametrize("impl,rows,widths", [
    (3, 50, [1040, 2032]),    # inputs that meet between the two runs of a thread; all rows resident
    (6, 900, [1040, 2032]),   # the same, more rows than are resident
    (3, 2500, [1024]),        # one block per row, signed
    (5, 60, [2048, 7168]),    # nine blocks, fp32: three CTAs per SM
    (2, 70, [10240]),         # ten blocks
    (5, 40, [16, 11248]),     # eleven blocks, a first input of one run
    (6, 300, [5008, 10352]),  # fifteen blocks, signed fp32
    (3, 480, [15360]),        # fifteen blocks, signed
    (3, 40, [256, 528, 752]),  # three inputs
])
def test_one_block_forms_bit_exact(impl, rows, widths):
    from diffusion_compiler_b200 import ops
    rng = np.random.default_rng(rows + sum(widths))
    x = activations(rng, rows, sum(widths))
    cuts = np.cumsum([0] + widths)
    parts = [np.ascontiguousarray(x[:, cuts[i]:cuts[i + 1]]) for i in range(len(widths))]
    tensors = [to_torch_bf16(p) for p in parts]
    want = ob.orc().quantize_int8_rows(parts, impl, 1.0, False)
    got = ops.quantize_int8_rows(tensors, impl)
    assert _bits_equal(want[0], got[0]) and _bits_equal(want[1], got[1])


@pytest.mark.parametrize("N,K,impl", [(77, 3072, 3), (30, 8192, 5), (25, 9216, 2), (12, 11264, 6), (9, 15360, 3)])
def test_equalised_packing_without_search_bit_exact(N, K, impl):
    from diffusion_compiler_b200 import ops
    rng = np.random.default_rng(N + K)
    w = bf16_normal(rng, (N, K), 0.02)
    eq = ob.orc().weight_equalization(w)
    want_codes, want_scales = ob.orc().quantize_weight_rows(w, impl, mse=False, equalise=eq)
    codes, scales = ops.quantize_weight_rows(to_torch_bf16(w), impl, input_scale=to_torch_bf16(eq))
    assert _bits_equal(want_scales, scales) and _bits_equal(want_codes, codes)


@pytest.mark.parametrize("K", [256, 1280, 2816])
@pytest.mark.parametrize("impl", [2, 3, 5])
def test_layer_norm_prologue_of_rows_with_a_large_mean(K, impl):
    """Widths that leave groups of a warp's 1024 columns without elements, and a mean far above the deviation: what
    stands in those groups must not enter the row's maximum. Equal to the two separate ops, bit for bit."""
    import ctypes as C

    import torch
    from diffusion_compiler_b200 import _lib, ops
    rng = np.random.default_rng(K + impl)
    t = lambda *shape, std=1.0: to_torch_bf16(bf16_normal(rng, shape, std))  # noqa: E731
    rows = 40
    x, w, b, s, h = t(rows, K) + 8.0, t(K, std=0.1), t(K, std=0.01), t(rows, K, std=0.1), t(rows, K, std=0.01)
    p = lambda v: C.c_void_p(v.data_ptr())  # noqa: E731
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    normed = torch.empty_like(x)
    _lib.check(_lib.lib().difb200_layer_norm_modulate(p(x), p(w), p(b), p(s), p(h), p(normed), 2, rows, K, rows, 1e-6,
                                                      stream))
    want = ops.quantize_int8_rows([normed], impl)
    got = ops.layer_norm_modulate_quant(x, w, b, s, h, 1e-6, impl)
    assert torch.equal(want[1], got[1]) and torch.equal(want[0], got[0])


@pytest.mark.parametrize("impl", [2, 3, 5])
@pytest.mark.parametrize("rows_per_modulation", [1, 2, 3, 7, 84, 1302, 20832])
def test_layer_norm_prologue_finds_the_modulation_of_a_row(rows_per_modulation, impl):
    """Scale and shift that several rows share: the bits of the same ones given row by row."""
    import torch
    from diffusion_compiler_b200 import ops
    rng = np.random.default_rng(rows_per_modulation + impl)
    t = lambda *shape, std=1.0: to_torch_bf16(bf16_normal(rng, shape, std))  # noqa: E731
    rows, K = 20832, 256
    x, w, b = t(rows, K), t(K), t(K, std=0.1)
    mods = [t(rows // rows_per_modulation, K, std=0.3) for _ in range(2)]
    got = ops.layer_norm_modulate_quant(x, w, b, *mods, 1e-6, impl)
    want = ops.layer_norm_modulate_quant(x, w, b, *[m.repeat_interleave(rows_per_modulation, 0) for m in mods], 1e-6, impl)
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])


@pytest.mark.parametrize("impl", [2, 3])
@pytest.mark.parametrize("K", [256, 3072, 9216])
def test_quotients_out_of_the_two_part_products_range(impl, K):
    """Rows whose scale is so large that the reciprocal's low part would be subnormal, and clips so small that quotients
    overflow: such rows take the fp32 quotient. The rows beside them do not."""
    from diffusion_compiler_b200 import ops
    rng = np.random.default_rng(K + impl)
    x = ob.bf16_to_f32(activations(rng, 24, K))
    x[3] *= np.float32(2.0 ** 113)
    x[4] *= np.float32(2.0 ** 106)
    x[5] *= np.float32(2.0 ** -120)
    x[6] = 0
    x = ob.f32_to_bf16(x)
    for clip in (1.0, 1.0e-3, 1.0e-6):
        want = ob.orc().quantize_int8_rows([x], impl, clip, False)
        got = ops.quantize_int8_rows([to_torch_bf16(x)], impl, clip)
        assert _bits_equal(want[1], got[1]) and _bits_equal(want[0], got[0]), clip
    for clip in (1.0e-12, 1.0e-30):  # beyond the integers the reference converts to: saturated by sign
        codes = ops.quantize_int8_rows([to_torch_bf16(x)], impl, clip)[0].cpu().numpy()
        assert np.all(codes[want[0] > 0] == 127) and np.all(codes[want[0] < 0] == -128), clip


@pytest.mark.parametrize("impl", [2, 3, 5, 6])
@pytest.mark.parametrize("more,width", [
    (0, 256),      # one warp per row: as many rows as the table of reciprocals is made for
    (1, 3072),     # three blocks per warp, a last round of one row
    (448, 2816),   # the same with a partial third block
    (72, 1280),    # two blocks, the second of one group
    (8, 8192),     # eight blocks
    (12, 12288),   # twelve
    (0, 14592),    # fifteen, the last of one group: the largest table
    (2, 15360),    # fifteen
])
def test_packing_with_a_table_of_reciprocals(impl, more, width):
    """Rows are packed one by one: all at once, where a CTA's rows share a table of the equalisation's reciprocals, and a few hundred
    at a time, where every row makes its own. Entries beyond the table's range, infinities and NaN among them."""
    import torch
    from diffusion_compiler_b200 import ops
    blocks = (width + 1023) // 1024
    rows = -(-72 * torch.cuda.get_device_properties(0).multi_processor_count // blocks) + more  # the least that share a table, and more
    rng = np.random.default_rng(rows + impl)
    w = to_torch_bf16(bf16_normal(rng, (rows, width), std=0.02))
    eq = to_torch_bf16(ob.f32_to_bf16(np.exp(0.7 * rng.standard_normal(width)).astype(np.float32)))
    w[1], w[2, 3], w[3, 5], w[4] = 0, float("inf"), float("nan"), w[4] * 2.0**-110
    for wild in (False, True):
        if wild:
            eq[7], eq[255], eq[100] = 2.0**-60, -eq[255], 2.0**70
        codes, scales = ops.quantize_weight_rows(w, impl, mse_scale=True, input_scale=eq)
        parts = [ops.quantize_weight_rows(w[i:i + 400], impl, mse_scale=True, input_scale=eq) for i in range(0, rows, 400)]
        assert torch.equal(codes, torch.cat([p[0] for p in parts]))
        assert torch.equal(scales.view(torch.int32), torch.cat([p[1] for p in parts]).view(torch.int32))


@pytest.mark.parametrize("impl", [2, 3])
@pytest.mark.parametrize("extra,widths", [(1, [12544]), (5, [3072, 12288]), (449, [16384])])  # rows beyond two per SM
def test_wide_rows_rotated_one_ahead_of_their_maximum(impl, extra, widths):
    """Rows of more than 12 blocks, more than two per SM: the next one is rotated before one is finished. Rows are independent: the same
    as a hundred at a time, which are not taken so; magnitudes that differ from row to row, so that a row's maximum in
    another's place would show."""
    import torch
    from diffusion_compiler_b200 import ops
    rows = 2 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    rng = np.random.default_rng(rows + impl)
    parts = [to_torch_bf16(bf16_normal(rng, (rows, w))) * torch.exp2((torch.arange(rows, device="cuda") % 23 - 11).float()).to(torch.bfloat16)[:, None]
             for w in widths]
    got = ops.quantize_int8_rows(parts, impl)
    want = [ops.quantize_int8_rows([p[i:i + 100].contiguous() for p in parts], impl) for i in range(0, rows, 100)]
    assert torch.equal(got[0], torch.cat([w[0] for w in want]))
    assert torch.equal(got[1].view(torch.int32), torch.cat([w[1] for w in want]).view(torch.int32))
    ops.poll_status()


_FIRST_CALL = """
import ctypes as C, threading
import torch
from diffusion_compiler_b200 import _lib, ops
rows = 2 * torch.cuda.get_device_properties(0).multi_processor_count + 7
g = torch.Generator(device="cuda").manual_seed(1)
x = torch.randn((rows, 12544), generator=g, device="cuda").to(torch.bfloat16)
out = torch.zeros(x.shape, dtype=torch.int8, device="cuda"), torch.zeros(rows, device="cuda")
f = torch.randn((4, 64), generator=g, device="cuda")
gated, base = torch.zeros_like(f), torch.ones(8, device="cuda")
side, errors = torch.cuda.Stream(), []
torch.cuda.synchronize()

def work():
    try:
        torch.cuda.set_device(0)
        with torch.cuda.stream(side):
            ops.quantize_int8_rows([x], 2, out=out)
        p = lambda t: C.c_void_p(t.data_ptr())  # a kernel whose launch is checked by the thread's last error
        _lib.check(_lib.lib().difb200_residual_gate(p(f), p(f), p(f), p(gated), 1, 4, 64, 4, C.c_void_p(side.cuda_stream)))
    except Exception as e:
        errors.append(e)

graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):  # (a capture in global mode: it ends where any thread allocates)
    y = base + 1
    thread = threading.Thread(target=work)
    thread.start()
    thread.join()
    z = y * 3
assert not errors, errors
graph.replay()
torch.cuda.synchronize()
assert bool((z == 6).all()) and torch.allclose(gated, f + f * f)
parts = [ops.quantize_int8_rows([x[i:i + 100]], 2) for i in range(0, rows, 100)]
assert torch.equal(out[0], torch.cat([q[0] for q in parts])) and torch.equal(out[1], torch.cat([q[1] for q in parts]))
ops.poll_status()
print("same codes")
"""


def test_first_quantiser_call_of_a_process_beside_a_capture():
    """A quantiser has no scratch: its first call on wide rows allocates nothing, so a capture on another thread stays valid, and
    no error is left behind for the thread's next launch."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    run = subprocess.run([sys.executable, "-c", _FIRST_CALL], cwd=root, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and "same codes" in run.stdout, run.stderr[-2000:]
