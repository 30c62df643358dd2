"""GPU parity of the W8A8 linear path (QuantizeInt8Rows + LinearInt8Scaled) against the CPU
oracle, through the C-ABI of libdifb200.so. INT8 codes, F32 scales and INT32 accumulators must
be bit-exact; bf16 outputs bit-exact without GELU and within rel-L2 <= 2e-3 with it."""
import numpy as np
import pytest

import oracle_bridge as ob
from helpers import activations, bf16_normal, cosine, from_torch_bf16, rel_l2, to_torch_bf16

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    import torch
    from diffusion_compiler_b200 import ops as _ops
    assert torch.cuda.is_available()
    return _ops


def _quant_case(ops, rng, impl, rows, K, clip, residual, parts=None):
    import torch
    x = activations(rng, rows, K)
    x[rows // 2] = 0  # an all-zero row exercises the guarded scale
    if parts is None:
        parts = [K]
    cuts = np.cumsum([0] + list(parts))
    xs = [np.ascontiguousarray(x[:, cuts[i]:cuts[i + 1]]) for i in range(len(parts))]
    want = ob.orc().quantize_int8_rows(xs, impl, clip, residual)
    got = ops.quantize_int8_rows([to_torch_bf16(a) for a in xs], impl, clip, residual=residual)
    torch.cuda.synchronize()
    names = ["codes", "scales", "rcodes", "rscales"]
    for name, w, g in zip(names, want, got):
        g = g.cpu().numpy().reshape(w.shape)
        assert np.array_equal(w.view(np.uint8), g.view(np.uint8)), \
            "%s differ: impl=%d rows=%d K=%d (%d mismatches)" % (
                name, impl, rows, K, int(np.sum(w.view(np.uint8) != g.view(np.uint8))))


@pytest.mark.parametrize("impl", [1, 2, 3, 5, 6])
@pytest.mark.parametrize("rows,K", [(1, 256), (37, 768), (64, 3072), (5, 12288)])
def test_quantize_h256_bit_exact(ops, impl, rows, K):
    rng = np.random.default_rng(100 + impl)
    _quant_case(ops, rng, impl, rows, K, 1.0, False)
    _quant_case(ops, rng, impl, rows, K, 0.9995, True)


@pytest.mark.parametrize("impl", [4, 7])
@pytest.mark.parametrize("rows,K", [(3, 4096), (9, 12288)])
def test_quantize_h4096_bit_exact(ops, impl, rows, K):
    rng = np.random.default_rng(200 + impl)
    _quant_case(ops, rng, impl, rows, K, 1.0, False)
    _quant_case(ops, rng, impl, rows, K, 0.97, True)


@pytest.mark.parametrize("impl", [1, 2, 6])
def test_quantize_concatenated_inputs(ops, impl):
    rng = np.random.default_rng(7)
    _quant_case(ops, rng, impl, 19, 1024, 1.0, False, parts=[256, 512, 256])


def test_quantize_direct_per_token_head(ops):
    """Direct on [B,S,H,128]: the per-token-per-head quantisation of attention Q/K."""
    rng = np.random.default_rng(8)
    _quant_case(ops, rng, 1, 2 * 33 * 4, 128, 1.0, False)
    _quant_case(ops, rng, 1, 11, 100, 1.0, True)  # odd width: scalar path


@pytest.mark.parametrize("impl", [2, 3, 5, 6])
@pytest.mark.parametrize("N,K", [(5, 256), (40, 768), (64, 3072), (6, 12288)])
def test_weight_rows_with_mse_scale_bit_exact(ops, impl, N, K):
    """Weight-side packing (offline packer's encoder, reference tools/difflux2sample.cpp:2994-3059)
    with and without the MSE scale search (:1225-1259) against the CPU restatement."""
    import torch
    rng = np.random.default_rng(1000 * impl + K)
    w = ob.f32_to_bf16((rng.standard_normal((N, K)) * 0.02).astype(np.float32))
    w[N // 2] = 0
    dw = torch.from_numpy(w.view(np.int16)).cuda().view(torch.bfloat16)
    for mse in (False, True):
        want_codes, want_scales = ob.orc().quantize_weight_rows(w, impl, mse=mse)
        codes, scales = ops.quantize_weight_rows(dw, impl, mse_scale=mse)
        torch.cuda.synchronize()
        assert np.array_equal(scales.cpu().numpy().view(np.uint32), want_scales.view(np.uint32)), mse
        assert np.array_equal(codes.cpu().numpy(), want_codes), mse
    ops.poll_status()


@pytest.mark.parametrize("impl,mse", [(2, False), (3, True), (5, True), (6, False)])
def test_weight_rows_with_input_equalization(ops, impl, mse):
    """Input equalisation of the offline packer (reference tools/difflux2sample.cpp:2967-2990 for
    the vector, :3005-3014 for its use): codes and scales bit-exact given the same vector; the
    vector computed on the GPU within one bf16 ulp of the CPU restatement (libm's logf against
    CUDA's)."""
    import torch
    rng = np.random.default_rng(77 + impl)
    N, K = 48, 768
    gains = np.exp(rng.standard_normal(K) * 0.8).astype(np.float32)  # uneven column magnitudes
    w = ob.f32_to_bf16((rng.standard_normal((N, K)) * 0.02).astype(np.float32) * gains)
    eq = ob.orc().weight_equalization(w)
    dw = torch.from_numpy(w.view(np.int16)).cuda().view(torch.bfloat16)
    got_eq = ops.weight_equalization(dw)
    diff = np.abs(got_eq.view(torch.int16).cpu().numpy().astype(np.int32) - eq.view(np.int16).astype(np.int32))
    assert diff.max() <= 1 and np.count_nonzero(diff) <= K // 50
    assert ob.bf16_to_f32(eq).min() >= 0.5 and ob.bf16_to_f32(eq).max() <= 2.0 and len(np.unique(eq)) > 8
    deq = torch.from_numpy(eq.view(np.int16)).cuda().view(torch.bfloat16)
    want_codes, want_scales = ob.orc().quantize_weight_rows(w, impl, mse=mse, equalise=eq)
    codes, scales = ops.quantize_weight_rows(dw, impl, mse_scale=mse, input_scale=deq)
    torch.cuda.synchronize()
    assert np.array_equal(scales.cpu().numpy().view(np.uint32), want_scales.view(np.uint32))
    assert np.array_equal(codes.cpu().numpy(), want_codes)
    plain_codes, _ = ob.orc().quantize_weight_rows(w, impl, mse=mse)
    assert not np.array_equal(plain_codes, want_codes)  # the vector does change the packing
    ops.poll_status()


def _weights(rng, N, K, impl):
    wf = bf16_normal(rng, (N, K), 0.02)
    return ob.orc().quantize_int8_rows([wf], impl, 1.0)


@pytest.fixture(params=["1", "2"], ids=["single-cta", "cta-pair"])
def gemm_form(request, monkeypatch):
    """Runs a test with the 128x256 single-CTA tiles and with the 256x256 CTA-pair (cta_group::2)
    tiles of the GEMM kernel."""
    monkeypatch.setenv("DIFB200_GEMM_CTAS", request.param)
    return request.param


@pytest.mark.parametrize("M,K,N", [(128, 256, 256), (100, 512, 200), (300, 1024, 520), (1024, 3072, 3072),
                                   (2000, 768, 1800)])
def test_linear_int8_scaled_bit_exact(ops, gemm_form, M, K, N):
    import torch
    rng = np.random.default_rng(M + N)
    ob.orc().lib.orc_set_threads(8)
    x = activations(rng, M, K)
    w8, ws = _weights(rng, N, K, 2)
    x8, xs = ob.orc().quantize_int8_rows([x], 2, 1.0)
    bias = bf16_normal(rng, (N,), 0.01)
    want, want_acc = ob.orc().linear_int8_scaled(x8, w8, xs, ws, want_acc=True)
    t = lambda a: torch.from_numpy(a).cuda()
    got, acc = ops.linear_int8_scaled(t(x8), t(w8), t(xs), t(ws), want_acc=True)
    torch.cuda.synchronize()
    assert np.array_equal(acc.cpu().numpy(), want_acc), "INT32 accumulators differ"
    assert np.array_equal(from_torch_bf16(got), want), "bf16 dequantised outputs differ"
    # + BiasAdd keeps the intermediate bf16 rounding of the two-op program
    want_b = ob.orc().bias_add(want, bias)
    got_b = ops.linear_int8_scaled(t(x8), t(w8), t(xs), t(ws), bias=to_torch_bf16(bias))
    assert np.array_equal(from_torch_bf16(got_b), want_b), "bias epilogue differs"
    # + Gelu(tanh): libm tanhf vs device tanhf, tolerance from the north star
    want_g = ob.orc().gelu_tanh(want_b)
    got_g = from_torch_bf16(ops.linear_int8_scaled(t(x8), t(w8), t(xs), t(ws), bias=to_torch_bf16(bias), gelu=True))
    a, b = ob.bf16_to_f32(got_g), ob.bf16_to_f32(want_g)
    assert rel_l2(a, b) <= 2e-3 and cosine(a, b) >= 0.9999
    assert np.mean(got_g != want_g) < 5e-3  # last-bit differences of tanh only
    ops.poll_status()


@pytest.mark.parametrize("form", ["2,192,1", "2,128,1", "1,256,1", "1,128,1", "1,128,2", "1,128,4", None])
@pytest.mark.parametrize("M,K,N", [(1, 3072, 3072), (2, 12288, 384), (33, 640, 256), (40, 656, 200), (127, 528, 128), (129, 656, 264),
                                   (257, 1168, 131), (520, 512, 1032), (300, 768, 577)])
def test_linear_int8_scaled_narrow_and_split_tiles(ops, monkeypatch, form, M, K, N):
    """The 128- and 192-column tiles and the splits over k-blocks (cluster exchange): tile edges in M and N, loads that end
    with the rows, ragged k-blocks
    (a split whose shares differ), odd N (no TMA stores); `None` is the form the dispatch picks."""
    import torch
    if form:
        monkeypatch.setenv("DIFB200_GEMM_FORM", form)
    g = torch.Generator().manual_seed(M + N + K)
    x8, w8 = (torch.randint(-127, 128, s, dtype=torch.int8, generator=g) for s in ((M, K), (N, K)))
    xs, ws = torch.rand(M, generator=g), torch.rand(N, generator=g)
    bias = torch.randn(N, generator=g).to(torch.bfloat16)
    want_acc = (x8.double() @ w8.double().T).to(torch.int32)  # exact: below 2^53
    want = ((want_acc.float() * xs[:, None]) * ws[None]).to(torch.bfloat16)
    dev = [t.cuda() for t in (x8, w8, xs, ws)]
    for _ in range(2):
        got, acc = ops.linear_int8_scaled(*dev, want_acc=True)
        assert torch.equal(acc.cpu(), want_acc)
        assert torch.equal(got.cpu(), want)
        got = ops.linear_int8_scaled(*dev, bias=bias.cuda())
        assert torch.equal(got.cpu(), (want.float() + bias.float()[None]).to(torch.bfloat16))
    ops.poll_status()


@pytest.mark.parametrize("form", ["2,256,1", "2,192,1", "2,128,1", "1,256,1", "1,128,1"])
@pytest.mark.parametrize("K", [256, 512])
def test_linear_int8_scaled_warps_without_rows_behind_full_tiles(ops, monkeypatch, form, K):
    """Three and more tiles per CTA, of which the last ones end with the rows in every quarter of a 128-row tile: a warp
    without rows there has just stored boxes of full tiles, which must not be filled again while they are read. Few
    k-blocks, so that the next accumulator is complete when a tile's epilogue ends. The bias would show in the full tiles."""
    import torch
    monkeypatch.setenv("DIFB200_GEMM_FORM", form)
    g = torch.Generator(device="cuda").manual_seed(K)
    N, rest = 74 * 256 + 8, (1, 33, 97, 129, 193, 224)
    x8, w8 = (torch.randint(-127, 128, s, generator=g, device="cuda", dtype=torch.int8) for s in ((512 + max(rest), K), (N, K)))
    xs, ws = torch.rand(len(x8), generator=g, device="cuda"), torch.rand(N, generator=g, device="cuda")
    bias = torch.randn(N, generator=g, device="cuda").to(torch.bfloat16) * 1000
    acc = (x8.double() @ w8.double().T).float()  # exact: |sum| < 2^24
    want = ((((acc * xs[:, None]) * ws[None]).to(torch.bfloat16)).float() + bias.float()[None]).to(torch.bfloat16)
    for M in (512 + r for r in rest):
        outs = [torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(4)]
        for out in outs:
            ops.linear_int8_scaled(x8[:M], w8, xs[:M], ws, bias=bias, out=out[:M])
        for out in outs:
            assert torch.equal(out[:M].view(torch.int16), want[:M].view(torch.int16)), M
            assert bool((out[M] == 7.0).all())
    ops.poll_status()


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 32, 33])  # 8, 16 and 32 rows per form; 33 is the tile kernel's
@pytest.mark.parametrize("K,N", [(16, 16), (48, 1), (80, 131), (3072, 40), (3136, 24), (12288, 17), (16, 3000)])
def test_linear_of_few_rows_bit_exact(ops, M, K, N):
    """The kernel of few rows: chunks of 64 k that end early, fewer chunks than warps, warps whose last batch is short,
    columns that do not fill 16, and each number of 8-row groups; with codes of -128, bias, GELU and the accumulators."""
    import torch
    g = torch.Generator().manual_seed(M + N + K)
    x8, w8 = (torch.randint(-128, 128, s, dtype=torch.int8, generator=g) for s in ((M, K), (N, K)))
    xs, ws = torch.rand(M, generator=g) * 0.01, torch.rand(N, generator=g) * 0.01
    bias = torch.randn(N, generator=g).to(torch.bfloat16)
    want_acc = (x8.double() @ w8.double().T).to(torch.int32)  # exact: below 2^53
    want = ((want_acc.float() * xs[:, None]) * ws[None]).to(torch.bfloat16)
    want_b = (want.float() + bias.float()[None]).to(torch.bfloat16)
    dev = [t.cuda() for t in (x8, w8, xs, ws)]
    got, acc = ops.linear_int8_scaled(*dev, want_acc=True)
    assert torch.equal(acc.cpu(), want_acc)
    assert torch.equal(got.cpu(), want)
    assert torch.equal(ops.linear_int8_scaled(*dev, bias=bias.cuda()).cpu(), want_b)
    gelu = ops.linear_int8_scaled(*dev, bias=bias.cuda(), gelu=True).cpu()
    want_g = ob.orc().gelu_tanh(want_b.view(torch.int16).numpy().view(np.uint16))
    assert rel_l2(gelu.float().numpy(), ob.bf16_to_f32(want_g)) <= 2e-3
    ops.poll_status()


@pytest.mark.parametrize("M", [8, 9, 16, 17, 32])
@pytest.mark.parametrize("K,N", [(16, 4736), (240, 4752), (256, 4752), (528, 9472), (528, 9488), (3072, 9472), (3088, 9472), (3088, 4736),
                                 (3856, 4352), (8176, 9488), (8192, 14208), (8192, 14224), (10240, 4096), (10240, 4100)])
def test_linear_on_both_sides_of_the_lines_of_few_rows(ops, monkeypatch, M, K, N):
    """Numbers of rows, columns (waves of 4736 on 148 SMs) and k at which the dispatch goes from the few-rows kernel to the tile
    kernel: the same bits from both, and never one that takes half as long again as the other would."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x8, w8 = (torch.randint(-128, 128, s, generator=g, device="cuda", dtype=torch.int8) for s in ((M, K), (N, K)))
    xs, ws = torch.rand(M, generator=g, device="cuda"), torch.rand(N, generator=g, device="cuda")

    def run():
        out = ops.linear_int8_scaled(x8, w8, xs, ws)
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            for _ in range(10):
                ops.linear_int8_scaled(x8, w8, xs, ws, out=out)
        times = []
        for _ in range(20):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            graph.replay()
            end.record()
            end.synchronize()
            times.append(start.elapsed_time(end))
        return out, min(times)

    got, time = run()
    monkeypatch.setenv("DIFB200_GEMM_FORM", "0,0,0")  # no such form: the tile kernel's own choice
    want, tile_time = run()
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert time <= 1.5 * tile_time, (time, tile_time)
    ops.poll_status()


@pytest.mark.parametrize("M,K,N", [(8, 256, 18944), (8, 256, 18960), (8, 1024, 32768), (4, 2048, 32768), (2, 3072, 20000), (3, 3072, 14208), (3, 3072, 14224), (16, 512, 12288), (32, 256, 16384)])
def test_w8a8_linear_on_both_sides_of_the_lines_of_few_rows(ops, monkeypatch, M, K, N):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    w8 = torch.randint(-128, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
    ws = torch.rand(N, generator=g, device="cuda") * 0.01
    got = ops.w8a8_linear(x, w8, ws)
    monkeypatch.setenv("DIFB200_GEMM_FORM", "0,0,0")
    assert torch.equal(got.view(torch.int16), ops.w8a8_linear(x, w8, ws).view(torch.int16))
    ops.poll_status()


@pytest.mark.parametrize("packer", ["quantize", "pack"])
@pytest.mark.parametrize("rows", [1, 9, 30])
def test_linear_of_few_rows_directly_behind_the_kernel_that_writes_its_weights(ops, rows, packer):
    """The weights' codes are written into the same buffer again and again, by kernels that let the linear start early, with no
    synchronisation in between: every linear reads the codes written directly in front of it."""
    import torch
    # a 256-wide quantiser with one batch of four rows per CTA, three CTAs on an SM, lets the next kernel start when it starts itself
    N = 1200
    assert N <= 3 * 4 * torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(rows)
    weights = [torch.randn((N, 2048), generator=g, device="cuda").to(torch.bfloat16) for _ in range(3)]
    codes, scales = torch.empty((N, 2048), dtype=torch.int8, device="cuda"), torch.empty(N, device="cuda")
    x8 = torch.randint(-127, 128, (rows, 2048), generator=g, device="cuda", dtype=torch.int8)
    xs = torch.rand(rows, generator=g, device="cuda")
    from diffusion_compiler_b200 import _lib

    def write(w):
        if packer == "quantize":
            ops.quantize_int8_rows([w], 2, out=(codes, scales))
        else:
            ops._call(_lib.lib().difb200_quantize_weight_rows, 0, w.data_ptr(), None, N, 2048, 2, 0, codes.data_ptr(),
                      scales.data_ptr())

    want = []
    for w in weights:
        write(w)
        torch.cuda.synchronize()
        want.append(((x8.double() @ codes.double().T).float() * xs[:, None] * scales[None]).to(torch.bfloat16))  # exact sums
    torch.cuda.synchronize()
    got = []
    for _ in range(4):
        for w in weights:
            torch.cuda._sleep(400_000)  # clocks: the host enqueues both meanwhile
            write(w)
            got.append(ops.linear_int8_scaled(x8, codes, xs, scales))
    for i, out in enumerate(got):
        assert torch.equal(out.view(torch.int16), want[i % 3].view(torch.int16)), i
    ops.poll_status()


@pytest.mark.parametrize("rows", [1, 16, 30])
def test_w8a8_linear_of_few_rows_matches_two_calls(ops, rows):
    """The single call, whose weights are requested before the quantiser in front is complete, back to back."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = [torch.randn((rows, 3072), generator=g, device="cuda").to(torch.bfloat16) for _ in range(4)]
    w8 = torch.randint(-127, 128, (520, 3072), generator=g, device="cuda", dtype=torch.int8)
    ws = torch.rand(520, generator=g, device="cuda") * 0.01
    want = []
    for a in x:
        codes, scales = ops.quantize_int8_rows([a], 2)
        torch.cuda.synchronize()
        want.append(ops.linear_int8_scaled(codes, w8, scales, ws))
        torch.cuda.synchronize()
    got = [ops.w8a8_linear(a, w8, ws) for a in x + x]
    for i, out in enumerate(got):
        assert torch.equal(out.view(torch.int16), want[i % 4].view(torch.int16)), i
    ops.poll_status()


@pytest.mark.parametrize("M,K", [(1, 256), (8, 768), (8, 1024), (4, 2048), (2, 3072), (3, 3072), (2, 2816), (1, 8192), (1, 9216),
                                 (2, 4096), (9, 1024)])
@pytest.mark.parametrize("N", [1, 17, 520, 9000])  # fewer tiles than the machine holds CTAs, and more
def test_w8a8_linear_in_one_launch_bit_exact(ops, M, K, N):
    """The one launch for the fewest rows (up to a block of 1024 columns for every warp, partial blocks, just too many
    of them) against quantise + linear: outputs, the codes and scales left in the caller's scratch, a clip, an input whose
    quotients leave the split product's range, and a call in place."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(M * K + N)
    x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    x[0, :7] = 2.0 ** 113 if M > 2 else 40.0
    w8 = torch.randint(-128, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
    ws = torch.rand(N, generator=g, device="cuda") * 0.01
    bias = torch.randn(N, generator=g, device="cuda").to(torch.bfloat16)
    for clip in (1.0, 0.9):
        codes, scales = ops.quantize_int8_rows([x], 2, clip)
        want = ops.linear_int8_scaled(codes, w8, scales, ws, bias=bias, gelu=True)
        scratch = (torch.zeros_like(codes), torch.zeros_like(scales))
        got = ops.w8a8_linear(x, w8, ws, bias=bias, gelu=True, clip=clip, scratch=scratch)
        assert torch.equal(got.view(torch.int16), want.view(torch.int16))
        assert torch.equal(scratch[0], codes) and torch.equal(scratch[1], scales)
        assert torch.equal(ops.w8a8_linear(x, w8, ws, clip=clip).view(torch.int16),
                           ops.linear_int8_scaled(codes, w8, scales, ws).view(torch.int16))
    if N <= K:
        room = x.clone()
        want = ops.w8a8_linear(x, w8, ws)
        got = ops.w8a8_linear(room, w8, ws, out=room.view(-1)[:M * N].view(M, N))
        assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    ops.poll_status()


def test_w8a8_linear_end_to_end_single_layer(ops):
    """The single-layer benchmark case (M=1024, K=N=3072, H256ConvRot activations, bias): GPU quant + GEMM chained."""
    import torch
    rng = np.random.default_rng(0)
    ob.orc().lib.orc_set_threads(8)
    M, K, N = 1024, 3072, 3072
    x = activations(rng, M, K)
    w8, ws = _weights(rng, N, K, 2)
    bias = bf16_normal(rng, (N,), 0.01)
    x8, xs = ob.orc().quantize_int8_rows([x], 2, 1.0)
    want = ob.orc().bias_add(ob.orc().linear_int8_scaled(x8, w8, xs, ws), bias)
    codes, scales = ops.quantize_int8_rows([to_torch_bf16(x)], 2)
    got = ops.linear_int8_scaled(codes, torch.from_numpy(w8).cuda(), scales, torch.from_numpy(ws).cuda(),
                                 bias=to_torch_bf16(bias))
    torch.cuda.synchronize()
    assert np.array_equal(codes.cpu().numpy(), x8)
    assert np.array_equal(from_torch_bf16(got), want)
    ops.poll_status()


def test_w8a8_linear_single_call_matches_two_calls(ops):
    """difb200_w8a8_linear (caller scratch) == quantize + linear through their own entry points."""
    import torch
    rng = np.random.default_rng(3)
    M, K, N = 640, 1024, 768
    x = to_torch_bf16(activations(rng, M, K))
    w8, ws = _weights(rng, N, K, 2)
    w8, ws = torch.from_numpy(w8).cuda(), torch.from_numpy(ws).cuda()
    bias = to_torch_bf16(bf16_normal(rng, (N,), 0.01))
    codes, scales = ops.quantize_int8_rows([x], 2)
    want = ops.linear_int8_scaled(codes, w8, scales, ws, bias=bias, gelu=True)
    got = ops.w8a8_linear(x, w8, ws, bias=bias, gelu=True)
    torch.cuda.synchronize()
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    ops.poll_status()


@pytest.mark.parametrize("form", ["2,256,1", "2,192,1", "2,128,1", "1,256,1", "1,128,1", "1,128,2", "1,128,4"])
@pytest.mark.parametrize("blocks", [1, 3, 4, 5, 6, 7, 8, 9, 15])
def test_w8a8_linear_with_k_blocks_around_the_ring_depth(ops, monkeypatch, form, blocks):
    """The single call requests the weights of the first k-blocks of a CTA's first tile ahead of everything else: fewer
    k-blocks than the ring has stages (4 to 7), as many, more, a last one that is not full, and several tiles per CTA. The
    same bits as the two calls, whose GEMM requests nothing ahead."""
    import torch
    split = int(form[-1])
    if split > blocks:
        pytest.skip("a split form needs a k-block per CTA")
    monkeypatch.setenv("DIFB200_GEMM_FORM", form)
    g = torch.Generator(device="cuda").manual_seed(blocks)
    M, N, K = (300, 640, 128 * blocks - 16) if split > 1 else (2700, 2600, 128 * blocks - 16)
    x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    w8 = torch.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
    ws = torch.rand(N, generator=g, device="cuda") * 0.01
    codes, scales = ops.quantize_int8_rows([x], 1)
    want = ops.linear_int8_scaled(codes, w8, scales, ws)
    torch.cuda.synchronize()
    for _ in range(3):
        got = ops.w8a8_linear(x, w8, ws, implementation=1)
        assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    acc = (codes.double() @ w8.double().T).float()  # exact: |sum| < 2^24
    assert torch.equal(((acc * scales[:, None]) * ws[None]).to(torch.bfloat16).view(torch.int16), want.view(torch.int16))
    ops.poll_status()


@pytest.mark.parametrize("impl", [2, 3, 5, 6])
@pytest.mark.parametrize("K", [256, 1024, 3072, 12288])  # rows of one warp and of several, one and three blocks per warp
def test_weight_scale_search_where_its_fp32_sums_do_not_decide(ops, impl, K):
    """The search compares fp32 sums first; rows in which candidates tie (constant magnitudes, one non-zero weight, zeros)
    or whose squares leave the range of fp32 (1e-18, 1e18) are decided in doubles. Such rows between ordinary ones,
    twice (rows of a CTA are not in step), bit for bit against the CPU restatement."""
    import torch
    rng = np.random.default_rng(impl + K)
    N = 1400
    w = (rng.standard_normal((N, K)) * 0.02).astype(np.float32)
    w[0::7] = np.where(rng.random((len(w[0::7]), K)) < 0.5, -0.5, 0.5)
    w[1::7] = 0
    w[1::14, 3] = 1
    w[2::7] *= 1e-18
    w[3::7] *= 1e18
    w[4::14] = 0.25
    w = ob.f32_to_bf16(w)
    want_codes, want_scales = ob.orc().quantize_weight_rows(w, impl, mse=True)
    dw = torch.from_numpy(w.view(np.int16)).cuda().view(torch.bfloat16)
    for _ in range(2):
        codes, scales = ops.quantize_weight_rows(dw, impl, mse_scale=True)
        torch.cuda.synchronize()
        assert np.array_equal(scales.cpu().numpy().view(np.uint32), want_scales.view(np.uint32))
        assert np.array_equal(codes.cpu().numpy(), want_codes)
    ops.poll_status()


def test_weight_rows_equal_the_reference_packers_own_files(ops):
    """The GPU weight quantiser against whole runs of the reference's own offline packer
    (rewrite_named_linear_w8a8 of reference tools/difflux2sample.cpp; its cache tensors are the
    committed fixture tests/golden/packer_mse_scale.npz): given the packer's input-equalisation
    vector, the codes and scales are the packer's, bit for bit, with and without the MSE search."""
    import os
    import torch
    data = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "packer_mse_scale.npz"))
    keys = sorted({k.split("/")[0] for k in data.files if k.startswith("pack_")})
    assert len(keys) == 6
    for key in keys:
        impl = int(key.split("_")[1][4:])
        equalise, mse = key.split("_")[2] == "eq1", key.split("_")[3] == "mse1"
        w = np.ascontiguousarray(data[key + "/weight"])
        dw = torch.from_numpy(w.view(np.int16)).cuda().view(torch.bfloat16)
        deq = None
        if equalise:
            eq = np.ascontiguousarray(data[key + "/input_scale"]).reshape(-1)
            deq = torch.from_numpy(eq.view(np.int16)).cuda().view(torch.bfloat16)
        if impl in (4, 7) and (equalise or mse):
            # the 4096-wide variants are packed here without the two options only: refused, not approximated
            from diffusion_compiler_b200 import _lib
            with pytest.raises(_lib.Difb200Error) as info:
                ops.quantize_weight_rows(dw, impl, mse_scale=mse, input_scale=deq)
            assert info.value.status == 2
            continue
        codes, scales = ops.quantize_weight_rows(dw, impl, mse_scale=mse, input_scale=deq)
        torch.cuda.synchronize()
        assert np.array_equal(scales.cpu().numpy().view(np.uint32), data[key + "/scale_bits"]), key
        assert np.array_equal(codes.cpu().numpy(), data[key + "/codes"]), key
    ops.poll_status()
