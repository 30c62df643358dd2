"""Kernels that start while the one in front of them on the stream still runs (the GEMM behind a quantiser or an attention,
the attention behind its operands, its split items behind the whole ones): results where the kernel in front has just
written the operands, weights included, back to back without a synchronisation and replayed from a graph."""
import pytest

pytestmark = pytest.mark.gpu


def _bits(t):
    return t.contiguous().view(__import__("torch").int16)


@pytest.mark.parametrize("rows", [1, 2, 130, 700, 4159])
def test_linear_behind_the_packing_of_its_weights(rows):
    import torch
    from diffusion_compiler_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows)
    normal = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    K, N = 1024, 1536
    x, bias = normal(rows, K), normal(N)
    weights = [normal(N, K) for _ in range(4)]
    want = []
    for w in weights:  # one launch at a time
        codes, scales = ops.quantize_weight_rows(w, 2)
        torch.cuda.synchronize()
        x8, xs = ops.quantize_int8_rows([x], 2)[:2]
        torch.cuda.synchronize()
        want.append(ops.linear_int8_scaled(x8, codes, xs, scales, bias=bias))
        torch.cuda.synchronize()
    w8, ws = torch.zeros((N, K), dtype=torch.int8, device="cuda"), torch.zeros(N, device="cuda")
    got = []
    for w in weights:  # weights into the same buffers, the linear right behind
        codes, scales = ops.quantize_weight_rows(w, 2)
        w8.copy_(codes)
        ws.copy_(scales)
        got.append(ops.w8a8_linear(x, w8, ws, bias=bias))
        x8, xs = ops.quantize_int8_rows([x], 2)[:2]
        codes, scales = ops.quantize_weight_rows(w, 2)
        got.append(ops.linear_int8_scaled(x8, codes, xs, scales, bias=bias))
    torch.cuda.synchronize()
    ops.poll_status()
    for i, out in enumerate(got):
        assert torch.equal(_bits(out), _bits(want[i // 2])), i


@pytest.mark.parametrize("tokens,heads", [(300, 4), (1700, 24), (2304, 24), (2048, 24)])  # no split; 3, 2 and (all SMs) 3 CTAs
def test_attention_back_to_back_and_from_a_graph(tokens, heads):
    import torch
    from diffusion_compiler_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(tokens)
    sets = [[torch.randn((1, tokens, heads, 128), generator=g, device="cuda").to(torch.bfloat16) for _ in range(3)]
            for _ in range(3)]
    want = []
    for q, k, v in sets:
        want.append(ops.attention(q, k, v))
        torch.cuda.synchronize()
    got = [ops.attention(*s) for s in sets + sets]
    q, k, v = (t.clone() for t in sets[0])
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        ops.attention(q, k, v)
    torch.cuda.current_stream().wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = ops.attention(q, k, v)
    for s in sets:
        for a, b in zip((q, k, v), s):
            a.copy_(b)
        graph.replay()
        got.append(out.clone())
    torch.cuda.synchronize()
    ops.poll_status()
    for i, o in enumerate(got):
        assert torch.equal(_bits(o), _bits(want[i % 3])), i


@pytest.mark.parametrize("rows", [2, 130, 4159])
def test_linear_from_a_graph_behind_new_weights(rows):
    """The captured single call, which requests its first weights before its quantiser is done: between two replays the
    inputs and the weights are overwritten on the stream, by copies and by a packing kernel that is captured in front."""
    import torch
    from diffusion_compiler_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows)
    normal = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    K, N = 1024, 1536
    sets = [(normal(rows, K), normal(N, K)) for _ in range(4)]
    want = []
    for x, w in sets:
        codes, scales = ops.quantize_weight_rows(w, 2)
        torch.cuda.synchronize()
        want.append(ops.w8a8_linear(x, codes, scales))
        torch.cuda.synchronize()
    x, w = (t.clone() for t in sets[0])
    w8, ws = ops.quantize_weight_rows(w, 2)
    graphs = []
    for packed in (False, True):  # the weights as they stand; packed inside the graph
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            ops.w8a8_linear(x, w8, ws)
        torch.cuda.current_stream().wait_stream(stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = ops.w8a8_linear(x, *(ops.quantize_weight_rows(w, 2) if packed else (w8, ws)))
        graphs.append((graph, out))
    got = []
    for i, (nx, nw) in enumerate(sets + sets):
        x.copy_(nx)
        w.copy_(nw)
        codes, scales = ops.quantize_weight_rows(w, 2)
        w8.copy_(codes)
        ws.copy_(scales)
        graph, out = graphs[i // len(sets)]
        graph.replay()
        got.append(out.clone())
    torch.cuda.synchronize()
    ops.poll_status()
    for i, o in enumerate(got):
        assert torch.equal(_bits(o), _bits(want[i % len(sets)])), i


@pytest.mark.parametrize("tokens", [130, 1700, 2048])  # no split; a split behind the whole items; one that starts together
def test_gemm_directly_behind_an_attention(tokens):
    """LinearInt8Scaled as the next launch after the attention's, with nothing in between: its scales are the attention's
    output (reinterpreted), so that a GEMM that read before the attention was done would show; also from a graph."""
    import torch
    from diffusion_compiler_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(tokens)
    H, N, K = 24, 256, 1024
    q, k, v = (torch.randn((1, tokens, H, 128), generator=g, device="cuda").to(torch.bfloat16) for _ in range(3))
    x8 = torch.randint(-127, 128, (tokens, K), generator=g, device="cuda", dtype=torch.int8)
    w8 = torch.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
    ws = torch.rand(N, generator=g, device="cuda")
    out = torch.empty_like(q)
    scales = out.view(torch.float32).view(-1)  # pairs of bf16 outputs as fp32 row scales, from the last rows of the output
    scales = scales[scales.numel() - tokens:]
    y = torch.empty((tokens, N), dtype=torch.bfloat16, device="cuda")

    def both():
        ops.attention(q, k, v, out=out)
        ops.linear_int8_scaled(x8, w8, scales, ws, out=y)

    ops.attention(q, k, v, out=out)
    torch.cuda.synchronize()
    want = ops.linear_int8_scaled(x8, w8, scales, ws).clone()
    torch.cuda.synchronize()
    got = []
    for _ in range(4):
        out.zero_()
        both()
        got.append(y.clone())
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        both()
    torch.cuda.current_stream().wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        both()
    for _ in range(4):
        out.zero_()
        y.zero_()
        graph.replay()
        got.append(y.clone())
    torch.cuda.synchronize()
    ops.poll_status()
    assert bool(torch.isfinite(want.float()).all()) and bool(want.float().any())
    for i, o in enumerate(got):
        assert torch.equal(_bits(o), _bits(want)), i


@pytest.mark.parametrize("rows,K", [(1, 256), (2, 3072), (8, 1024)])  # with the quantiser in the same launch: at most 8 blocks of 1024 columns
def test_linears_of_few_rows_one_behind_the_other(rows, K):
    """Single-call linears in one launch each, which starts as the CTAs of the one in front end: every one reads what the
    last one wrote and writes the buffer that the last one read, on the stream and from a graph. (Behind a kernel that lets it start
    earlier: "linear" of 4 rows below.)"""
    import torch
    from diffusion_compiler_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows * K)
    normal = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    x, weights = normal(rows, K), [ops.quantize_weight_rows(normal(K, K), 2) for _ in range(4)]
    want = x
    for i in range(12):
        want = ops.w8a8_linear(want, *weights[i % 4]).clone()
        torch.cuda.synchronize()
    assert bool(torch.isfinite(want.float()).all()) and bool(want.float().any())
    a, b = x.clone(), torch.empty_like(x)

    def chain():
        for i in range(6):
            ops.w8a8_linear(a, *weights[2 * i % 4], out=b)
            ops.w8a8_linear(b, *weights[(2 * i + 1) % 4], out=a)

    got = []
    for _ in range(3):
        a.copy_(x)
        chain()
        got.append(a.clone())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain()
    for _ in range(3):
        a.copy_(x)
        graph.replay()
        got.append(a.clone())
    torch.cuda.synchronize()
    ops.poll_status()
    for i, o in enumerate(got):
        assert torch.equal(_bits(o), _bits(want)), i


def _readers(rows):
    """name -> a call whose first kernel, with nothing else in front of it, reads bf16 rows [rows, 1024] (8 heads of 128)."""
    import ctypes as C

    import torch
    from diffusion_compiler_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(7)
    normal = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    K = 1024
    vector, table, equalisation = normal(K), normal(1200, 96), normal(K).abs().clamp(0.5, 2.0)
    w8, ws = ops.quantize_weight_rows(normal(1536, K), 2)
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    stream = lambda: C.c_void_p(torch.cuda.current_stream().cuda_stream)  # noqa: E731

    gated, halves = (torch.zeros((rows, columns), dtype=torch.bfloat16, device="cuda") for columns in (K, K // 2))
    codes, scales = torch.zeros((rows, K), dtype=torch.int8, device="cuda"), torch.zeros(8 * rows, device="cuda")

    def glue(name, o, *args):
        _lib.check(getattr(_lib.lib(), name)(*(ptr(a) if torch.is_tensor(a) else a for a in args), stream()))
        return o

    def rope(x):
        _lib.check(_lib.lib().difb200_qk_norm_rope_quant(ptr(x), ptr(vector), ptr(table), ptr(table), None, ptr(codes), ptr(scales), 2,
                                                         x.shape[0], 8, 96, 96, x.shape[0], 1200, 0, 1e-5, 0, stream()))
        return codes, scales

    heads = lambda x: x.view(1, x.shape[0], 8, 128)  # noqa: E731
    calls = {"variant %d" % i: (lambda x, i=i: ops.quantize_int8_rows([x if i not in (4, 7) else x.view(-1, 4096)], i)) for i in range(1, 8)}
    calls.update({
        "residual": lambda x: ops.quantize_int8_rows([x], 3, residual=True),
        "two inputs": lambda x: ops.quantize_int8_rows([x, x], 2),
        "direct heads": lambda x: ops.quantize_int8_rows([x.view(-1, 128)], 1),
        "packing": lambda x: ops.quantize_weight_rows(x, 2, mse_scale=True, input_scale=equalisation),
        "rms norm": lambda x: ops.rms_norm_modulate_quant(x, vector, x, x),
        "layer norm": lambda x: ops.layer_norm_modulate_quant(x, vector, vector, x, x),
        "linear": lambda x: ops.w8a8_linear(x, w8, ws),
        "attention": lambda x: ops.attention(heads(x), heads(x), heads(x)),
        "gate": lambda x: glue("difb200_residual_gate", gated, x, x, x, gated, 2, rows, K, rows),
        "swiglu": lambda x: glue("difb200_swiglu", halves, x, halves, 2, rows, K // 2, K, 0, 0),
        "rope": rope,
    })
    return calls


@pytest.mark.parametrize("rows", [4, 332, 1200])
def test_kernels_launched_ahead_read_what_the_kernel_in_front_writes(rows):
    """Every kernel that is launched ahead, behind a quantiser that lets it start at once (a 256-wide one, all of whose rows are in one
    batch per CTA: its CTAs say so when they start) and whose codes (as the bits of bf16 numbers) are what it reads: the
    buffer holds other numbers until that quantiser is done. A delay in front lets the host enqueue both before the first starts."""
    import torch
    from diffusion_compiler_b200 import ops
    # four rows of 2048 columns per CTA, three CTAs on an SM
    assert rows <= 3 * 4 * torch.cuda.get_device_properties(0).multi_processor_count
    unit = ops.quantize_int8_rows([torch.eye(256, device="cuda").to(torch.bfloat16)], 5)[0].float()
    assert bool((unit.abs() == 127).all())  # the rotation is orthogonal, all its entries +-1/16
    g = torch.Generator(device="cuda").manual_seed(rows)
    sources = [0.55 + 0.2 * torch.rand((rows, 2048), generator=g, device="cuda") for _ in range(2)]
    for s in sources:
        s[:, 5] = 1.0  # the largest of a row: its code with clip 2 is 64, the others' are 34 to 49
    sources = [(s.view(rows, 8, 256) @ (unit.T / (127 * 16))).view(rows, 2048).to(torch.bfloat16) for s in sources]
    codes, scales = torch.zeros((rows, 2048), dtype=torch.int8, device="cuda"), torch.zeros(rows, device="cuda")
    x = codes.view(torch.bfloat16)
    write = lambda i: ops.quantize_int8_rows([sources[i]], 2, clip=2.0, out=(codes, scales))  # noqa: E731
    for i in range(2):
        write(i)
        assert 32 <= int(codes.min()) and int(codes.max()) <= 66, "the codes are not the numbers that were rotated back"
    tensors = lambda r: [r] if torch.is_tensor(r) else list(r)  # noqa: E731
    for name, call in _readers(rows).items():
        want = []
        for i in range(2):
            write(i)
            torch.cuda.synchronize()
            want.append([t.clone() for t in tensors(call(x))])
            torch.cuda.synchronize()
        assert any(not torch.equal(a, b) for a, b in zip(*want)), name
        for i in range(6):
            torch.cuda._sleep(400_000)  # clocks, about 0.2 ms
            write(i % 2)
            got = tensors(call(x))
            torch.cuda.synchronize()
            for a, b in zip(got, want[i % 2]):
                assert torch.equal(a.view(torch.uint8), b.view(torch.uint8)), (name, i)
    ops.poll_status()
