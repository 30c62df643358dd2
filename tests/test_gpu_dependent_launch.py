"""Kernels that start while the one in front of them on the stream still runs (the GEMM behind a quantiser, the attention
behind its operands, its split items behind the whole ones): results where the kernel in front has just written the
operands, weights included, back to back without a synchronisation and replayed from a graph."""
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
