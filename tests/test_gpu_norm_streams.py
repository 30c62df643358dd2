"""Norm ops whose row statistic passes from one kernel to the next, used from several streams and threads at once, under
stream capture and in place: the memory it passes through belongs to one call, so every result equals the one of a
call by itself."""
import threading

import numpy as np
import pytest

from helpers import bf16_normal, to_torch_bf16

pytestmark = pytest.mark.gpu


def _operands(seed, rows, K):
    rng = np.random.default_rng(seed)
    t = lambda *shape, std=1.0: to_torch_bf16(bf16_normal(rng, shape, std))  # noqa: E731
    return t(rows, K, std=1.0 + seed), t(K), t(K, std=0.1), t(rows, K, std=0.1), t(rows, K, std=0.1)


def _call(ops, layer, x, w, b, s, h):
    return ops.layer_norm_modulate_quant(x, w, b, s, h, 1e-6) if layer else ops.rms_norm_modulate_quant(x, w, s, h, 1e-5)


def _same(a, b):
    import torch
    return torch.equal(a[0], b[0]) and torch.equal(a[1].view(torch.int32), b[1].view(torch.int32))


@pytest.mark.parametrize("layer", [False, True])
def test_two_streams_do_not_share_the_statistics(layer):
    import torch
    from diffusion_compiler_b200 import ops
    sides = [_operands(k, 700 + 900 * k, 3072) for k in range(2)]  # the second needs more scratch than the first
    alone = [_call(ops, layer, *o) for o in sides]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in sides]
    got = [[], []]
    for _ in range(20):
        for k, stream in enumerate(streams):
            with torch.cuda.stream(stream):
                got[k].append(_call(ops, layer, *sides[k]))
    torch.cuda.synchronize()
    assert all(_same(alone[k], g) for k in range(2) for g in got[k])


def test_threads_with_streams_of_their_own():
    import torch
    from diffusion_compiler_b200 import ops
    sides = [_operands(k, 100 + 400 * k, 1024) for k in range(4)]
    alone = [_call(ops, k % 2 == 1, *o) for k, o in enumerate(sides)]
    torch.cuda.synchronize()
    got, errors = [None] * 4, []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                got[k] = [_call(ops, k % 2 == 1, *sides[k]) for _ in range(30)]
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    assert all(_same(alone[k], g) for k in range(4) for g in got[k])


def test_captured_call_keeps_its_statistics_apart_from_later_calls():
    """A captured call replays on another stream while plain calls with more rows run beside it."""
    import torch
    from diffusion_compiler_b200 import ops
    small, large = _operands(1, 300, 1024), _operands(2, 5000, 1024)
    want, beside = _call(ops, True, *small), _call(ops, True, *large)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = _call(ops, True, *small)
    side = torch.cuda.Stream()
    others = []
    for _ in range(10):
        graph.replay()
        with torch.cuda.stream(side):
            others.append(_call(ops, True, *large))
    torch.cuda.synchronize()
    assert _same(want, got) and all(_same(beside, o) for o in others)


@pytest.mark.parametrize("K", [3072, 1280])
@pytest.mark.parametrize("over", ["x", "scale", "shift"])
def test_norm_ops_in_place(K, over):
    """The output in the place of an input: the statistic then cannot stand in the output's rows."""
    import ctypes as C

    import torch
    from diffusion_compiler_b200 import _lib
    lib = _lib.lib()
    x, w, b, s, h = _operands(3, 200, K)
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def run(layer, out, x, s, h):
        if layer:
            _lib.check(lib.difb200_layer_norm_modulate(p(x), p(w), p(b), p(s), p(h), p(out), 2, 200, K, 200, 1e-6, stream))
        else:
            _lib.check(lib.difb200_rms_norm_modulate(p(x), p(w), p(s), p(h), p(out), 2, 200, K, 1e-5, stream))
        return out

    for layer in (False, True):
        want = run(layer, torch.empty_like(x), x, s, h)
        own = {"x": x.clone(), "scale": s.clone(), "shift": h.clone()}
        got = run(layer, own[over], own["x"], own["scale"], own["shift"])
        torch.cuda.synchronize()
        assert torch.equal(want.view(torch.int16), got.view(torch.int16)), layer


def _rows_of_all_kinds(rows, cols, g):
    """Outliers, equal numbers (ties in every step), rows whose sums meet powers of two, zeros, steps over many binades, infinities, NaN."""
    import torch
    x = torch.randn((rows, cols), generator=g, device="cuda")
    x[:, :: cols // 32] *= 16.0  # (and so that single parts cross several binades)
    x[100:400] = x[100:400].round()
    x[400:500] = torch.exp2(torch.arange(100, device="cuda").remainder(12).float() - 6.0)[:, None]
    x[500:600] *= torch.exp(4.0 * torch.randn((100, cols), generator=g, device="cuda"))
    x[600:650, : cols // 2] = 0.0
    x[650], x[651, 7], x[652, 9], x[653] = 0.0, float("inf"), float("nan"), x[653] * 2.0**-40
    x[654:700] *= 2.0 ** torch.arange(-23, 23, device="cuda").float()[:, None]
    return x.to(torch.bfloat16)


@pytest.mark.parametrize("layer", [False, True])
@pytest.mark.parametrize("cols", [1024, 2048, 2816, 3072, 8192])
def test_statistics_of_few_rows_are_those_of_many(layer, cols):
    """Few rows have their sums of squares from a kernel that cuts the sequential chain in 16 parts; many from the chain itself. Rows are
    independent, so any slice of a tensor gives the bits of the whole: with outliers, equal numbers (ties in every step), rows whose
    sums meet powers of two, zeros, steps over many binades, infinities and NaN."""
    import torch
    from diffusion_compiler_b200 import ops
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = 20 * sms + 5
    g = torch.Generator(device="cuda").manual_seed(cols)
    x = _rows_of_all_kinds(rows, cols, g)
    normal = lambda *s: (0.1 * torch.randn(s, generator=g, device="cuda")).to(torch.bfloat16)  # noqa: E731
    w, b, s, h = normal(cols) + 1, normal(cols), normal(rows, cols), normal(rows, cols)
    want = _call(ops, layer, x, w, b, s, h)
    for first, count in ((0, 1), (3, sms - 8), (90, 502), (600, sms + 1), (0, rows - 5), (5, rows - 5)):
        at = slice(first, first + count)
        got = _call(ops, layer, x[at].contiguous(), w, b, s[at].contiguous(), h[at].contiguous())
        assert torch.equal(got[0], want[0][at]) and torch.equal(got[1].view(torch.int32), want[1][at].view(torch.int32)), (first, count)


@pytest.mark.parametrize("layer", [False, True])
@pytest.mark.parametrize("cols", [1024, 1152, 2048, 2816, 3072, 4992, 8192])
def test_sums_in_parts_are_the_chains(layer, cols):
    """The statistics themselves, all bits: a tensor of more rows than are cut in parts has them from the chain, its slices from the parts. A
    wrong last bit shows here; behind a norm and a quantiser it hardly would."""
    import ctypes as C

    import torch
    from diffusion_compiler_b200 import _lib
    lib = _lib.lib()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    line = (20 if cols >= 2048 else 4) * sms  # the most rows that are cut in parts

    def statistics(x):
        pairs = torch.empty((x.shape[0], 2), device="cuda")
        _lib.check(lib.difb200_test_row_statistics(C.c_void_p(x.data_ptr()), x.shape[0], cols, 1e-5, int(layer), C.c_void_p(pairs.data_ptr()),
                                                   C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return pairs.view(torch.int32)

    for seed in range(6):
        x = _rows_of_all_kinds(20 * sms + 700, cols, torch.Generator(device="cuda").manual_seed(100 * cols + seed))
        want = statistics(x)
        starts = list(range(0, x.shape[0], line - seed))
        for first, count in [(0, 1), (101, sms + seed), (400, 333)] + [(i, line - seed) for i in starts]:
            got = statistics(x[first:first + count].contiguous())
            assert torch.equal(got, want[first:first + count]), (seed, first)
