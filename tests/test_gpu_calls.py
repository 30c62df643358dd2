"""The native binding for torch tensors against the general way through ctypes: the same bits from both, and everything the
binding does not serve itself (copies, conversions, other devices' rules, errors) as before."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def both(monkeypatch):
    """Runs a call natively and, with a binding that serves nothing, the general way."""
    from diffusion_compiler_b200 import ops

    class Nothing:
        def __getattr__(self, name):
            return lambda *args: None

    def run(call):
        native = call()
        with monkeypatch.context() as m:
            m.setattr(ops, "_calls", Nothing)
            general = call()
        return native, general

    return run


def _same(a, b):
    import torch
    if isinstance(a, tuple):
        return len(a) == len(b) and all(_same(x, y) for x, y in zip(a, b))
    return (a.dtype == b.dtype and a.shape == b.shape and a.device == b.device
            and torch.equal(a.contiguous().view(torch.uint8), b.contiguous().view(torch.uint8)))


def test_native_calls_equal_the_general_way(both):
    import torch
    from diffusion_compiler_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(1)
    n = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    x, y, bias, weight = n(3, 7, 512), n(3, 7, 256), n(48), n(512)
    w8, ws = ops.quantize_int8_rows([n(48, 512)], 2)
    rows, mods = n(20, 512), n(20, 512)
    q, k, v = n(2, 70, 4, 128), n(2, 70, 2, 128), n(2, 70, 2, 128)
    valid = (torch.rand((2, 70), generator=g, device="cuda") < 0.8).to(torch.uint8)
    calls = [
        lambda: ops.w8a8_linear(x, w8, ws, bias=bias, gelu=True),
        lambda: ops.w8a8_linear(x[0, 0], w8, ws, implementation=3, clip=0.9),
        lambda: ops.w8a8_linear(x, w8, ws, implementation=2.0, clip=1),
        lambda: ops.w8a8_linear(x.transpose(0, 1), w8, ws),               # a copy first
        lambda: ops.w8a8_linear(x.clone().requires_grad_(), w8, ws),
        lambda: ops.quantize_int8_rows([x, y], 5, clip=0.99),
        lambda: ops.quantize_int8_rows(x, 2),
        lambda: ops.quantize_int8_rows((y,), 1),
        lambda: ops.rms_norm_modulate_quant(rows, None, mods, mods),
        lambda: ops.rms_norm_modulate_quant(rows, weight, mods, rows, 1e-6, 3, 0.95),
        lambda: ops.layer_norm_modulate_quant(rows, weight, weight, mods[:4], mods[4:8]),
        lambda: ops.attention(q, k, v),
        lambda: ops.attention(q, k, v, key_valid=valid, scale=0.1),
        lambda: ops.attention(q, k, v, key_valid=valid.bool()),
    ]
    for i, call in enumerate(calls):
        native, general = both(call)
        assert _same(native, general), i
    wide = n(64)  # more entries than are read
    native, general = both(lambda: ops.w8a8_linear(x, w8, torch.cat([ws, ws]), bias=wide))
    assert _same(native, ops.w8a8_linear(x, w8, ws, bias=wide[:48])) and _same(native, general)
    stream = torch.cuda.Stream()  # the current stream's, whichever it is
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        native, general = both(calls[0])
    stream.synchronize()
    assert _same(native, general)
    for bad in (lambda: ops.quantize_int8_rows([n(4, 100)], 2), lambda: ops.quantize_int8_rows([x], 2, clip=0.0),
                lambda: ops.attention(n(1, 5, 2, 64), n(1, 5, 2, 64), n(1, 5, 2, 64))):
        with pytest.raises(_lib.Difb200Error):
            bad()
    for bad in (lambda: ops.quantize_int8_rows([x.float()], 2), lambda: ops.quantize_int8_rows([x.cpu()], 2),
                lambda: ops.quantize_int8_rows([x, y[:2]], 2), lambda: ops.rms_norm_modulate_quant(rows, None, mods[:4], mods[:4])):
        with pytest.raises(ValueError):
            bad()
    ops.poll_status()


def test_inputs_live_as_long_as_the_call(both):
    """A list of inputs that loses them while the arguments are converted."""
    import torch
    from diffusion_compiler_b200 import ops
    x, y = (torch.randn(5, k, device="cuda").to(torch.bfloat16) for k in (512, 256))
    want = ops.quantize_int8_rows([x, y], 2, clip=0.75)

    class Clip:
        def __init__(self, parts):
            self.parts = parts

        def __float__(self):
            self.parts.clear()
            return 0.75

    def call():
        parts = [x.clone(), y.clone()]
        return ops.quantize_int8_rows(parts, 2, clip=Clip(parts))

    native, general = both(call)
    assert _same(native, want) and _same(general, want)
    ops.poll_status()


def test_operands_of_too_few_elements_are_refused():
    """Refused on the host, before a launch, natively and the general way: weights of another width, vectors that end early,
    keys of fewer tokens than the queries."""
    import torch
    from diffusion_compiler_b200 import _lib, ops
    z = lambda *s, dtype=torch.bfloat16: torch.zeros(s, dtype=dtype, device="cuda")  # noqa: E731
    x, w8, ws = z(2, 512), z(48, 512, dtype=torch.int8), z(48, dtype=torch.float32)
    x8, xs = z(2, 512, dtype=torch.int8), z(2, dtype=torch.float32)
    q, k = z(1, 70, 4, 128), z(1, 70, 2, 128)
    launches = _lib.lib().difb200_launch_count()
    for bad in (lambda **o: ops.w8a8_linear(x, w8[:, :256].contiguous(), ws, **o), lambda **o: ops.w8a8_linear(x, w8[:, :496], ws, **o),
                lambda **o: ops.w8a8_linear(x, z(48, 768, dtype=torch.int8), ws, **o), lambda **o: ops.w8a8_linear(x, w8, ws[:47], **o),
                lambda **o: ops.w8a8_linear(x, w8, ws, bias=x[0, :47], **o)):
        for kwargs in ({}, {"out": z(2, 48)}):  # with `out` the general way takes the call
            with pytest.raises(ValueError):
                bad(**kwargs)
    for bad in (lambda: ops.linear_int8_scaled(x8, w8, xs, ws, bias=x[0, :47]),
                lambda: ops.rms_norm_modulate_quant(x, x[0, :511], x, x),
                lambda: ops.layer_norm_modulate_quant(x, x[0, :511], x[0], x, x),
                lambda: ops.layer_norm_modulate_quant(x, x[0], x[0, :511], x, x),
                lambda: ops.attention(q, k[:, :69], k), lambda: ops.attention(q, k, k[:, :69]),
                lambda: ops.attention(q, k, k, key_valid=z(1, 69, dtype=torch.uint8)),
                lambda: ops.attention(q, k, k[:, :, :1], out=z(1, 70, 4, 128))):
        with pytest.raises(ValueError):
            bad()
    assert _lib.lib().difb200_launch_count() == launches
