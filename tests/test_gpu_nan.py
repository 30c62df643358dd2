"""NaN through the block glue on bf16 tensors: what arithmetic makes of it on this GPU (0x7fffffff) is a NaN in bf16 too, in
the fast forms and in the generic ones (odd widths), as the reference's rounding of a CPU's NaN is. Against the same
operation in torch; other elements are compared by the tests of each operator."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _glue(name, *args):
    from diffusion_compiler_b200 import _lib
    _lib.check(getattr(_lib.lib(), name)(*[C.c_void_p(a.data_ptr()) if hasattr(a, "data_ptr") else a for a in args], None))


def _tensors(rows, cols, count):
    import torch
    g = torch.Generator(device="cuda").manual_seed(cols)
    ts = [torch.randn((rows, cols), generator=g, device="cuda").to(torch.bfloat16) for _ in range(count)]
    ts[0][3, 7], ts[0][5, 1], ts[0][5, 2] = float("nan"), float("inf"), float("-inf")
    return ts


def _same_nan(got, want):
    import torch
    torch.cuda.synchronize()
    assert bool(torch.isnan(want).any()) and not bool(torch.isnan(want).all())
    assert torch.equal(torch.isnan(got), torch.isnan(want))


@pytest.mark.parametrize("cols", [3072, 256, 100])
def test_layer_norm_modulate(cols):
    import torch
    x, scale, shift = _tensors(9, cols, 3)
    w, b = torch.ones(cols, device="cuda").bfloat16(), torch.zeros(cols, device="cuda").bfloat16()
    out = torch.zeros_like(x)
    _glue("difb200_layer_norm_modulate", x, w, b, scale, shift, out, 2, 9, cols, 9, 1e-6)
    _same_nan(out, torch.nn.functional.layer_norm(x.float(), (cols,)) * (1 + scale.float()) + shift.float())


@pytest.mark.parametrize("cols", [3072, 256, 100])
def test_rms_norm_modulate(cols):
    import torch
    x, scale, shift = _tensors(9, cols, 3)
    w = torch.ones(cols, device="cuda").bfloat16()
    out = torch.zeros_like(x)
    _glue("difb200_rms_norm_modulate", x, w, scale, shift, out, 2, 9, cols, 1e-6)
    x = x.float()
    _same_nan(out, x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * (1 + scale.float()) + shift.float())


@pytest.mark.parametrize("cols", [256, 100])
def test_residual_gate(cols):
    import torch
    res, branch, gate = _tensors(9, cols, 3)
    out = torch.zeros_like(res)
    _glue("difb200_residual_gate", res, branch, gate, out, 2, 9, cols, 9)
    _same_nan(out, res.float() + gate.float() * branch.float())


@pytest.mark.parametrize("width", [128, 50])
def test_swiglu(width):
    import torch
    x, = _tensors(9, 2 * width, 1)
    out = torch.zeros((9, width), dtype=torch.bfloat16, device="cuda")
    _glue("difb200_swiglu", x, out, 2, 9, width, 2 * width, 0, 0)
    a, b = x.float()[:, :width], x.float()[:, width:]
    both = torch.isnan(a) | torch.isnan(b)
    torch.cuda.synchronize()
    assert bool(torch.isnan(out)[both].all()) and bool(both.any())


@pytest.mark.parametrize("dim", [128, 64])  # the fast form, the generic one
def test_qk_norm_rope(dim):
    import torch
    x, = _tensors(9, 3 * dim, 1)
    w = torch.ones(dim, device="cuda").bfloat16()
    angle = torch.rand((9, dim), device="cuda")
    out = torch.zeros_like(x)
    _glue("difb200_qk_norm_rope", x, w, angle.cos(), angle.sin(), out, 2, 1, 9, 3, dim, dim, dim, 9, 9, 0, 1e-5, 0)
    f = x.float().view(9, 3, dim)
    n = f * torch.rsqrt(f.square().mean(-1, keepdim=True) + 1e-5)
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    half = torch.cat([-n[..., dim // 2:], n[..., :dim // 2]], -1)
    _same_nan(out.view(9, 3, dim), n * c + half * s)


@pytest.mark.parametrize("rows,width,start,gate_first", [(1, 8, 0, 0), (5, 24, 8, 1), (300, 3072, 0, 1), (77, 8192, 16, 0), (1101, 136, 0, 0)])
def test_swiglu_rows_and_columns_of_the_fast_form(rows, width, start, gate_first):
    """The form that takes 16 bytes at a time finds rows and columns by a reciprocal of the width; the general form, which
    operands that start on two bytes take, divides. The same bits, and nothing written behind the last row."""
    import ctypes as C
    import torch
    from diffusion_compiler_b200 import _lib
    in_width = start + 2 * width + 8
    n, m = rows * in_width, rows * width
    x = torch.randn(n + 8, generator=torch.Generator().manual_seed(rows + width)).to(torch.bfloat16).cuda()
    moved = torch.cat([x[:1], x[:n]])
    fast, general = (torch.full((m + 16,), 3.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))

    def call(src, dst):
        _lib.check(_lib.lib().difb200_swiglu(C.c_void_p(src.data_ptr()), C.c_void_p(dst.data_ptr()), 2, C.c_uint64(rows), C.c_uint64(width),
                                             C.c_uint64(in_width), C.c_uint64(start), gate_first, None))
        torch.cuda.synchronize()

    call(x, fast)
    call(moved[1:], general[1:])
    assert torch.equal(fast[:m].view(torch.int16), general[1:m + 1].view(torch.int16))
    assert bool((fast[m:] == 3.0).all()) and bool((general[m + 1:] == 3.0).all()) and bool(general[0] == 3.0)
