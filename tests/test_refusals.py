"""Calls that the device-resident entry points refuse on the host, before anything is launched or
allocated: their status and text need no GPU (the pointers are never read)."""
import ctypes as C

import pytest

from diffusion_compiler_b200 import _lib

UNSUPPORTED = 2


@pytest.fixture(scope="module")
def lib():
    return _lib.lib()


def _refused(lib, call, text):
    before = lib.difb200_launch_count()
    assert call() == UNSUPPORTED
    assert text in lib.difb200_last_error().decode()
    assert lib.difb200_launch_count() == before


@pytest.mark.parametrize("layer", [False, True])
@pytest.mark.parametrize("offset", [2, 8])
def test_norm_prologue_refuses_an_unaligned_input(lib, layer, offset):
    """x that does not start on 16 bytes: refused before the row statistic (16-byte loads) is launched."""
    at = lambda k: C.c_void_p(0x700000000000 + 0x1000000 * k)  # noqa: E731
    x, w, b, s, h, codes, scales = C.c_void_p(at(1).value + offset), at(2), at(3), at(4), at(5), at(6), at(7)
    if layer:
        call = lambda: lib.difb200_layer_norm_modulate_quant(x, w, b, s, h, 64, 3072, 64, 1e-6, 2, 1.0, codes,  # noqa: E731
                                                             scales, None)
    else:
        call = lambda: lib.difb200_rms_norm_modulate_quant(x, w, s, h, 64, 3072, 1e-5, 2, 1.0, codes, scales,  # noqa: E731
                                                           None)
    _refused(lib, call, "16-byte aligned")


@pytest.mark.parametrize("rows", [3, 1000000])
@pytest.mark.parametrize("columns,impl", [(16640, 2), (24576, 3), (18432, 5), (20480, 4)])
def test_convrot_width_limit_does_not_depend_on_the_rows(lib, rows, columns, impl):
    """Rows of more than 16384 columns are refused whatever their number: plain, residual and packing forms."""
    at = lambda k: C.c_void_p(0x700000000000 + 0x10000000000 * k)  # noqa: E731
    parts, widths = (C.c_void_p * 1)(at(1).value), (C.c_uint64 * 1)(columns)
    for residual in (False, True):
        _refused(lib, lambda: lib.difb200_quantize_int8_rows(parts, widths, 1, rows, impl, 1.0, None, at(2), at(3),
                                                             at(4) if residual else None, at(5) if residual else None,
                                                             None), "16384")
    if impl != 4:
        _refused(lib, lambda: lib.difb200_quantize_weight_rows(at(1), None, rows, columns, impl, 1, at(2), at(3), None),
                 "16384")
        _refused(lib, lambda: lib.difb200_rms_norm_modulate_quant(at(1), at(2), at(3), at(4), rows, columns, 1e-5, impl,
                                                                  1.0, at(5), at(6), None), "16384")
