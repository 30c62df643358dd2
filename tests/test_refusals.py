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
