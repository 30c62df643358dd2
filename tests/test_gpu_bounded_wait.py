"""The give-up path of the kernels' bounded waits, exercised without hanging or faulting
anything: with the wait limit lowered to a few milliseconds, one tiny single-CTA GEMM is
launched whose producer announces but never issues the loads of one k-block (the library's
test aid). The consumer's wait on that stage must run out, the kernel must return through its
normal teardown (tensor memory freed), difb200_poll_status must report status 5 with the place,
and the next ordinary call must be bit-exact. The reference has no counterpart (its kernels
use unbounded barriers); its host-side error contract is DIF_BACKEND_EXECUTION_ERROR with text
(reference include/dif/backend/abi.h:22-30)."""
import numpy as np
import pytest

import oracle_bridge as ob
from helpers import bf16_normal, from_torch_bf16

pytestmark = pytest.mark.gpu


def _operands(rng, M, N, K):
    import torch
    x8 = rng.integers(-127, 128, size=(M, K), dtype=np.int8)
    w8 = rng.integers(-127, 128, size=(N, K), dtype=np.int8)
    xs = (rng.random(M, dtype=np.float32) * 1e-2 + 1e-3).astype(np.float32)
    ws = (rng.random(N, dtype=np.float32) * 1e-2 + 1e-3).astype(np.float32)
    t = lambda a: torch.from_numpy(a).cuda()
    return (x8, w8, xs, ws), (t(x8), t(w8), t(xs), t(ws))


@pytest.mark.parametrize("k_block", [0, 1])
def test_gemm_wait_runs_out_is_reported_and_recovered(k_block):
    import torch
    from diffusion_compiler_b200 import _lib, ops
    lib = _lib.lib()
    rng = np.random.default_rng(5)
    M, N, K = 128, 256, 384  # one 128x256 tile, three k-blocks, single-CTA form
    host, dev = _operands(rng, M, N, K)
    ops.linear_int8_scaled(*dev)  # a plain call first: one-time set-up is behind us
    ops.poll_status()
    lib.difb200_set_wait_limit_ns(5_000_000)  # 5 ms instead of 1.5 s
    try:
        lib.difb200_test_withhold_gemm_load(k_block)
        ops.linear_int8_scaled(*dev)      # result undefined; must return by itself
        torch.cuda.synchronize()          # no fault: the context stays usable
        with pytest.raises(_lib.Difb200Error) as info:
            ops.poll_status()
        assert info.value.status == 5 and "bounded device-side wait ran out" in str(info.value)
        assert "kernel 2" in str(info.value)
    finally:
        lib.difb200_set_wait_limit_ns(0)
    ops.poll_status()  # the words were cleared by the failing poll
    got = from_torch_bf16(ops.linear_int8_scaled(*dev))
    ops.poll_status()
    want = ob.orc().linear_int8_scaled(host[0], host[1], host[2], host[3])
    assert np.array_equal(got, want), "the call after a timed-out one is not bit-exact"


def _wide_rows(columns):
    import torch
    rows = 2 * torch.cuda.get_device_properties(0).multi_processor_count + 9  # the least that are rotated one ahead
    g = torch.Generator(device="cuda").manual_seed(columns)
    return torch.randn((rows, columns), generator=g, device="cuda").to(torch.bfloat16)


@pytest.mark.parametrize("impl,columns", [(2, 12544), (3, 16384)])
def test_row_maximum_wait_runs_out_is_reported_and_recovered(impl, columns):
    """Rows that are rotated one ahead of their maximum: the first CTA waits for one announcement more of its second row than
    its warps make. They give up (5 ms), the CTA's rows from there on stay as they were, all others have their codes, and the next call has them all."""
    import torch
    from diffusion_compiler_b200 import _lib, ops
    x = _wide_rows(columns)
    rows, sms = x.shape[0], torch.cuda.get_device_properties(0).multi_processor_count
    want = ops.quantize_int8_rows([x], impl)
    ops.poll_status()
    out = torch.full_like(want[0], -128), torch.full_like(want[1], -1.0)
    _lib.lib().difb200_test_withhold_row_maximum(5_000_000)
    ops.quantize_int8_rows([x], impl, out=out)
    with pytest.raises(_lib.Difb200Error) as info:
        ops.poll_status()
    assert info.value.status == 5 and "bounded device-side wait ran out (kernel 1" in str(info.value)
    missing = torch.arange(sms, rows, sms, device="cuda")  # the first CTA's rows, a CTA per SM
    others = torch.ones(rows, dtype=torch.bool, device="cuda")
    others[missing] = False
    assert bool((out[0][missing] == -128).all()) and bool((out[1][missing] == -1.0).all())
    assert torch.equal(out[0][others], want[0][others]) and torch.equal(out[1][others], want[1][others])
    ops.quantize_int8_rows([x], impl, out=out)
    ops.poll_status()
    assert torch.equal(out[0], want[0]) and torch.equal(out[1], want[1])


def test_static_linear_reports_a_wait_of_its_quantiser():
    """The linear that keeps its scratch in the library reports every wait of its kernels in status words of its own: to the next
    call that asks for them, once, and not to difb200_poll_status."""
    import ctypes as C

    import torch
    from diffusion_compiler_b200 import _lib, ops
    lib = _lib.lib()
    x = _wide_rows(12544)
    w8, ws = ops.quantize_int8_rows([x[:256] * 0.02], 2)
    want = ops.w8a8_linear(x, w8, ws)
    out = torch.zeros_like(want)
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731

    def call(rows, check):
        return lib.difb200_w8a8_linear_static(p(x), p(w8), p(ws), None, 0, 2, 1.0, rows, 256, 12544, p(out), check,
                                              C.c_void_p(torch.cuda.current_stream().cuda_stream))

    assert call(x.shape[0], 0) == 0 and call(0, 1) == 0
    lib.difb200_test_withhold_row_maximum(5_000_000)
    assert call(x.shape[0], 0) == 0
    torch.cuda.synchronize()
    ops.poll_status()
    assert call(0, 1) == 5 and b"bounded device-side wait ran out" in lib.difb200_last_error()
    assert call(x.shape[0], 1) == 0 and call(0, 1) == 0
    ops.poll_status()
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))


def test_exchange_flag_wait_runs_out_is_reported_and_recovered():
    """The one-CTA kernel that orders an attention launch behind the slices pushed by other ranks
    (direct exchange): with the flag set beforehand it returns at once; with a flag that nothing
    sets it gives up after its limit (10 ms here), which the status poll reports as status 5 with the
    place (kernel 5), and the device goes on working."""
    import torch
    from diffusion_compiler_b200 import _lib, ops
    lib = _lib.lib()
    assert lib.difb200_world_selftest_flags(10_000_000, 1) == 0, lib.difb200_last_error().decode()
    assert lib.difb200_world_selftest_flags(10_000_000, 0) == 5
    text = lib.difb200_last_error().decode()
    assert "bounded device-side wait ran out" in text and "kernel 5" in text
    ops.poll_status()  # cleared by the failing poll
    assert lib.difb200_world_selftest_flags(10_000_000, 1) == 0
    x = torch.arange(8, device="cuda")
    assert int(x.sum().item()) == 28
