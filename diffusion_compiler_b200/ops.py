"""Device-resident operators on torch CUDA tensors (torch is only the memory/stream plumbing;
every op below is one call into libdifb200.so).

Names and argument meaning follow the reference opcodes (``QuantizeInt8Rows``,
``LinearInt8Scaled``; reference ``include/dif/ir/ir.hpp:123-139``).
"""
from __future__ import annotations

import ctypes as C
from typing import List, Optional, Sequence, Tuple

import torch

from . import _lib
from ._calls import calls as _calls

EPILOGUE_BIAS = 1
EPILOGUE_GELU_TANH = 2


_PTR_ARRAYS = [C.c_void_p * n for n in range(9)]
_WIDTH_ARRAYS = [C.c_uint64 * n for n in range(9)]


def _done(result):
    """What the native binding made of a call: its outputs, or the status of one that failed."""
    if type(result) is int:
        _lib.check(result)
    return result


def _ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


def _call(fn, index: int, *args) -> None:
    """One call into the library on the current stream of CUDA device ``index`` (the stream is the
    entry point's last argument). The raw stream handle and the test for the current device are what
    keeps a call short: torch.cuda.current_stream() builds a Stream object (3.2 us) and the device
    context manager switches twice (1.4 us) where the device is nearly always current already."""
    if index == torch._C._cuda_getDevice():
        status = fn(*args, torch._C._cuda_getCurrentRawStream(index))
    else:
        with torch.cuda.device(index):
            status = fn(*args, torch._C._cuda_getCurrentRawStream(index))
    if status != 0:
        _lib.check(status)


def _require(t: torch.Tensor, dtype: torch.dtype, name: str) -> torch.Tensor:
    if not t.is_cuda:
        raise ValueError("%s must be a CUDA tensor (there is no CPU path)" % name)
    if t.dtype != dtype:
        raise ValueError("%s must be %s, got %s" % (name, dtype, t.dtype))
    return t.contiguous()


def _require_elements(t: Optional[torch.Tensor], count: int, name: str) -> None:
    """The kernels read ``count`` elements behind the pointer they are given."""
    if t is not None and t.numel() < count:
        raise ValueError("%s has %d elements, %d are needed" % (name, t.numel(), count))


def quantize_int8_rows(parts: Sequence[torch.Tensor], implementation: int = 2, clip: float = 1.0,
                       clip_tensor: Optional[torch.Tensor] = None, residual: bool = False,
                       out: Optional[Tuple[torch.Tensor, torch.Tensor]] = None) -> Tuple[torch.Tensor, ...]:
    """QuantizeInt8Rows: bf16 inputs concatenated on the last axis -> (codes i8, scales f32
    [, residual codes, residual scales]). ``implementation`` is the Int8RowQuantization value.
    ``out`` = (codes, scales) writes into existing contiguous buffers (e.g. a slice of an
    all-gather buffer)."""
    if out is None and clip_tensor is None and not residual:
        result = _calls().quantize_int8_rows(parts, implementation, clip)
        if result is not None:
            return _done(result)
    if isinstance(parts, torch.Tensor):
        parts = [parts]
    parts = [_require(p, torch.bfloat16, "input") for p in parts]
    lead = parts[0].shape[:-1]
    rows = 1
    for d in lead:
        rows *= d
    widths = [p.shape[-1] for p in parts]
    for p in parts:
        if p.shape[:-1] != lead:
            raise ValueError("all inputs must share their leading dimensions")
    total = sum(widths)
    dev = parts[0].device
    if out is not None:
        codes, scales = out
        if (codes.dtype != torch.int8 or scales.dtype != torch.float32 or not codes.is_contiguous()
                or not scales.is_contiguous() or codes.numel() != rows * total or scales.numel() != rows):
            raise ValueError("out buffers must be contiguous int8 [rows*width] and float32 [rows]")
    else:
        codes = torch.empty(tuple(lead) + (total,), dtype=torch.int8, device=dev)
        scales = torch.empty((rows,), dtype=torch.float32, device=dev)
    rcodes = torch.empty_like(codes) if residual else None
    rscales = torch.empty_like(scales) if residual else None
    n = len(parts)
    ptrs = (_PTR_ARRAYS[n] if n < 9 else C.c_void_p * n)(*[p.data_ptr() for p in parts])
    ws = (_WIDTH_ARRAYS[n] if n < 9 else C.c_uint64 * n)(*widths)
    if clip_tensor is not None:
        clip_tensor = _require(clip_tensor, torch.float32, "clip_tensor")
    _call(_lib.lib().difb200_quantize_int8_rows, dev.index, ptrs, ws, n, rows, int(implementation), float(clip),
          _ptr(clip_tensor), codes.data_ptr(), scales.data_ptr(), _ptr(rcodes), _ptr(rscales))
    return (codes, scales, rcodes, rscales) if residual else (codes, scales)


def rms_norm_modulate_quant(x: torch.Tensor, weight: Optional[torch.Tensor], scale: torch.Tensor,
                            shift: torch.Tensor, epsilon: float = 1e-5, implementation: int = 2, clip: float = 1.0):
    """RmsNormModulate (explicit scale / shift) + QuantizeInt8Rows in one kernel: bf16 [M, K] inputs
    -> (codes i8 [M, K], row scales f32 [M]); the normalised tensor is never written."""
    result = _calls().norm_modulate_quant(x, weight, None, scale, shift, epsilon, implementation, clip)
    if result is not None:
        return _done(result)
    x = _require(x, torch.bfloat16, "x")
    scale, shift = _require(scale, torch.bfloat16, "scale"), _require(shift, torch.bfloat16, "shift")
    if weight is not None:
        weight = _require(weight, torch.bfloat16, "weight")
    M, K = x.shape
    if scale.shape != x.shape or shift.shape != x.shape:
        raise ValueError("scale and shift must have the shape of x")
    _require_elements(weight, K, "weight")
    codes = torch.empty((M, K), dtype=torch.int8, device=x.device)
    scales = torch.empty((M,), dtype=torch.float32, device=x.device)
    _call(_lib.lib().difb200_rms_norm_modulate_quant, x.device.index, x.data_ptr(), _ptr(weight), scale.data_ptr(),
          shift.data_ptr(), M, K, epsilon, implementation, clip, codes.data_ptr(), scales.data_ptr())
    return codes, scales


def layer_norm_modulate_quant(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor, scale: torch.Tensor,
                              shift: torch.Tensor, epsilon: float = 1e-5, implementation: int = 2,
                              clip: float = 1.0):
    """LayerNormModulate + QuantizeInt8Rows in one kernel: x bf16 [M, K], weight / bias bf16 [K],
    scale / shift bf16 [M / r, K] (r rows of x share one modulation row) -> (codes i8 [M, K], row
    scales f32 [M])."""
    result = None if bias is None else _calls().norm_modulate_quant(x, weight, bias, scale, shift, epsilon, implementation, clip)
    if result is not None:
        return _done(result)
    x = _require(x, torch.bfloat16, "x")
    weight, bias = _require(weight, torch.bfloat16, "weight"), _require(bias, torch.bfloat16, "bias")
    scale, shift = _require(scale, torch.bfloat16, "scale"), _require(shift, torch.bfloat16, "shift")
    M, K = x.shape
    if scale.shape != shift.shape or scale.shape[-1] != K or M % scale.shape[0] != 0:
        raise ValueError("scale and shift must be [M / r, K]")
    _require_elements(weight, K, "weight")
    _require_elements(bias, K, "bias")
    codes = torch.empty((M, K), dtype=torch.int8, device=x.device)
    scales = torch.empty((M,), dtype=torch.float32, device=x.device)
    _call(_lib.lib().difb200_layer_norm_modulate_quant, x.device.index, x.data_ptr(), weight.data_ptr(),
          bias.data_ptr(), scale.data_ptr(), shift.data_ptr(), M, K, M // scale.shape[0], epsilon, implementation, clip,
          codes.data_ptr(), scales.data_ptr())
    return codes, scales


def weight_equalization(weight: torch.Tensor) -> torch.Tensor:
    """The offline packer's input-equalisation vector for a bf16 [N, K] weight (reference
    tools/difflux2sample.cpp:2967-2990): sqrt(column absmax / geometric mean of the column
    absmaxes), clamped to [0.5, 2], as bf16 [K]. Weights are divided by it before packing and
    activations multiplied by it at run time."""
    weight = _require(weight, torch.bfloat16, "weight")
    maxima = weight.float().abs().amax(dim=0)
    logs = torch.log(torch.clamp(maxima, min=1.0e-30)).double()
    center = torch.exp(logs.sum() / maxima.numel()).float()
    ratio = torch.sqrt(maxima / torch.clamp(center, min=1.0e-30))
    return torch.clamp(ratio, 0.5, 2.0).to(torch.bfloat16)


def quantize_weight_rows(weight: torch.Tensor, implementation: int = 2, mse_scale: bool = False,
                         input_scale: Optional[torch.Tensor] = None):
    """Weight-side packing of a bf16 [N, K] matrix: I8 codes [N, K] and per-output-channel scales
    [N] (reference tools/difflux2sample.cpp:2994-3059); ``mse_scale`` picks each row's scale by the
    offline packer's MSE search (:1225-1259); ``input_scale`` is the bf16 [K] equalisation vector
    the weights are divided by first."""
    weight = _require(weight, torch.bfloat16, "weight")
    if weight.dim() != 2:
        raise ValueError("weight must be a bf16 [N, K] matrix")
    N, K = weight.shape
    if input_scale is not None:
        input_scale = _require(input_scale, torch.bfloat16, "input_scale")
        if input_scale.numel() != K:
            raise ValueError("input_scale must have K entries")
    codes = torch.empty((N, K), dtype=torch.int8, device=weight.device)
    scales = torch.empty((N,), dtype=torch.float32, device=weight.device)
    _call(_lib.lib().difb200_quantize_weight_rows, weight.device.index, weight.data_ptr(), _ptr(input_scale), N, K,
          implementation, 1 if mse_scale else 0, codes.data_ptr(), scales.data_ptr())
    return codes, scales


def linear_int8_scaled(x8: torch.Tensor, w8: torch.Tensor, row_scales: torch.Tensor,
                       col_scales: torch.Tensor, bias: Optional[torch.Tensor] = None, gelu: bool = False,
                       want_acc: bool = False, out: Optional[torch.Tensor] = None):
    """LinearInt8Scaled (+ fused BiasAdd / tanh-Gelu): x8 [..,K] i8, w8 [N,K] i8 -> bf16 [..,N]."""
    x8 = _require(x8, torch.int8, "x8")
    w8 = _require(w8, torch.int8, "w8")
    row_scales = _require(row_scales, torch.float32, "row_scales")
    col_scales = _require(col_scales, torch.float32, "col_scales")
    K = x8.shape[-1]
    M = x8.numel() // K
    N = w8.shape[0]
    if w8.shape[1] != K or row_scales.numel() != M or col_scales.numel() != N:
        raise ValueError("shapes must flatten as [M,K] x [N,K] with row [M] and column [N] scales")
    flags = 0
    if bias is not None:
        bias = _require(bias, torch.bfloat16, "bias")
        _require_elements(bias, N, "bias")
        flags |= EPILOGUE_BIAS
    if gelu:
        flags |= EPILOGUE_GELU_TANH
    if out is None:
        out = torch.empty(tuple(x8.shape[:-1]) + (N,), dtype=torch.bfloat16, device=x8.device)
    acc = torch.empty((M, N), dtype=torch.int32, device=x8.device) if want_acc else None
    _call(_lib.lib().difb200_linear_int8_scaled, x8.device.index, x8.data_ptr(), w8.data_ptr(), row_scales.data_ptr(),
          col_scales.data_ptr(), _ptr(bias), flags, M, N, K, out.data_ptr(), _ptr(acc))
    return (out, acc) if want_acc else out


def w8a8_linear(x: torch.Tensor, w8: torch.Tensor, col_scales: torch.Tensor,
                bias: Optional[torch.Tensor] = None, gelu: bool = False, implementation: int = 2,
                clip: float = 1.0, out: Optional[torch.Tensor] = None,
                scratch: Optional[Tuple[torch.Tensor, torch.Tensor]] = None) -> torch.Tensor:
    """The W8A8 int8-convrot linear in one call: quantize x [..,K] bf16, multiply with w8 [N,K].
    ``scratch`` = (codes int8 [M,K], row scales f32 [M]) may be passed to reuse buffers."""
    if out is None and scratch is None:
        result = _calls().w8a8_linear(x, w8, col_scales, bias, gelu, implementation, clip)
        if result is not None:
            return _done(result)
    x = _require(x, torch.bfloat16, "x")
    w8 = _require(w8, torch.int8, "w8")
    col_scales = _require(col_scales, torch.float32, "col_scales")
    K = x.shape[-1]
    M = x.numel() // K
    N = w8.shape[0]
    if w8.numel() != N * K:
        raise ValueError("w8 must be [N,K] for an x of K columns")
    _require_elements(col_scales, N, "col_scales")
    flags = 0
    if bias is not None:
        bias = _require(bias, torch.bfloat16, "bias")
        _require_elements(bias, N, "bias")
        flags |= EPILOGUE_BIAS
    if gelu:
        flags |= EPILOGUE_GELU_TANH
    if scratch is None:  # one allocation: the codes, then the row scales on the next 16 bytes
        at = (M * K + 15) // 16 * 16
        scratch = x.new_empty((at + 4 * M + 1) // 2)
        codes = scratch.data_ptr()
        scales = codes + at
    else:
        codes, scales = scratch
        if codes.numel() < M * K or scales.numel() < M:
            raise ValueError("scratch buffers are too small")
        codes, scales = codes.data_ptr(), scales.data_ptr()
    if out is None:
        out = x.new_empty((M, N) if x.dim() == 2 else tuple(x.shape[:-1]) + (N,))
    _call(_lib.lib().difb200_w8a8_linear, x.device.index, x.data_ptr(), w8.data_ptr(), col_scales.data_ptr(), _ptr(bias),
          flags, int(implementation), float(clip), M, N, K, codes, scales, out.data_ptr())
    return out


def attention_int8(q8: torch.Tensor, qs: torch.Tensor, k8: torch.Tensor, ks: torch.Tensor, v: torch.Tensor,
                   key_valid: Optional[torch.Tensor] = None, scale: Optional[float] = None,
                   out: Optional[torch.Tensor] = None, scratch: Optional[torch.Tensor] = None) -> torch.Tensor:
    """INT8 attention on quantised Q/K ([B,Sq,H,128] / [B,Sk,KV,128] int8 + per token-head f32
    scales) and bf16 V [B,Sk,KV,128]; key_valid is an optional [B,Sk] uint8/bool key mask.
    Sq < Sk is the token-sharded form (local queries, all-gathered keys/values)."""
    q8 = _require(q8, torch.int8, "q8")
    k8 = _require(k8, torch.int8, "k8")
    qs = _require(qs, torch.float32, "qs")
    ks = _require(ks, torch.float32, "ks")
    v = _require(v, torch.bfloat16, "v")
    B, Sq, H, D = (int(d) for d in q8.shape)
    Sk, KV = int(k8.shape[1]), int(k8.shape[2])
    if tuple(v.shape) != (B, Sk, KV, D) or qs.numel() != B * Sq * H or ks.numel() != B * Sk * KV:
        raise ValueError("q8/qs, k8/ks and v shapes do not agree")
    if key_valid is not None:
        key_valid = key_valid.to(torch.uint8).contiguous()
        if key_valid.numel() != B * Sk:
            raise ValueError("key_valid must be [B,Sk]")
    if scale is None:
        scale = 1.0 / (D ** 0.5)
    if out is None:
        out = torch.empty((B, Sq, H, D), dtype=torch.bfloat16, device=q8.device)
    L = _lib.lib()
    nbytes = int(L.difb200_attention_int8_scratch_bytes(B, Sk, KV))
    if scratch is None or scratch.numel() < nbytes:
        scratch = torch.empty(nbytes, dtype=torch.uint8, device=q8.device)
    _call(L.difb200_attention_int8, q8.device.index, q8.data_ptr(), qs.data_ptr(), k8.data_ptr(), ks.data_ptr(),
          v.data_ptr(), _ptr(key_valid), B, Sq, Sk, H, KV, D, float(scale), scratch.data_ptr(), scratch.numel(),
          out.data_ptr())
    return out


def attention_int8_chunked(q8: torch.Tensor, qs: torch.Tensor, k8: torch.Tensor, ks: torch.Tensor, v: torch.Tensor,
                           tile_groups: Sequence[Sequence[Tuple[int, int]]], key_valid: Optional[torch.Tensor] = None,
                           scale: Optional[float] = None, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """attention_int8 as a sequence of launches, one per entry of ``tile_groups``; an entry is one or
    two (first tile, tile count) ranges of 128-key tiles. The unnormalised state of every query row
    is carried from launch to launch; the last launch writes the bf16 result. The groups must
    cover every key tile exactly once (the token-sharded block launches one group per set of
    key / value slices that have arrived)."""
    q8 = _require(q8, torch.int8, "q8")
    k8 = _require(k8, torch.int8, "k8")
    qs, ks = _require(qs, torch.float32, "qs"), _require(ks, torch.float32, "ks")
    v = _require(v, torch.bfloat16, "v")
    B, Sq, H, D = (int(d) for d in q8.shape)
    Sk, KV = int(k8.shape[1]), int(k8.shape[2])
    if key_valid is not None:
        key_valid = key_valid.to(torch.uint8).contiguous()
    if scale is None:
        scale = 1.0 / (D ** 0.5)
    if out is None:
        out = torch.empty((B, Sq, H, D), dtype=torch.bfloat16, device=q8.device)
    L = _lib.lib()
    scratch = torch.empty(int(L.difb200_attention_int8_scratch_bytes(B, Sk, KV)), dtype=torch.uint8, device=q8.device)
    state = torch.empty(int(L.difb200_attention_int8_state_bytes(B, Sq, H)), dtype=torch.uint8, device=q8.device)
    groups = [list(g) for g in tile_groups]
    for i, group in enumerate(groups):
        if not 1 <= len(group) <= 2:
            raise ValueError("a launch covers one or two tile ranges")
        flat = [int(x) for r in group for x in r] + [0, 0] * (2 - len(group))
        ranges = (C.c_uint32 * 4)(*flat)
        _call(L.difb200_attention_int8_chunk, q8.device.index, q8.data_ptr(), qs.data_ptr(), k8.data_ptr(),
              ks.data_ptr(), v.data_ptr(), _ptr(key_valid), B, Sq, Sk, H, KV, D, float(scale), scratch.data_ptr(),
              scratch.numel(), out.data_ptr(), ranges, 1 if i > 0 else 0, 1 if i + 1 < len(groups) else 0,
              state.data_ptr())
    return out


def attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, key_valid: Optional[torch.Tensor] = None,
              scale: Optional[float] = None, out: Optional[torch.Tensor] = None,
              scratch: Optional[torch.Tensor] = None) -> torch.Tensor:
    """DiffIR Attention on bf16 q [B,S,H,128], k/v [B,S,KV,128] through the INT8 lowering."""
    if out is None and scratch is None:
        result = _calls().attention(q, k, v, key_valid, scale)
        if result is not None:
            return _done(result)
    q = _require(q, torch.bfloat16, "q")
    k = _require(k, torch.bfloat16, "k")
    v = _require(v, torch.bfloat16, "v")
    B, S, H, D = q.shape
    KV = k.shape[2]
    _require_elements(k, B * S * KV * D, "k")
    _require_elements(v, B * S * KV * D, "v")
    if key_valid is not None:
        if key_valid.dtype != torch.uint8:
            key_valid = key_valid.to(torch.uint8)
        key_valid = key_valid.contiguous()
        _require_elements(key_valid, B * S, "key_valid")
    if scale is None:
        scale = 1.0 / (D ** 0.5)
    if out is None:
        out = q.new_empty((B, S, H, D))
    L = _lib.lib()
    nbytes = int(L.difb200_attention_scratch_bytes(B, S, H, KV))
    if scratch is None:
        scratch = torch.empty(nbytes, dtype=torch.uint8, device=q.device)
    _call(L.difb200_attention, q.device.index, q.data_ptr(), k.data_ptr(), v.data_ptr(), _ptr(key_valid), B, S, H, KV, D,
          float(scale), scratch.data_ptr(), scratch.numel(), out.data_ptr())
    return out


def poll_status() -> None:
    """Raises if a kernel recorded that one of its bounded device-side waits ran out."""
    _lib.check(_lib.lib().difb200_poll_status())
