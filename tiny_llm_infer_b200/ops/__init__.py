"""Python face of the hand-written CUDA kernels (``csrc/*.cu``) and of the library matrix
product.  Every function here works on CUDA tensors on the current stream and has no
other implementation: if the kernel library cannot be built or loaded, the first call
raises ``KernelLibraryError``.

The matrix product (``linear``, ``linear_swiglu``) has two kernels of this package for
bfloat16, chosen by the number of rows: up to 8, and up to 16 with short sums or few columns
(``skinny_pays``), the weight-streaming mma.sync product (``gemm_skinny``), from 256 on, where the tiles fill the GPU, the TMA + tcgen05 product
(``gemm_tcgen05``).  Everything else is the library's (cuBLAS through ``torch.mm``), as in the reference, which calls
``cublasHgemm`` for every projection with more than one row
(kernels/src/matmul_kernel_cuda.cu:83-91); in float32 mode it runs with the
reduced-precision matrix modes switched off, and large products (64 rows or more, ``f32_tcgen05_pays``) run on the tensor cores with
every operand in three bfloat16 parts (``gemm_f32_tcgen05``), closer to 64 bits than the library's.  So the last bits of a row depend
on how many rows share its product, in float32 too (there from 64 rows on, where the shares of K follow the rows).
"""
from __future__ import annotations

import ctypes
import functools
from typing import Optional

import torch

from ..csrc import build as _build

F32, BF16 = 0, 1
_DT = {torch.float32: F32, torch.bfloat16: BF16}

# flags of qk_norm_rope_store (csrc/qk_rope_store.cu)
QK_NORM, QK_ROPE, QK_STORE, QK_QOUT, QK_KVOUT = 1, 2, 4, 8, 16


class KernelLibraryError(RuntimeError):
    pass


class KernelError(RuntimeError):
    pass


_lib = None


def lib():
    """The loaded kernel library (built on first use)."""
    global _lib
    if _lib is not None:
        return _lib
    try:
        path = _build.library_path()
    except Exception as exc:  # BuildError and anything the toolchain throws
        raise KernelLibraryError(f"the CUDA kernel library is not available: {exc}") from exc
    try:
        handle = ctypes.CDLL(str(path))
    except OSError as exc:
        raise KernelLibraryError(f"cannot load {path}: {exc}") from exc
    _declare(handle)
    _lib = handle
    return handle


def _declare(h) -> None:
    vp, i32, f32, i64 = ctypes.c_void_p, ctypes.c_int, ctypes.c_float, ctypes.c_longlong
    h.tllm_last_error.restype = ctypes.c_char_p
    h.tllm_last_error.argtypes = []
    sigs = {
        "tllm_embedding": [vp, vp, i32, vp, i32, i32, i32, f32, vp],
        "tllm_postnorm_add_rmsnorm": [vp, vp, vp, f32, vp, i32, f32, vp, i32, vp, i32, i32, vp],
        "tllm_qkv_unit_store": [vp, i32, vp, vp, f32, i32, vp, vp, vp, i32, i32, vp, vp, i64, vp, i32, i32,
                                i32, i32, i32, i32, i32, vp, i32, i32, f32, i32, i32, vp, vp, i32, vp, f32, vp],
        "tllm_attention_biased_general": [vp, vp, vp, i64, vp, vp, vp, i32, i32, i32, i32, i32, i32, i32, i32,
                                          f32, f32, i32, i32, i32, vp, vp, vp, i32, i32, vp, i32, i32, i32, f32, f32, f32, vp, vp],
        "tllm_attention_biased_prefill": [vp, vp, vp, i64, vp, vp, i32, vp, i32, i32, i32, i32, i32, i32,
                                          f32, f32, i32, i32, i32, vp, vp, vp, i32, i32, vp, i32, i32, i32, f32, f32, f32, vp, vp],
        "tllm_attention_biased_decode": [vp, vp, vp, i64, vp, vp, vp, i32, vp, i32, i32, i32, i32, i32, i32,
                                         f32, f32, i32, i32, i32, vp, vp, vp, i32, i32, vp, i32, i32, i32, f32, f32, f32, i32, vp, vp, vp],
        "tllm_scaled_add_layernorm": [vp, vp, vp, i32, vp, i32, f32, vp, i32, vp, i32, i32, vp],
        "tllm_whole_finish": [vp, vp, i32, i32, vp, f32, vp, i32, i32, vp, i32, i32, vp],
        "tllm_linear_prepare": [vp, i32, i32, vp, i32, vp, i32, i32, f32, vp, i32, i32, i32, f32, vp, vp, vp, vp, vp, vp,
                                i32, vp],
        "tllm_embedding_norm": [vp, vp, vp, vp, i32, vp, f32, f32, vp, i32, i32, i32, i32, vp],
        "tllm_softcap": [vp, f32, i64, vp],
        "tllm_stream_add": [vp, vp, vp, i32, f32, vp, i32, i32, i32, vp],
        "tllm_activation": [vp, vp, i32, i32, i32, i32, vp, vp, i32, i32, i32, vp],
        "tllm_delta_prepare": [vp, i32, i32, vp, vp, i32, vp, i32, vp, vp, vp, vp, i64, i32, i32, i32, i32, f32, f32,
                               vp, vp, vp, vp, vp, i32, i32, i32, vp],
        "tllm_delta_scan": [vp, i32, i32, vp, vp, vp, vp, vp, vp, vp, i64, i32, i32, i32, i32, vp, i32, vp, vp, i64, f32, vp, vp],
        "tllm_chunk_scan": [vp, i32, i32, vp, vp, vp, vp, vp, vp, vp, vp, i64, i32, i32, i32, i32, vp, i32, vp],
        "tllm_erase_prepare": [vp, i32, i32, i32, vp, i32, vp, vp, f32, vp, i32, i32, i32, f32, vp, vp, vp, vp, vp, i32, vp],
        "tllm_stream_read": [vp, vp, vp, vp, vp, vp, vp, vp, vp, vp, f32, vp, i32, vp, vp, vp, i64, i32, vp, vp, i32, i32, i32, vp],
        "tllm_stream_tails": [vp, i32, vp, i32, vp, i64, i32, vp],
        "tllm_embedding_sinusoid": [vp, vp, vp, i32, vp, f32, vp, i32, i32, i32, i32, vp],
        "tllm_delta_finish": [vp, vp, i32, i32, vp, f32, vp, i32, i32, i32, i32, i32, vp, i32, vp, i32, i32, vp, i64,
                              vp, i32, i32, vp],
        "tllm_latent_norm_store": [vp, i32, i32, i32, i32, i32, i32, vp, vp, f32, vp, f32, vp, vp, vp, i32, i32,
                                   vp, i64, vp, i32, i32, i32, vp],
        "tllm_latent_query": [vp, i32, vp, i32, i32, i32, i32, i32, i32, vp, f32, vp, vp, i32, vp, i32, vp],
        "tllm_heads_gate": [vp, vp, i32, i32, i32, i32, i32, vp, vp, i32, vp],
        "tllm_moe_route": [vp, i32, i32, i32, i32, vp, vp, vp],
        "tllm_moe_route_grouped": [vp, i32, i32, i32, i32, i32, vp, i32, i32, f32, vp, vp, vp],
        "tllm_moe_plan": [vp, i32, i32, i32, i32, vp, vp, vp, vp, vp, vp, vp, vp],
        "tllm_moe_grouped": [vp, i32, vp, vp, i32, vp, i64, vp, vp, vp, vp, vp, i32, i32, i32, i32, i32, i32,
                             i32, i32, f32, f32, i32, i32, vp, vp],
        "tllm_moe_gather": [vp, vp, vp, i32, vp, i32, i32, vp],
        "tllm_moe_combine": [vp, i32, vp, vp, i32, vp, vp, i32, i32, i32, vp, vp, i32, vp, i32, vp],
        "tllm_sum_rmsnorm": [vp, vp, vp, i32, f32, vp, vp, f32, vp, i32, i32, i32, vp],
        "tllm_ssd_prepare": [vp, i32, i32, vp, vp, vp, i32, vp, vp, vp, vp, i64, i64, i32, i32, i32, i32, vp, vp, vp,
                             vp, vp, i32, vp],
        "tllm_ssd_finish": [vp, vp, vp, i32, vp, i32, i32, vp, f32, i32, vp, i32, i32, i32, i32, vp, i64, i64, vp, vp],
        "tllm_moe_tcgen05": [vp, vp, vp, i32, i32, i32, i32, i32, i32, vp, vp, vp, vp, i32, f32, f32, vp, vp],
        "tllm_add_rmsnorm": [vp, vp, vp, i32, f32, vp, i32, vp, i32, i32, vp],
        "tllm_swiglu": [vp, vp, i32, i32, i32, i32, i32, f32, f32, vp],
        "tllm_cast": [vp, i32, vp, i32, i64, vp],
        "tllm_feed_tokens": [vp, vp, vp, vp, i32, vp],
        "tllm_qk_norm_rope_store": [vp, vp, vp, i32, f32, vp, i32, vp, vp, vp, i32, vp, i32, vp,
                                    i32, i32, i32, i32, i32, i32, vp, vp],
        "tllm_rope_table": [vp, vp, i32, i32, vp, vp],
        "tllm_paged_attention_general": [vp, vp, vp, vp, vp, i32, i32, i32, i32, i32, i32, i32,
                                         i32, f32, vp, vp, vp],
        "tllm_paged_attention_f32": [vp, vp, vp, vp, i32, vp, i32, i32, i32, i32, i32, i32, f32, vp, vp],
        "tllm_sample": [vp, i32, i32, i64, vp, vp, vp, vp],
        "tllm_sample_split": [vp, i32, i32, i64, vp, vp, vp, vp, i32, vp, vp],
        "tllm_gemm_skinny": [vp, vp, vp, i32, i32, i32, i32, vp],
        "tllm_gemm_plain": [vp, i32, vp, i32, vp, i32, i32, i32, i32, vp],
        "tllm_gemm_tcgen05": [vp, vp, vp, i32, i32, i32, i32, f32, f32, vp, vp],
        "tllm_gemm_f32_tcgen05": [vp, vp, vp, i32, i32, i32, i32, vp, vp, vp],
        "tllm_gemm_skinny_swiglu": [vp, vp, vp, i32, i32, i32, i32, f32, f32, vp],
        "tllm_gemm_skinny_act": [vp, vp, vp, i32, i32, i32, i32, vp],
        "tllm_paged_attention_decode_rows": [vp, vp, vp, vp, vp, i32, vp, i32, i32, i32, i32, i32, i32, f32,
                                             i32, vp, vp, vp, i32, vp],
        "tllm_paged_attention_prefill": [vp, vp, vp, vp, i32, vp, i32, i32, i32, i32, i32, i32, f32, vp, vp],
        "tllm_paged_attention_prefill_tc": [vp, i32, vp, i32, vp, vp, i32, vp, i32, i32, i32, i32, i32, i32, f32,
                                            vp, i32, vp, vp, vp, vp],
        "tllm_attention_planes_prefill_tc": [vp, i32, vp, vp, ctypes.c_longlong, i32, vp, vp, i32, vp, i32, i32,
                                             i32, i32, i32, f32, vp, i32, vp, f32, i32, i32, vp, vp, i32, i32, vp, i32, vp,
                                             vp, vp, vp],
    }
    for name, args in sigs.items():
        fn = getattr(h, name)
        fn.argtypes = args
        fn.restype = i32
    h.tllm_delta_rule_lanes.argtypes = [i32]
    h.tllm_delta_rule_lanes.restype = i32
    h.tllm_delta_rule_state_floats.argtypes = [i32, i32, i32, i32, i32]
    h.tllm_delta_rule_state_floats.restype = i64
    h.tllm_attention_biased_fast_ok.argtypes = [i32, i32, i32, i32]
    h.tllm_attention_biased_fast_ok.restype = i32
    h.tllm_attention_maps_fast_ok.argtypes = [i32, i32, i32, i32, i32]
    h.tllm_attention_maps_fast_ok.restype = i32
    h.tllm_moe_tile_rows.argtypes = []
    h.tllm_moe_tile_rows.restype = i32
    h.tllm_paged_attention_prefill_tc_rows.argtypes = [i32, i32]
    h.tllm_paged_attention_prefill_tc_rows.restype = i32
    h.tllm_sample_nucleus_scratch_bytes.argtypes = [i32]
    h.tllm_sample_nucleus_scratch_bytes.restype = i64
    h.tllm_uniform_of.argtypes = [ctypes.c_ulonglong, i32]
    h.tllm_uniform_of.restype = f32


launches = 0      # kernels of csrc/ launched so far (graph replays are added by the runner)


def _check(code: int, what: str, kernels: int = 1) -> None:
    global launches
    launches += kernels
    if code != 0:
        raise KernelError(f"{what}: {lib().tllm_last_error().decode(errors='replace')} (code {code})")


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)
_raw_device = getattr(torch._C, "_cuda_getDevice", torch.cuda.current_device)


def _stream() -> int:
    """Handle of the current CUDA stream of the current device (the raw getter costs a fraction
    of a microsecond, the Stream object several)."""
    if _raw_stream is not None:
        return _raw_stream(_raw_device())             # (there are CUDA tensors: nothing is left to initialise)
    return torch.cuda.current_stream().cuda_stream


def _p(t: Optional[torch.Tensor]):
    return None if t is None else t.data_ptr()


def _cuda(*tensors) -> None:
    for t in tensors:
        if t is not None and (not t.is_cuda or not t.is_contiguous()):
            raise KernelError("kernels take contiguous CUDA tensors")


def _dt(t: torch.Tensor) -> int:
    try:
        return _DT[t.dtype]
    except KeyError:
        raise KernelError(f"unsupported dtype {t.dtype}") from None


# --------------------------------------------------------------------------- ops
def embedding(ids: torch.Tensor, table: torch.Tensor, out: torch.Tensor, scale: float = 1.0) -> torch.Tensor:
    """out[t] = table[ids[t]] * scale as float32; rows with a negative id become zero."""
    _cuda(ids, table, out)
    assert ids.dtype == torch.int32 and out.dtype == torch.float32
    vocab, hidden = table.shape
    _check(lib().tllm_embedding(_p(ids), _p(table), _dt(table), _p(out), ids.numel(), hidden, vocab,
                                float(scale), _stream()), "embedding")
    return out


def add_rmsnorm(h: torch.Tensor, delta: Optional[torch.Tensor], gain: torch.Tensor, eps: float,
                out: torch.Tensor, rows: Optional[torch.Tensor] = None,
                post_gain: Optional[torch.Tensor] = None, post_eps: float = 0.0) -> torch.Tensor:
    """h += delta (float32 sum, written back) and out = gain * h / sqrt(mean(h^2) + eps).
    With ``rows`` only those rows are normed, into out[0..len(rows)), and h is not written.
    With ``post_gain`` the delta is normed itself before it is added:
    h += post_gain * delta / sqrt(mean(delta^2) + post_eps), in float32 inside the same kernel."""
    _cuda(h, delta, gain, out, rows, post_gain)
    assert h.dtype == torch.float32
    if delta is not None:
        assert delta.dtype == out.dtype and delta.shape == h.shape
    n_out = out.shape[0] if rows is None else rows.numel()
    if post_gain is not None:
        assert delta is not None and post_gain.dtype == gain.dtype
        _check(lib().tllm_postnorm_add_rmsnorm(_p(h), _p(delta), _p(post_gain), float(post_eps), _p(gain), _dt(gain),
                                               float(eps), _p(out), _dt(out), _p(rows), n_out, h.shape[-1], _stream()),
               "postnorm_add_rmsnorm")
        return out
    _check(lib().tllm_add_rmsnorm(_p(h), _p(delta), _p(gain), _dt(gain), float(eps), _p(out), _dt(out),
                                  _p(rows), n_out, h.shape[-1], _stream()), "add_rmsnorm")
    return out


def scaled_add_layernorm(h: torch.Tensor, deltas, scales, gain: torch.Tensor, eps: float, out: torch.Tensor,
                         rows: Optional[torch.Tensor] = None) -> torch.Tensor:
    """h += sum_i scales[i] * deltas[i] (float32, written back; ``scales[i]`` a float32 vector of the row's width,
    ``deltas[i]`` [T, width] in the storage type; at most four), then out = gain * (h - mean) / sqrt(mean of the
    squared deviations + eps).  With ``rows`` only those rows are normed, into out[0..len(rows)), and h is not
    written."""
    _cuda(h, gain, out, rows, *deltas, *scales)
    assert h.dtype == torch.float32 and len(deltas) == len(scales) <= 4
    for d, s in zip(deltas, scales):
        assert d.dtype == out.dtype and d.shape == h.shape and s.dtype == torch.float32 and s.numel() == h.shape[1]
    n = len(deltas)
    dp = (ctypes.c_void_p * 4)(*[d.data_ptr() for d in deltas])
    sp = (ctypes.c_void_p * 4)(*[s.data_ptr() for s in scales])
    n_out = out.shape[0] if rows is None else rows.numel()
    _check(lib().tllm_scaled_add_layernorm(_p(h), ctypes.cast(dp, ctypes.c_void_p), ctypes.cast(sp, ctypes.c_void_p), n,
                                           _p(gain), _dt(gain), float(eps), _p(out), _dt(out), _p(rows), n_out,
                                           h.shape[-1], _stream()), "scaled_add_layernorm")
    return out


def sum_rmsnorm(h: torch.Tensor, deltas, coefs, alpha: float, gain: torch.Tensor, eps: float, out: torch.Tensor,
                bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """h <- gain * v / sqrt(mean(v^2) + eps) with v = alpha * h + sum_i coefs[i] * deltas[i] (+ bias), for every row:
    the norm of a weighted sum becomes the stream itself (float32); ``out`` receives the new stream in the storage
    type.  ``deltas[i]`` [T, width] in the storage type with one float each (at most four), ``gain`` and ``bias``
    float32 vectors."""
    _cuda(h, gain, out, bias, *deltas)
    assert h.dtype == torch.float32 and gain.dtype == torch.float32 and len(deltas) == len(coefs) <= 4
    assert out.shape == h.shape and gain.numel() == h.shape[1] and (bias is None or (bias.dtype == torch.float32 and bias.numel() == h.shape[1]))
    for d in deltas:
        assert d.dtype == out.dtype and d.shape == h.shape
    n = len(deltas)
    dp = (ctypes.c_void_p * 4)(*[d.data_ptr() for d in deltas])
    cp = (ctypes.c_float * 4)(*[float(c) for c in coefs])
    _check(lib().tllm_sum_rmsnorm(_p(h), ctypes.cast(dp, ctypes.c_void_p), ctypes.cast(cp, ctypes.c_void_p), n, float(alpha),
                                  _p(bias), _p(gain), float(eps), _p(out), _dt(out), h.shape[0], h.shape[1], _stream()),
           "sum_rmsnorm")
    return out


def interleave_gate_up(gate: torch.Tensor, up: torch.Tensor) -> torch.Tensor:
    """[2 I, K] with the rows of ``gate`` and ``up`` ([I, K], I a multiple of 8) interleaved by
    eight: eight gate rows, the eight up rows that belong to them, and so on.  A block of the
    weight-streaming product and a tile of the tcgen05 product then read neighbouring rows and
    find a gate and its up in one accumulator, so SwiGLU fits their epilogues."""
    inter, k = gate.shape
    assert up.shape == gate.shape and inter % 8 == 0
    return torch.stack([gate.reshape(inter // 8, 8, k), up.reshape(inter // 8, 8, k)], dim=1).reshape(2 * inter, k)


ACTIVATIONS = {"silu": 0, "gelu_tanh": 1, "clamped_swish": 4, "relu": 6}      # of gated units: codes of csrc/common.cuh (GateAct)
NO_CONSTS = (0.0, 0.0)       # ``consts``: (limit, slope) of ``clamped_swish``, g sigmoid(slope g) (u + 1) with g = min(gate,
                             # limit) and u = up held within -limit .. limit; the other activations have none


def _consts(act: str, consts):
    limit, slope = NO_CONSTS if consts is None else consts
    if act == "clamped_swish" and not limit > 0.0:
        raise KernelError("clamped_swish needs its constants (limit, slope)")
    return float(limit), float(slope)


def swiglu(gate_up: torch.Tensor, out: torch.Tensor, interleaved: bool = False, act: str = "silu",
           consts=None) -> torch.Tensor:
    """out[t, i] = act(gate) * up with gate = gate_up[t, i], up = gate_up[t, I + i], or, for columns
    interleaved by eight, gate = gate_up[t, 16 (i // 8) + i % 8] and up eight columns further.
    ``act``: ``silu``, ``gelu_tanh``, ``relu`` or ``clamped_swish`` (with its ``consts``)."""
    _cuda(gate_up, out)
    tokens, two_i = gate_up.shape
    assert out.shape == (tokens, two_i // 2) and out.dtype == gate_up.dtype
    _check(lib().tllm_swiglu(_p(gate_up), _p(out), _dt(out), tokens, two_i // 2, int(interleaved),
                             ACTIVATIONS[act], *_consts(act, consts), _stream()), "swiglu")
    return out


def cast(src: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    _cuda(src)
    if src.dtype == dtype:
        return src
    dst = torch.empty_like(src, dtype=dtype)
    _check(lib().tllm_cast(_p(src), _dt(src), _p(dst), _dt(dst), src.numel(), _stream()), "cast")
    return dst


def feed_tokens(ids: torch.Tensor, places: torch.Tensor, rows: torch.Tensor, sampled: torch.Tensor) -> None:
    """ids[places[i]] = sampled[rows[i]] (all int32, on the device): the tokens that the step before
    is still sampling go into this step's token ids without passing through the host."""
    _cuda(ids, places, rows, sampled)
    assert ids.dtype == places.dtype == rows.dtype == sampled.dtype == torch.int32 and places.numel() == rows.numel()
    _check(lib().tllm_feed_tokens(_p(ids), _p(places), _p(rows), _p(sampled), places.numel(), _stream()), "feed_tokens")


def rope_table(positions: torch.Tensor, inv_freq: torch.Tensor) -> torch.Tensor:
    """[tokens, 2, half] float32: cosines and sines of position * inv_freq (the float32 product), made
    once per step and read by every layer's ``qk_norm_rope_store``."""
    _cuda(positions, inv_freq)
    assert positions.dtype == torch.int32 and inv_freq.dtype == torch.float32
    tokens, half = positions.numel(), inv_freq.numel()
    table = torch.empty((tokens, 2, half), dtype=torch.float32, device=positions.device)
    _check(lib().tllm_rope_table(_p(positions), _p(inv_freq), half, tokens, _p(table), _stream()), "rope_table")
    return table


def qk_norm_rope_store(qkv: torch.Tensor, q_gain, k_gain, eps: float, inv_freq, rotary_dim: int,
                       positions: torch.Tensor, token_slot: torch.Tensor, block_table, cache,
                       page_size: int, q_out, q_heads: int, kv_heads: int, head_dim: int,
                       flags: int, table: Optional[torch.Tensor] = None) -> None:
    """One pass over the fused q|k|v rows [T, (q_heads + 2 kv_heads) * head_dim]: per-head
    RMSNorm of q and k (QK_NORM), rotate-half rotation (QK_ROPE), write of k and v into
    their page (QK_STORE), write of q to ``q_out`` (QK_QOUT), write of the processed k back
    in place (QK_KVOUT).  Rows whose token_slot is negative are skipped.  ``table``: the step's
    ``rope_table`` for these positions and frequencies (same values, no sincosf per layer)."""
    _cuda(qkv, q_gain, k_gain, inv_freq, positions, token_slot, block_table, cache, q_out, table)
    if table is not None:
        assert table.dtype == torch.float32 and tuple(table.shape) == (qkv.shape[0], 2, rotary_dim // 2)
    tokens = qkv.shape[0]
    assert qkv.shape[1] == (q_heads + 2 * kv_heads) * head_dim
    gain_dt = _dt(q_gain) if q_gain is not None else F32
    max_pages = block_table.shape[1] if block_table is not None else 0
    if cache is not None:
        assert cache.dtype == qkv.dtype and tuple(cache.shape[1:]) == (2, kv_heads, page_size, head_dim)
    _check(lib().tllm_qk_norm_rope_store(
        _p(qkv), _p(q_gain), _p(k_gain), gain_dt, float(eps), _p(inv_freq), rotary_dim,
        _p(positions), _p(token_slot), _p(block_table), max_pages, _p(cache), page_size, _p(q_out),
        _dt(qkv), tokens, q_heads, kv_heads, head_dim, flags, _p(table), _stream()), "qk_norm_rope_store")


_workspaces = {}


WORKSPACE_FLOATS = 16 << 20


def workspace(device, floats: int) -> torch.Tensor:
    """Float32 scratch for one call.  Up to WORKSPACE_FLOATS it is one buffer per device
    that lives as long as the process and never moves (captured CUDA graphs keep its
    address); a larger request gets a tensor of its own."""
    if floats > WORKSPACE_FLOATS:
        return torch.empty(floats, dtype=torch.float32, device=device)
    key = str(device)
    buf = _workspaces.get(key)
    if buf is None:
        buf = torch.empty(WORKSPACE_FLOATS, dtype=torch.float32, device=device)
        _workspaces[key] = buf
    return buf


SM_COUNT = 148


def decode_splits(rows: int, kv_heads: int, max_context: int) -> int:
    """How many blocks share the keys of one (row, key/value head): enough blocks for
    about four per multiprocessor, each with at least 128 keys."""
    by_length = -(-max_context // 1024)                       # about a thousand keys per block
    by_count = -(-128 // max(rows * kv_heads, 1))             # but at least 128 blocks in all
    return max(1, min(max(by_length, by_count), -(-max_context // 128), 64))


def fast_attention_ok(dtype, page_size: int, q_heads: int, kv_heads: int, head_dim: int) -> bool:
    return (dtype == torch.bfloat16 and head_dim in (64, 128) and page_size % 16 == 0
            and q_heads % kv_heads == 0 and q_heads // kv_heads <= 16)


def paged_attention_decode(q, cache, positions, token_slot, rows, n_rows, block_table, page_size,
                           q_heads, kv_heads, head_dim, window, scale, out, max_context, splits=None, shared=False):
    """Attention of one-token rows (``rows``: their indices, None for all; ``shared``: several may belong to one
    request), keys split over
    ``splits`` blocks per (row, key/value head); the splits' partial results go through scratch
    in global memory to a second small kernel that combines them in the order of the splits."""
    _cuda(q, cache, positions, token_slot, rows, block_table, out)
    if splits is None:
        splits = decode_splits(n_rows, kv_heads, max_context)
    part_o = part_ml = None
    if splits > 1:
        n = n_rows * q_heads * splits
        ws = workspace(q.device, n * (head_dim + 2))
        part_o, part_ml = ws[:n * head_dim], ws[n * head_dim:n * (head_dim + 2)]
    _check(lib().tllm_paged_attention_decode_rows(
        _p(q), _p(cache), _p(positions), _p(token_slot), _p(rows), n_rows, _p(block_table),
        block_table.shape[1], page_size, q_heads, kv_heads, head_dim, int(window or 0), float(scale),
        splits, _p(part_o), _p(part_ml), _p(out), int(shared), _stream()), "paged_attention_decode",
        kernels=2 if splits > 1 else 1)
    return out


def paged_attention_prefill(q, cache, seg_info, tiles, n_tiles, block_table, page_size, q_heads,
                            kv_heads, head_dim, window, scale, out):
    """Attention of the segments' query blocks listed in ``tiles`` ([n, 2] = segment, offset)."""
    _cuda(q, cache, seg_info, tiles, block_table, out)
    _check(lib().tllm_paged_attention_prefill(
        _p(q), _p(cache), _p(seg_info), _p(tiles), n_tiles, _p(block_table), block_table.shape[1],
        page_size, q_heads, kv_heads, head_dim, int(window or 0), float(scale), _p(out), _stream()),
        "paged_attention_prefill")
    return out


PREFILL_TCGEN05 = True     # head width 128 takes the tcgen05 kernel; False keeps the mma.sync one


def prefill_tcgen05_block_rows(q_heads: int, kv_heads: int) -> int:
    """Query rows per entry of the tile list that ``paged_attention_prefill_tcgen05`` wants: 128
    where two heads of one key/value head share a thread block (an even group), else 256."""
    return int(lib().tllm_paged_attention_prefill_tc_rows(q_heads, kv_heads))


def prefill_splits(blocks: int, max_context: int) -> int:
    """Runs of keys per block of query rows in ``paged_attention_prefill_tcgen05``: 1, 2, 4 or 8.
    A step with few query rows (a short portion of a prompt) has few blocks, each walking all keys
    of its request; cutting the keys fills the GPU (148 SMs, one block each), as long as a run
    keeps eight tiles of 64 keys, below which a block's start and end outweigh its work."""
    fit = min(SM_COUNT // max(blocks, 1), -(-max_context // 64) // 8)
    splits = 1
    while splits * 2 <= min(fit, 8):
        splits *= 2
    return splits



def paged_attention_prefill_tcgen05(q, cache, seg_info, tiles, n_tiles, block_table, page_size, q_heads,
                                    kv_heads, head_dim, window, scale, out, splits=1):
    """As ``paged_attention_prefill`` on tcgen05 tensor cores with TMA loads: bfloat16, head width
    128, ``tiles`` at multiples of ``prefill_tcgen05_block_rows`` rows.  With ``splits`` > 1 every
    block's keys are shared by that many blocks and a second kernel combines what they leave.
    The kernel's waits are bounded; what they report is read by ``check_error_word``."""
    _cuda(q, cache, seg_info, tiles, block_table, out)
    assert q.dtype == torch.bfloat16 and cache.dtype == torch.bfloat16 and out.dtype == torch.bfloat16
    assert q.shape[1] == q_heads * head_dim and tuple(out.shape) == tuple(q.shape)
    global tcgen05_calls
    tcgen05_calls += 1
    part_o = part_ml = None
    if splits > 1:
        n = q.shape[0] * q_heads * splits
        ws = workspace(q.device, n * (head_dim + 2))
        part_o, part_ml = ws[:n * head_dim], ws[n * head_dim:n * (head_dim + 2)]
    _check(lib().tllm_paged_attention_prefill_tc(
        _p(q), q.shape[0], _p(cache), cache.shape[0], _p(seg_info), _p(tiles), n_tiles, _p(block_table),
        block_table.shape[1], page_size, q_heads, kv_heads, head_dim, int(window or 0), float(scale),
        _p(out), splits, _p(part_o), _p(part_ml), _p(error_word(q.device)), _stream()), "paged_attention_prefill_tc",
        kernels=2 if splits > 1 else 1)
    return out


def paged_attention(q: torch.Tensor, cache: torch.Tensor, positions, token_slot, block_table,
                    page_size: int, q_heads: int, kv_heads: int, head_dim: int,
                    window: Optional[int], scale: float, out: torch.Tensor, ctx=None) -> torch.Tensor:
    """Attention of every row of ``q`` over the keys of its own request in the paged cache:
    positions max(0, pos - window + 1) .. pos.  With the step's context and a shape the
    tensor-core kernels take (bfloat16, head width 64 or 128, pages of a multiple of 16),
    one-token rows go to the split-key decode kernel and longer segments to the tiled
    prefill kernel; in float32 at those widths longer segments go to tiles on the float32 pipe;
    everything else runs the general kernel."""
    _cuda(q, cache, positions, token_slot, block_table, out)
    tokens = q.shape[0]
    assert tuple(cache.shape[1:]) == (2, kv_heads, page_size, head_dim) and cache.dtype == q.dtype
    if ctx is not None and ctx.pf_tiles is not None and ctx.tokens == tokens \
            and fast_attention_ok(q.dtype, page_size, q_heads, kv_heads, head_dim):
        if ctx.n_dec:
            paged_attention_decode(q, cache, positions, token_slot, ctx.dec_rows, ctx.n_dec, block_table,
                                   page_size, q_heads, kv_heads, head_dim, window, scale, out,
                                   ctx.max_context, shared=getattr(ctx, "shared_rows", False))
        if ctx.n_tiles:
            if PREFILL_TCGEN05 and head_dim == 128 and getattr(ctx, "n_tiles256", 0):
                pairs = prefill_tcgen05_block_rows(q_heads, kv_heads) == 128
                blocks = ctx.n_tiles128 if pairs else ctx.n_tiles256
                keys = ctx.max_context if not window else min(ctx.max_context, window + 256)
                splits = prefill_splits(blocks * (q_heads // 2 if pairs else q_heads), keys)
                paged_attention_prefill_tcgen05(q, cache, ctx.seg_info, ctx.pf_tiles, blocks,
                                                block_table, page_size, q_heads, kv_heads, head_dim,
                                                window, scale, out, splits)
            else:
                paged_attention_prefill(q, cache, ctx.seg_info, ctx.pf_tiles, ctx.n_tiles, block_table,
                                        page_size, q_heads, kv_heads, head_dim, window, scale, out)
        return out
    rows, n = None, tokens
    if ctx is not None and ctx.pf_tiles is not None and ctx.tokens == tokens and 0 < ctx.n_tiles <= 65535 \
            and q.dtype == torch.float32 and head_dim in (64, 128) \
            and (q.data_ptr() | cache.data_ptr() | out.data_ptr()) % 16 == 0:
        # float32 portions: tiles of 64 rows; what is left are the one-token rows
        _check(lib().tllm_paged_attention_f32(
            _p(q), _p(cache), _p(ctx.seg_info), _p(ctx.pf_tiles), ctx.n_tiles, _p(block_table), block_table.shape[1], page_size,
            q_heads, kv_heads, head_dim, int(window or 0), float(scale), _p(out), _stream()), "paged_attention_f32")
        rows, n = ctx.dec_rows, ctx.n_dec
    if n:
        _check(lib().tllm_paged_attention_general(
            _p(q), _p(cache), _p(positions), _p(token_slot), _p(block_table), block_table.shape[1],
            page_size, _dt(q), n, q_heads, kv_heads, head_dim, int(window or 0), float(scale), _p(rows),
            _p(out), _stream()), "paged_attention")
    return out


SAMPLE_BLOCKS = 1024     # blocks over all rows beyond which a row's vocabulary is cut less finely


def sample(logits: torch.Tensor, params: torch.Tensor, seeds: torch.Tensor,
           out: torch.Tensor, any_nucleus: Optional[bool] = None) -> torch.Tensor:
    """Token per row of float32 ``logits`` [S, V]: params[s] = (temperature, top_p), seeds[s]
    an int64 key.  temperature <= 1e-6 is argmax (lowest id on ties).  ``any_nucleus`` says
    whether some row samples with top_p < 1 (None: not known, assume so)."""
    _cuda(logits, params, seeds, out)
    assert logits.dtype == torch.float32 and params.dtype == torch.float32
    assert seeds.dtype == torch.int64 and out.dtype == torch.int32
    rows, vocab = logits.shape
    if vocab >= 4096 and rows > 0:
        # a row's vocabulary shared by several blocks; rows with top-p take four more passes
        blocks = min(64, -(-vocab // 2048), max(8, SAMPLE_BLOCKS // rows))
        partial = torch.empty((rows, blocks, 2), dtype=torch.float32, device=logits.device)
        scratch = None
        if any_nucleus is None or any_nucleus:
            size = lib().tllm_sample_nucleus_scratch_bytes(rows)
            scratch = torch.empty(size // 8, dtype=torch.int64, device=logits.device)
        _check(lib().tllm_sample_split(_p(logits), rows, vocab, logits.stride(0), _p(params), _p(seeds),
                                       _p(out), _p(partial), blocks, _p(scratch), _stream()), "sample",
               kernels=2 if scratch is None else 7)
        return out
    _check(lib().tllm_sample(_p(logits), rows, vocab, logits.stride(0), _p(params), _p(seeds),
                             _p(out), _stream()), "sample")
    return out


def uniform_of(seed: int, token: int) -> float:
    """The uniform number the sampler draws for (seed, token); for host-side checks."""
    return float(lib().tllm_uniform_of(seed & 0xFFFFFFFFFFFFFFFF, token))


SKINNY_MAX_ROWS = 8       # up to this many rows the weight-streaming product beats the library
SKINNY_WIDE_ROWS = 16     # and up to this many with few blocks or short sums: see skinny_pays


def skinny_pays(x: torch.Tensor, weight: torch.Tensor, gated: bool = False) -> bool:
    """Whether a bfloat16 product goes to the weight-streaming kernel, which gives 16 weight rows to a block.
    Beyond eight rows of x a block holds two row tiles and its registers leave two blocks per SM, so it is ahead of the library
    only where a block's sums are short or half the SMs are enough for all blocks.  16 rows, weights from HBM, this kernel and the
    library's, us: columns x K 4096 x 1024 3.8 and 4.3, 4736 x 1536 4.9 and 5.2, 1024 x 2048 4.9 and 6.4, 1024 x 3072 6.1 and 8.3,
    1184 x 4096 6.8 and 7.5; but 2560 x 2048 5.4 and 5.2, 4096 x 12288 21.6 and 20.9, 2560 x 9728 17.2 and 14.7, 1184 x 8192 12.7
    and 12.2.  A gated product also saves the activation's kernel: two blocks per SM and K up to 8192 pay (inter x K 2368 x 4096 10.0
    and 12.3, 2048 x 8192 16.9 and 17.3), three only with short sums (3072 x 1024 6.3 and 7.7, 3552 x 1536 8.3 and 9.0, 2560 x 1664
    9.1 and 8.6, 3552 x 2560 12.5 and 11.4)."""
    rows, k = x.shape
    if not 0 < rows <= SKINNY_WIDE_ROWS or k % 8 or not x.is_contiguous() or not weight.is_contiguous():
        return False
    if rows <= SKINNY_MAX_ROWS:
        return True
    blocks = -(-weight.shape[0] // 16)
    if gated:
        fast = blocks <= 3 * SM_COUNT and k <= 1536 or blocks <= 2 * SM_COUNT and k <= 8192
    else:
        fast = blocks <= 2 * SM_COUNT and k <= 1536 or blocks <= SM_COUNT // 2 and k <= 4096
    return fast and (x.data_ptr() | weight.data_ptr()) % 16 == 0


def gemm_skinny(x: torch.Tensor, weight: torch.Tensor, out_dtype: torch.dtype) -> torch.Tensor:
    """y = x . weight^T for at most 32 bfloat16 rows: every weight is read once, straight from
    HBM into tensor-core fragments (csrc/gemm_skinny.cu)."""
    _cuda(x, weight)
    rows, k = x.shape
    n = weight.shape[0]
    assert weight.shape[1] == k and x.dtype == weight.dtype == torch.bfloat16
    y = torch.empty((rows, n), dtype=out_dtype, device=x.device)
    _check(lib().tllm_gemm_skinny(_p(x), _p(weight), _p(y), _DT[out_dtype], rows, n, k, _stream()),
           "gemm_skinny")
    return y


def gemm_plain(x: torch.Tensor, weight: torch.Tensor, out_dtype: torch.dtype = torch.float32) -> torch.Tensor:
    """y = x . weight^T by the plain kernel (csrc/gemm_plain.cu): one thread per output, the sum over
    k in order in float32, any sizes, bfloat16 or float32 operands.  Slow; it is what the fast products
    are checked against at sizes too large for the host."""
    _cuda(x, weight)
    rows, k = x.shape
    n = weight.shape[0]
    assert weight.shape[1] == k
    y = torch.empty((rows, n), dtype=out_dtype, device=x.device)
    _check(lib().tllm_gemm_plain(_p(x), _dt(x), _p(weight), _dt(weight), _p(y), _dt(y), rows, n, k, _stream()), "gemm_plain")
    return y


_error_words = {}


def error_word(device) -> torch.Tensor:
    """Device int32 that kernels with bounded waits (the tcgen05 product) set to a non-zero
    code when a wait ran out.  ``check_error_word`` reads it (a synchronisation)."""
    key = str(device)
    if key == "cuda":                        # without an index: the word of the current device, as its tensors name it
        key = f"cuda:{torch.cuda.current_device()}"
    if key not in _error_words:
        _error_words[key] = torch.zeros(1, dtype=torch.int32, device=device)
    return _error_words[key]


def check_error_word(device) -> None:
    code = int(error_word(device).item())
    if code:
        error_word(device).zero_()
        raise KernelError(f"a bounded wait ran out inside a kernel (code {code}); its result is invalid")


tcgen05_calls = 0          # products issued on the tcgen05 path (their bounded waits report to error_word)


def tcgen05_pays(rows: int, out_cols: int, k: int, dtype, col_tile: int = 256) -> bool:
    """Whether the hand-written tcgen05 product is used instead of the library's: bfloat16, at
    least 256 rows, and a tile count that fills the SMs' last round to 85% (blocks of 256 rows;
    with fewer tiles per round the library's 2-CTA kernels are faster)."""
    if dtype != torch.bfloat16 or rows < 256 or k % 8 or out_cols % 8:
        return False
    tiles = -(-rows // 256) * -(-out_cols // col_tile)
    rounds = -(-tiles // SM_COUNT)
    return tiles / (rounds * SM_COUNT) >= 0.85


def gemm_tcgen05(x: torch.Tensor, weight: torch.Tensor, swiglu: bool = False, short_tiles: bool = False,
                 interleaved: bool = False, act: str = "silu", unary: bool = False, consts=None) -> torch.Tensor:
    """y = x . weight^T on tcgen05 tensor cores fed by TMA (csrc/gemm_tcgen05.cu), bfloat16 in
    and out, float32 accumulation in tensor memory.  With ``swiglu`` the weight is [gate; up]
    (or, ``interleaved``, gate and up rows interleaved by eight) and the result is
    silu(x . gate^T) * (x . up^T), [rows, weight rows / 2].  ``short_tiles`` keeps blocks of 128
    rows even when there are more (for measurements)."""
    _cuda(x, weight)
    rows, k = x.shape
    n = weight.shape[0]
    assert weight.shape[1] == k and x.dtype == weight.dtype == torch.bfloat16
    y = torch.empty((rows, n // 2 if swiglu else n), dtype=torch.bfloat16, device=x.device)
    if rows == 0:
        return y
    global tcgen05_calls
    tcgen05_calls += 1
    _check(lib().tllm_gemm_tcgen05(_p(x), _p(weight), _p(y), rows, n, k, int(swiglu) | (2 if short_tiles else 0) | (4 if interleaved else 0) | (16 if unary else 0)
                                   | ((ELEMENTWISE_ACTIVATIONS[act] if unary else ACTIVATIONS[act]) << 8 if (swiglu or unary) else 0),
                                   *(_consts(act, consts) if swiglu else NO_CONSTS),
                                   _p(error_word(x.device)), _stream()), "gemm_tcgen05")
    return y


def f32_splits(rows: int, out_cols: int, k: int) -> int:
    """Shares of K in ``gemm_f32_tcgen05``: tiles of 128 x 128 go to one block per SM, so K is cut where few tiles would leave
    SMs idle, as far as the saved rounds outweigh the second kernel that adds the shares (a slab of 64 takes 1.65 us, the
    shares 3 us and their bytes at 5 TB/s)."""
    tiles, slabs = -(-rows // 128) * -(-out_cols // 128), -(-k // 64)

    def us(s):
        each = -(-slabs // s)
        used = -(-slabs // each)
        return -(-tiles * used // SM_COUNT) * each * 1.65 + (0.0 if used == 1 else 3.0 + (2 * used + 1) * rows * out_cols * 4 / 5e6)
    return min(range(1, min(slabs, 16) + 1), key=us)


def f32_tcgen05_pays(x: torch.Tensor, weight: torch.Tensor) -> bool:
    """Whether a float32 product runs on the tensor cores rather than in the library: enough work for their start, and operands in
    16-byte pieces.  The library's kernel and this one, rows x columns x K: 64 x 1024 x 2048 37 and 28 us, 64 x 4096 x 4096 78 and
    38, 128 x 4096 x 1024 32 and 30 (64 rows 23 and 28), 595 x 4096 x 1024 123 and 62, 595 x 1024 x 2048 87 and 33,
    2048 x 24576 x 4096 6955 and 2223; 595 x 96 x 64 11 and 12.  (With fewer rows it is ahead only from K = 3072 on.)  At the lines,
    weights from HBM and the kernels back to back: 64 x 8192 x 1024 33 and 23, 512 x 1024 x 1024 30 and 17, 64 x 2048 x 1028 26 and 12,
    128 x 832 x 1280 30 and 14, 64 x 1408 x 1536 37 and 14.  (Back to back, weights in L2, it is ahead below the
    lines too: 64 x 1024 x 1024 19 and 10.)"""
    rows, k = x.shape
    n = weight.shape[0]
    return (rows >= 64 and rows * n * k >= (1 << 29 if k <= 1024 else 1 << 27) and k % 4 == 0 and n % 4 == 0
            and x.is_contiguous() and weight.is_contiguous() and (x.data_ptr() | weight.data_ptr()) % 16 == 0
            and not (x.requires_grad or weight.requires_grad))


def gemm_f32_tcgen05(x: torch.Tensor, weight: torch.Tensor, splits: Optional[int] = None) -> torch.Tensor:
    """y = x . weight^T in float32 on tcgen05 tensor cores, both operands as sums of three bfloat16 parts
    (csrc/gemm_f32.cu)."""
    _cuda(x, weight)
    rows, k = x.shape
    n = weight.shape[0]
    assert weight.shape[1] == k and x.dtype == weight.dtype == torch.float32
    y = torch.empty((rows, n), dtype=torch.float32, device=x.device)
    if rows == 0:
        return y
    splits = f32_splits(rows, n, k) if splits is None else splits
    shares = torch.empty(splits * rows * n, dtype=torch.float32, device=x.device) if splits > 1 else None
    global tcgen05_calls
    tcgen05_calls += 1
    _check(lib().tllm_gemm_f32_tcgen05(_p(x), _p(weight), _p(y), rows, n, k, splits, _p(shares), _p(error_word(x.device)), _stream()),
           "gemm_f32_tcgen05", kernels=2 if splits > 1 else 1)
    return y


def linear(x: torch.Tensor, weight: torch.Tensor, out_dtype: Optional[torch.dtype] = None,
           bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """y[T, N] = x[T, K] . weight[N, K]^T with float32 accumulation.  A weight kept in
    float32 is multiplied in float32 whatever the activations are stored in.  ``bias`` [N] (the weight's type) is
    added in the library product's epilogue."""
    if not x.is_cuda:
        raise KernelError("linear takes CUDA tensors")
    want = out_dtype or x.dtype
    if bias is not None:
        if weight.dtype == torch.float32 and (torch.backends.cuda.matmul.allow_tf32 or torch.get_float32_matmul_precision() != "highest"):
            raise KernelError("float32 products need the reduced-precision matrix modes off")
        y = torch.addmm(bias.to(weight.dtype), cast(x, weight.dtype), weight.t())
        return y if want == y.dtype else cast(y, want)
    if weight.dtype == torch.float32:
        if torch.backends.cuda.matmul.allow_tf32 or torch.get_float32_matmul_precision() != "highest":
            raise KernelError("float32 products need the reduced-precision matrix modes off")
        x = cast(x, torch.float32)
        y = gemm_f32_tcgen05(x, weight) if f32_tcgen05_pays(x, weight) else torch.mm(x, weight.t())
        return y if want == torch.float32 else cast(y, want)
    if x.dtype != weight.dtype:
        x = cast(x, weight.dtype)
    rows, k = x.shape
    if weight.dtype == torch.bfloat16 and want in _DT and skinny_pays(x, weight):
        return gemm_skinny(x, weight, want)
    if want == torch.bfloat16 and tcgen05_pays(rows, weight.shape[0], k, weight.dtype) \
            and x.is_contiguous() and weight.is_contiguous():
        return gemm_tcgen05(x, weight)
    if want == weight.dtype:
        return torch.mm(x, weight.t())
    return torch.mm(x, weight.t(), out_dtype=want)


def gemm_skinny_swiglu(x: torch.Tensor, w_gate_up: torch.Tensor, act: str = "silu", consts=None) -> torch.Tensor:
    """silu(x . Wg^T) * (x . Wu^T) for at most 16 bfloat16 rows as one weight-streaming kernel;
    ``w_gate_up`` holds the rows of Wg and Wu interleaved by eight (``interleave_gate_up``)."""
    _cuda(x, w_gate_up)
    rows, k = x.shape
    inter = w_gate_up.shape[0] // 2
    out = torch.empty((rows, inter), dtype=torch.bfloat16, device=x.device)
    _check(lib().tllm_gemm_skinny_swiglu(_p(x), _p(w_gate_up), _p(out), rows, inter, k, ACTIVATIONS[act],
                                         *_consts(act, consts), _stream()), "gemm_skinny_swiglu")
    return out


def linear_swiglu(x: torch.Tensor, w_gate_up: torch.Tensor, out_dtype: torch.dtype,
                  interleaved: bool = False, act: str = "silu", consts=None) -> torch.Tensor:
    """silu(x . Wg^T) * (x . Wu^T) for w_gate_up = [Wg; Wu], or with the rows of Wg and Wu
    interleaved by eight (``interleave_gate_up``).  With enough bfloat16 rows the product and the
    activation are one tcgen05 kernel, with few rows and interleaved weights one weight-streaming
    kernel; otherwise the product is followed by the SwiGLU kernel."""
    rows, k = x.shape
    inter = w_gate_up.shape[0] // 2
    plain = x.dtype == w_gate_up.dtype == out_dtype == torch.bfloat16 and x.is_contiguous() \
        and w_gate_up.is_contiguous()
    if plain and tcgen05_pays(rows, inter, k, w_gate_up.dtype, col_tile=128):
        return gemm_tcgen05(x, w_gate_up, swiglu=True, interleaved=interleaved, act=act, consts=consts)
    if plain and interleaved and skinny_pays(x, w_gate_up, gated=True):
        return gemm_skinny_swiglu(x, w_gate_up, act, consts)
    gate_up = linear(x, w_gate_up, out_dtype=out_dtype)
    out = torch.empty((rows, inter), dtype=out_dtype, device=x.device)
    return swiglu(gate_up, out, interleaved, act, consts)


# --------------------------------------------------------------------------- attention with a modified score
def _plane(plane: torch.Tensor):
    """(pointer, elements from one page to the next) of a cache plane [pages, heads, page, width]: a
    view into the pages whose last three axes are dense."""
    heads, page, width = plane.shape[1:]
    assert plane.stride(3) == 1 and plane.stride(2) == width and plane.stride(1) == page * width
    return plane.data_ptr(), plane.stride(0)


BIASED_FAST = True       # False: every row takes the general kernel (for comparisons)


@functools.lru_cache(maxsize=4096)      # up to 64 candidates, asked for once per layer of a step
def biased_decode_splits(rows: int, kv_heads: int, reach: int) -> int:
    """Runs of keys per (row, key/value head) of ``attention_biased``'s one-token kernel, by the time its grid takes: rounds of the
    blocks that are resident at once (two per multiprocessor), each as long as a run's tiles of 64 keys and some three more
    for its start and end; more than one run costs the kernel that adds them, as long as a tile.  What is empty of the last round
    counts by half: where the rows' lengths differ, the short ones' places are free early.  A run keeps at least 192 keys of
    the ``reach`` a row can see.  (Against runs for two blocks per multiprocessor whatever the last round, 1184 steps of 1 to 128
    rows, 1 to 8 key/value heads, 260 to 8000 keys: a tenth less time on average where all rows are as long, 7% where the
    shortest has half the keys; of these 8 rows of 8 heads at 2000 keys 40 us, now 34, 16 at 4000 105 and 87, 40 at 4000 201 and 170,
    64 at 2000 139 both.  Ten of the uneven steps take 3 to 15% longer, most of them with one key/value head; with whole rounds
    and three tiles for the adding kernel eighteen did: 80 rows of 2 heads at 1000 44 us, 40 with two runs or three.  These are
    figures of the kernel with the heads as rows, two blocks per multiprocessor.  Steps of at most eight heads per block run three
    and gain at every point, but not always the most with these runs, this rule's and the best: 8 rows of 8 heads at 2000 27.6 us both,
    16 at 4000 66.6 both, 40 at 4000 136 and 126 (four), 64 at 2000 124 and 110 (four), 80 of 2 at 1000 36 and 29 (one).)"""
    tiles, resident = -(-reach // 64), 2 * SM_COUNT
    best, least = 1, None
    for splits in range(1, max(1, min(reach // 192, 64)) + 1):
        blocks = rows * kv_heads * splits
        half_rounds = -(-blocks // resident) + max(1.0, blocks / resident)
        cost = half_rounds * (-(-tiles // splits) + 3) + (2 if splits > 1 else 0)
        if least is None or cost < least:
            best, least = splits, cost
    return best


QK_WHOLE = 2             # norm of all heads together (csrc/attention_biased.cu, QkNorm)


def qkv_unit_store(proj: torch.Tensor, q_out: torch.Tensor, positions, token_slot, block_table,
                   k_plane: Optional[torch.Tensor], v_plane: Optional[torch.Tensor], page_size: int,
                   q_heads: int, kv_heads: int, dk: int, dv: int, eps: Optional[float],
                   q_gain: Optional[torch.Tensor] = None, k_gain: Optional[torch.Tensor] = None,
                   store: bool = True, inv_freq: Optional[torch.Tensor] = None, rot_dims: int = 0,
                   q_temperature=None, values_are_keys: bool = False, bias: Optional[torch.Tensor] = None,
                   norm_whole: bool = False, rot_pairs: bool = False, value_mix=None) -> None:
    """Rows of ``proj`` = q heads | k heads | v heads | anything: queries and keys divided per head by
    their root mean square (``eps`` None: left as they are; gains optional), queries to ``q_out``,
    keys and values of every row into their planes of the paged cache (``store``).  Keys have width
    ``dk``, values ``dv``.  Rows with a negative slot are skipped.  ``inv_freq`` [rot_dims / 2] float32: the first
    ``rot_dims`` elements of every query and key head turn by position * inv_freq (pairs half the rotated width
    apart), after the norm.  ``q_temperature`` (coef, every): queries times 1 + coef ln(floor((pos + 1) / every) + 1).
    ``values_are_keys``: the rows carry no values; a value is its key as projected, before the norm (dv = dk).
    ``bias`` float32, one number per q | k | v column: added to the rows, in float32, before anything else.
    ``norm_whole``: the queries of a row are normed as one vector of all heads, and so are its keys; the gains then
    have q_heads * dk and kv_heads * dk numbers.  ``rot_pairs``: elements 2 i and 2 i + 1 turn together.
    ``value_mix`` (other, its bias or None, share): values become (1 - share) v + share (other + bias) before they
    are written, with ``other`` [T, kv_heads * dv] the values of the same rows elsewhere (a view, rows may be strided)."""
    _cuda(proj, q_out, positions, token_slot, block_table, q_gain, k_gain, inv_freq, bias)
    if bias is not None:
        assert bias.dtype == torch.float32 and bias.numel() == (q_heads + kv_heads) * dk + (0 if values_are_keys else kv_heads * dv)
    if inv_freq is not None:
        assert inv_freq.dtype == torch.float32 and inv_freq.numel() == rot_dims // 2
    if q_gain is not None:
        assert q_gain.dtype == k_gain.dtype == proj.dtype
        assert (q_gain.numel(), k_gain.numel()) == ((q_heads * dk, kv_heads * dk) if norm_whole else (dk, dk))
    other, other_bias, share = value_mix if value_mix is not None else (None, None, 0.0)
    if other is not None:
        assert other.is_cuda and other.dtype == proj.dtype and other.stride(1) == 1
        assert tuple(other.shape) == (proj.shape[0], kv_heads * dv)
        if other_bias is not None:
            assert other_bias.dtype == torch.float32 and other_bias.is_contiguous() and other_bias.numel() == kv_heads * dv
    coef, every = q_temperature if q_temperature is not None else (0.0, 0)
    assert q_out.dtype == proj.dtype and tuple(q_out.shape) == (proj.shape[0], q_heads * dk)
    kp = vp = None
    stride = 0
    if store:
        assert k_plane.dtype == v_plane.dtype == proj.dtype
        assert tuple(k_plane.shape[1:]) == (kv_heads, page_size, dk) and tuple(v_plane.shape[1:]) == (kv_heads, page_size, dv)
        (kp, stride), (vp, stride_v) = _plane(k_plane), _plane(v_plane)
        assert stride == stride_v
    _check(lib().tllm_qkv_unit_store(
        _p(proj), proj.shape[1], _p(q_gain), _p(k_gain), float(eps or 1.0),
        QK_WHOLE if eps is not None and norm_whole else int(eps is not None), _p(positions),
        _p(token_slot), _p(block_table), block_table.shape[1] if block_table is not None else 0, page_size,
        kp, vp, stride, _p(q_out), _dt(proj), proj.shape[0], q_heads, kv_heads, dk, dv, int(store),
        _p(inv_freq), int(rot_dims if inv_freq is not None else 0), int(rot_pairs), float(coef), int(every),
        int(values_are_keys), _p(bias), None if other is None else other.data_ptr(),
        0 if other is None else other.stride(0), _p(other_bias), float(share), _stream()), "qkv_unit_store")


def attention_biased(q: torch.Tensor, k_plane: torch.Tensor, v_plane: torch.Tensor, positions, token_slot,
                     block_table, page_size: int, q_heads: int, kv_heads: int, dk: int, dv: int, scale: float,
                     out: torch.Tensor, softcap: float = 0.0, chunk: int = 0, window: int = 0,
                     sink: bool = False, slopes: Optional[torch.Tensor] = None,
                     gate: Optional[torch.Tensor] = None, ctx=None, sink_logits: Optional[torch.Tensor] = None,
                     values_in_keys: bool = False, distance_bias: Optional[torch.Tensor] = None,
                     gate_per_head: bool = False, difference=None) -> torch.Tensor:
    """Attention of every row of ``q`` [T, q_heads * dk] over the keys of its own request, with the
    score s = (q . k) * scale changed in this order by whatever is given: ``softcap`` (s <- cap *
    tanh(s / cap)), ``slopes`` [q_heads] float32 (s <- s - slope * (pos - key pos)); keys j <= pos from
    the row's own ``chunk`` of positions and from its ``window``; ``sink``: one is added to the softmax's
    denominator, or exp(sink_logits[head]) with ``sink_logits`` [q_heads] float32 (a learned score that is
    neither scaled nor capped).  ``gate`` (a view [T, q_heads * dv], or with ``gate_per_head`` [T, q_heads],
    whose rows may be strided): out *= sigmoid(gate).  ``values_in_keys``: a value is the first ``dv`` elements of its key's row (``v_plane`` is
    not looked at), as in attention over compressed vectors that are key and, in part, value at once.
    ``distance_bias`` [q_heads, L] float32: entry [h, min(pos - key pos, L - 1)] is added to the score after
    everything else (a learned bias by distance; it is not scaled).
    ``difference`` (lambda, eps, scale): two attention maps per head over the same values; ``q`` is [T, q_heads * 2 dk] and
    a key 2 dk wide, head by head map 1 | map 2, and the result a1 - lambda a2, divided by its root mean square over dv
    (``eps``) and times ``scale``."""
    _cuda(q, positions, token_slot, block_table, out, slopes, sink_logits, distance_bias)
    dist_len = 0
    if distance_bias is not None:
        assert distance_bias.dtype == torch.float32 and distance_bias.dim() == 2 and distance_bias.shape[0] == q_heads
        dist_len = distance_bias.shape[1]
    tokens = q.shape[0]
    maps = 1 if difference is None else 2
    assert tuple(out.shape) == (tokens, q_heads * dv) and out.dtype == q.dtype and q.shape[1] == q_heads * maps * dk
    assert k_plane.shape[3] == maps * dk and (maps == 1 or not values_in_keys)
    kp, stride = _plane(k_plane)
    if values_in_keys:
        assert dv <= dk
        vp, stride_v, v_row = kp, stride, dk
    else:
        (vp, stride_v), v_row = _plane(v_plane), dv
    assert stride == stride_v and k_plane.dtype == q.dtype
    if sink_logits is not None:
        assert sink and sink_logits.dtype == torch.float32 and sink_logits.numel() == q_heads
    gate_stride = 0
    if gate is not None:
        assert gate.dtype == q.dtype and gate.stride(1) == 1
        assert tuple(gate.shape) == ((tokens, q_heads) if gate_per_head else tuple(out.shape))
        gate_stride = gate.stride(0)
    if slopes is not None:
        assert slopes.dtype == torch.float32 and slopes.numel() == q_heads
    gate_ptr = None if gate is None else gate.data_ptr()
    mods = (float(scale), float(softcap or 0.0), int(chunk or 0), int(window or 0), int(bool(sink)), _p(slopes),
            _p(sink_logits), _p(distance_bias), dist_len, v_row, gate_ptr, gate_stride, int(gate_per_head), maps,
            *((0.0, 0.0, 0.0) if difference is None else (float(v) for v in difference)))
    consts = mods + (_p(out), _stream())
    # width 128 on both sides, one map and not a table of biases beside other changes: prompt portions go to the
    # tcgen05 kernel of the plain cache, which reads the two planes
    changed = bool(softcap) or bool(chunk) or slopes is not None or gate is not None or (sink and sink_logits is None)
    tcgen05 = PREFILL_TCGEN05 and dk == 128 and dv == 128 and maps == 1 and not values_in_keys \
        and not (changed and distance_bias is not None) \
        and page_size % 16 == 0 and stride % 128 == 0 and q_heads <= 65535 \
        and (q.data_ptr() | out.data_ptr() | kp | vp) % 16 == 0
    if BIASED_FAST and ctx is not None and ctx.pf_tiles is not None and ctx.tokens == tokens \
            and q.dtype == torch.bfloat16 and (gate_stride % 2 == 0 or gate_per_head) and v_row % 8 == 0 \
            and lib().tllm_attention_maps_fast_ok(q_heads, kv_heads, dk, dv, maps):
        # one-token rows: keys read once per group of query heads; longer portions: tensor-core tiles
        if ctx.n_dec:
            reach = min(v for v in (chunk, window, ctx.max_context or 1 << 30) if v)
            splits = biased_decode_splits(ctx.n_dec, kv_heads, reach)
            part = None
            if splits > 1:
                part = workspace(q.device, ctx.n_dec * q_heads * maps * splits * (dv + 2))
            _check(lib().tllm_attention_biased_decode(
                _p(q), kp, vp, stride, _p(positions), _p(token_slot), _p(ctx.dec_rows), ctx.n_dec, _p(block_table),
                block_table.shape[1], page_size, q_heads, kv_heads, dk, dv, *mods, splits, _p(part), _p(out), _stream()),
                "attention_biased_decode", kernels=2 if splits > 1 else 1)
        if ctx.n_tiles and tcgen05 and getattr(ctx, "n_tiles256", 0):
            pairs = prefill_tcgen05_block_rows(q_heads, kv_heads) == 128
            blocks = ctx.n_tiles128 if pairs else ctx.n_tiles256
            keys = min([ctx.max_context] + [v + 256 for v in (window, chunk) if v])
            splits = prefill_splits(blocks * (q_heads // 2 if pairs else q_heads), keys)
            part_o = part_ml = None
            if splits > 1:
                n = tokens * q_heads * splits
                ws = workspace(q.device, n * (dv + 2))
                part_o, part_ml = ws[:n * dv], ws[n * dv:n * (dv + 2)]
            global tcgen05_calls
            tcgen05_calls += 1
            _check(lib().tllm_attention_planes_prefill_tc(
                _p(q), tokens, kp, vp, stride, k_plane.shape[0], _p(ctx.seg_info), _p(ctx.pf_tiles), blocks,
                _p(block_table), block_table.shape[1], page_size, q_heads, kv_heads, int(window or 0), float(scale),
                _p(distance_bias), dist_len, _p(sink_logits), float(softcap or 0.0), int(chunk or 0), int(bool(sink)), _p(slopes),
                gate_ptr, gate_stride, int(gate_per_head), _p(out), splits, _p(part_o), _p(part_ml),
                _p(error_word(q.device)), _stream()), "attention_planes_prefill_tc", kernels=2 if splits > 1 else 1)
        elif ctx.n_tiles:
            _check(lib().tllm_attention_biased_prefill(
                _p(q), kp, vp, stride, _p(ctx.seg_info), _p(ctx.pf_tiles), ctx.n_tiles, _p(block_table),
                block_table.shape[1], page_size, q_heads, kv_heads, dk, dv, *consts), "attention_biased_prefill")
        return out
    _check(lib().tllm_attention_biased_general(
        _p(q), kp, vp, stride, _p(positions), _p(token_slot), _p(block_table), block_table.shape[1], page_size,
        _dt(q), tokens, q_heads, kv_heads, dk, dv, *consts), "attention_biased")
    return out


# --------------------------------------------------------------------------- stream, embedding with positions, activations
ELEMENTWISE_ACTIVATIONS = {"silu": 0, "gelu_tanh": 1, "gelu_erf": 2, "relu2": 3, "tanh": 5}      # codes of csrc/common.cuh (GateAct); relu2 = max(x, 0)^2


def embedding_norm(ids: torch.Tensor, table: torch.Tensor, out: torch.Tensor, scale: float = 1.0,
                   positions: Optional[torch.Tensor] = None, pos_table: Optional[torch.Tensor] = None,
                   gain: Optional[torch.Tensor] = None, eps: float = 0.0) -> torch.Tensor:
    """out[t] = norm(table[ids[t]] * scale + pos_table[positions[t]]) in float32: the position table and the
    norm (``gain`` float32, the factor itself; x / sqrt(mean(x^2) + eps) * gain) only where they are given."""
    _cuda(ids, table, out, positions, pos_table, gain)
    assert ids.dtype == torch.int32 and out.dtype == torch.float32
    vocab, hidden = table.shape
    if pos_table is not None:
        assert pos_table.dtype == table.dtype and pos_table.shape[1] == hidden and positions.dtype == torch.int32
    if gain is not None:
        assert gain.dtype == torch.float32 and gain.numel() == hidden
    _check(lib().tllm_embedding_norm(_p(ids), _p(positions), _p(table), _p(pos_table), _dt(table), _p(gain), float(eps),
                                     float(scale), _p(out), ids.numel(), hidden, vocab,
                                     0 if pos_table is None else pos_table.shape[0], _stream()), "embedding_norm")
    return out


def stream_add(h: torch.Tensor, delta: Optional[torch.Tensor], out: torch.Tensor,
               post_gain: Optional[torch.Tensor] = None, post_eps: float = 0.0) -> torch.Tensor:
    """h += delta (float32, written back) and out = h in the storage type, with no norm on the way out.  With
    ``post_gain`` the delta is normed first: h += post_gain * delta / sqrt(mean(delta^2) + post_eps)."""
    _cuda(h, delta, out, post_gain)
    assert h.dtype == torch.float32 and out.shape == h.shape
    if delta is not None:
        assert delta.dtype == out.dtype and delta.shape == h.shape
    gdt = _dt(post_gain) if post_gain is not None else F32
    _check(lib().tllm_stream_add(_p(h), _p(delta), _p(post_gain), gdt, float(post_eps), _p(out), _dt(out), h.shape[0],
                                 h.shape[1], _stream()), "stream_add")
    return out


def linear_act(x: torch.Tensor, weight: torch.Tensor, act: str, out_dtype: torch.dtype) -> torch.Tensor:
    """act(x . weight^T) with ``act`` one of ``ELEMENTWISE_ACTIVATIONS``.  In bfloat16 the activation sits in the
    product's epilogue where this package's own products run (at most 8 rows: the weight-streaming kernel; from
    256 rows on, where the tiles fill the GPU: the tcgen05 kernel); else the product is followed by the
    activation kernel."""
    rows, k = x.shape
    plain = x.dtype == weight.dtype == out_dtype == torch.bfloat16 and x.is_contiguous() and weight.is_contiguous()
    if plain and 0 < rows <= SKINNY_MAX_ROWS and k % 8 == 0:
        _cuda(x, weight)
        out = torch.empty((rows, weight.shape[0]), dtype=torch.bfloat16, device=x.device)
        _check(lib().tllm_gemm_skinny_act(_p(x), _p(weight), _p(out), rows, weight.shape[0], k,
                                          ELEMENTWISE_ACTIVATIONS[act], _stream()), "gemm_skinny_act")
        return out
    if plain and tcgen05_pays(rows, weight.shape[0], k, weight.dtype):
        return gemm_tcgen05(x, weight, act=act, unary=True)
    return activation(linear(x, weight, out_dtype=out_dtype), act)


def softcap(x: torch.Tensor, cap: float) -> torch.Tensor:
    """x <- cap * tanh(x / cap) in place, float32."""
    _cuda(x)
    assert x.dtype == torch.float32
    _check(lib().tllm_softcap(_p(x), float(cap), x.numel(), _stream()), "softcap")
    return x


def activation(x: torch.Tensor, act: str, ids: Optional[torch.Tensor] = None, table: Optional[torch.Tensor] = None,
               col0: int = 0) -> torch.Tensor:
    """act(x) element by element (``silu``, ``gelu_tanh``, ``gelu_erf``; float32 inside); with ``table`` [vocab,
    columns] and ``ids``, times table[ids[t], col0 + j]: a gate on a vector looked up by the row's token."""
    _cuda(x, ids, table)
    tokens, width = x.shape
    out = torch.empty_like(x)
    if table is not None:
        assert table.dtype == x.dtype and ids.dtype == torch.int32 and ids.numel() == tokens
    _check(lib().tllm_activation(_p(x), _p(out), _dt(x), ELEMENTWISE_ACTIVATIONS[act], tokens, width, _p(ids), _p(table),
                                 0 if table is None else table.shape[1], int(col0),
                                 0 if table is None else table.shape[0], _stream()), "activation")
    return out


# --------------------------------------------------------------------------- several residual streams
def embedding_sinusoid(ids: torch.Tensor, positions: torch.Tensor, table: torch.Tensor, freq: torch.Tensor, scale: float,
                       streams: int = 1) -> torch.Tensor:
    """[T, streams * width] float32, every stream the same: table[ids[t]] * scale + the position's sinusoids (column 2 i
    the sine, 2 i + 1 the cosine of position * frequency i).  ``freq`` [ceil(width / 2), 2] float32: a frequency and the
    rest that rounding it left.  Rows with a negative id become zero."""
    _cuda(ids, positions, table, freq)
    vocab, width = table.shape
    assert ids.dtype == positions.dtype == torch.int32 and freq.dtype == torch.float32 and tuple(freq.shape) == ((width + 1) // 2, 2)
    out = torch.empty((ids.numel(), streams * width), dtype=torch.float32, device=ids.device)
    _check(lib().tllm_embedding_sinusoid(_p(ids), _p(positions), _p(table), _dt(table), _p(freq), float(scale), _p(out),
                                         ids.numel(), width, vocab, int(streams), _stream()), "embedding_sinusoid")
    return out


def stream_read(x: torch.Tensor, streams: int, gain: torch.Tensor, eps: float, dtype: torch.dtype,
                w_in: Optional[torch.Tensor] = None, delta: Optional[torch.Tensor] = None, mix: Optional[torch.Tensor] = None,
                w_out: Optional[torch.Tensor] = None, delta_bias: Optional[torch.Tensor] = None,
                gate: Optional[torch.Tensor] = None, gate_bias: Optional[torch.Tensor] = None,
                shift: Optional[torch.Tensor] = None, tail: Optional[torch.Tensor] = None, token_slot=None,
                seg_info=None, single_tokens: bool = False, rows: Optional[torch.Tensor] = None):
    """What stands between two sub-layers of a model with several residual streams ``x`` [T, streams * width] float32:

    * the update that the last sub-layer left, if ``delta`` [T, width] (storage type) is given: with y = (delta +
      delta_bias) * sigmoid(gate + gate_bias) (the biases float32 [width], ``gate`` logits in the storage type; each
      only where given), x_t <- sum_s mix[s, t] x_s + w_out[t] y, all streams at once from the old ones;
    * the next sub-layer's input h = gain * u / sqrt(mean(u^2) + eps), u = sum_t w_in[t] x_t (None: the plain sum);
    * with ``shift`` [width] also h + (h' - h) * shift, h' the previous token's h (rounded to the storage type as it is),
      which before a portion's first row comes from ``tail[slot]`` ([slots, width] float32), moved on to the portion's
      last row.  ``single_tokens``: every portion is one token; otherwise ``seg_info`` [segments, 4] lists them.

    Returns (x after the update (a new tensor; ``x`` itself without one), h, shifted h or None).  With ``rows`` (int32)
    only h of those rows is made and the first entry is None."""
    _cuda(x, gain, w_in, delta, mix, w_out, delta_bias, gate, gate_bias, shift, tail, token_slot, seg_info, rows)
    tokens, width = x.shape[0], x.shape[1] // streams
    assert x.dtype == gain.dtype == torch.float32 and x.shape[1] == streams * width and gain.numel() == width
    for v, n in ((w_in, streams), (mix, streams * streams), (w_out, streams), (delta_bias, width), (gate_bias, width), (shift, width)):
        assert v is None or (v.dtype == torch.float32 and v.numel() == n)
    for v in (delta, gate):
        assert v is None or (v.dtype == dtype and tuple(v.shape) == (tokens, width))
    n = tokens if rows is None else rows.numel()
    h = torch.empty((n, width), dtype=dtype, device=x.device)
    if n == 0:                                  # nothing is wanted (an empty tensor has no address to tell apart from none)
        return None, h, None
    x_new = torch.empty_like(x) if delta is not None and rows is None else None
    shifted = torch.empty_like(h) if shift is not None else None
    assert shift is None or (tail is not None and tail.dtype == torch.float32 and tail.shape[1] == width and (single_tokens or seg_info is not None))
    _check(lib().tllm_stream_read(
        _p(x), _p(x_new), _p(delta), _p(delta_bias), _p(gate), _p(gate_bias), _p(mix), _p(w_out), _p(w_in), _p(gain), float(eps),
        _p(h), _DT[dtype], _p(shift), _p(shifted), _p(tail), 0 if tail is None else tail.stride(0), int(single_tokens),
        _p(token_slot), _p(rows), n, width, streams, _stream()), "stream_read")
    if shift is not None and not single_tokens:
        _check(lib().tllm_stream_tails(_p(seg_info), seg_info.shape[0], _p(h), _DT[dtype], _p(tail), tail.stride(0), width,
                                       _stream()), "stream_tails")
    if rows is not None:
        return None, h, None
    return (x if x_new is None else x_new), h, shifted


# --------------------------------------------------------------------------- delta rule with channel-wise decay
def delta_rule_state_floats(heads: int, kv_heads: int, dk: int, dv: int, taps: int) -> int:
    """Float32 words of one request's state: S of every head in the scan kernel's layout, then the
    convolution's last ``taps - 1`` inputs."""
    return int(lib().tllm_delta_rule_state_floats(heads, kv_heads, dk, dv, taps))


SCAN_DELTA, SCAN_PLAIN, SCAN_MEMORY, SCAN_HEAD_DECAY, SCAN_ERASE, SCAN_FIXED_DECAY = 0, 1, 2, 3, 4, 5     # recurrences of the scan kernel (csrc/delta_rule.cu, ScanMode)
CHUNK_MODES = (SCAN_DELTA, SCAN_PLAIN, SCAN_HEAD_DECAY, SCAN_FIXED_DECAY)      # that csrc/chunk_scan.cu knows
# Tokens per portion, on average, from which on the recurrences run by chunks if the step is large (64 * 32768 tokens x heads x
# key elements), and from two and a half times which on in any case.  Token by token a portion takes a quarter of a
# microsecond per token whatever else there is, and a step of many portions or heads as long as its work; by chunks there
# are two kernels and less work.  The delta rule with 32 heads of 128 x 128, token by token and by chunks: one portion of 64
# tokens 27 and 32 us, of 256 80 and 65; eight of 48 tokens 82 and 77, of 64 104 and 91.  Between the lines both take some 40 us,
# and the second launch costs more than it saves (four portions of 90 tokens, 16 heads of 64 x 128: 29 and 30 us, of the whole
# op 40 and 48).  The chunks' figures are those of kernels on the float32 pipe; the present ones, on the tensor cores, are faster, so
# nothing that goes by chunks is slower by them (32 points on that side of the lines, 8 to 69% less time), but some portions on the
# other side would be faster by chunks now: the delta rule, one portion of 100 tokens 37 and 32 us (eight of 48 not: 80 and 83).
CHUNK_TOKENS = 64


def chunks_pay(mode: int, segments: int, tokens: int, heads: int, dk: int, cols: int) -> bool:
    """Whether a recurrence over portions is faster by chunks than token by token, with ``cols`` value columns per head.

    Beside the lines at ``CHUNK_TOKENS`` (which move with it): the chunks' matrices are made once per (portion, head), whatever
    the columns, and token by token every column is a thread's own work.  So with many of either the chunks pay only where a head
    has enough columns.  Token by token and by chunks, portions of 256 tokens: decays per channel, eight portions of 64 heads
    of 64 x 16 82 and 112 us, of 64 x 48 (32 heads) 100 and 112, of 64 x 64 101 and 110; of 128 x 16 129 and 147; one decay
    per head, twelve of 64 heads of 64 x 16 96 and 114.  The delta rule's chunks do twice the work of the others', so with keys of
    64 elements they win only while the columns of a step are few: 16 heads of 64 x 128 529 and 169 us for 2048 tokens, three
    portions of 32 heads up to a fifth faster, four 111 and 126, twelve of 64 heads of 64 x 64 310 and 341.  (On the float32 pipe;
    on the tensor cores these lines lie further out: four portions of 32 heads 110 and 95, eight of 32 heads of 64 x 64 with decays
    per channel 100 and 85, of one decay per head, twelve of 64 heads of 64 x 16, 96 and 87; of 64 x 16 with decays per channel 82 and
    99, of 128 x 16 with the delta rule 112 and 126 as before.)"""
    if tokens < CHUNK_TOKENS * segments or not (2 * tokens >= 5 * CHUNK_TOKENS * segments or tokens * heads * dk >= CHUNK_TOKENS << 15):
        return False
    pairs = segments * heads * CHUNK_TOKENS / 64
    if mode == SCAN_DELTA and dk == 64:
        return pairs <= 160 and pairs * cols <= 96 * 128
    return pairs <= 160 or cols >= (48 if dk == 128 else 64 if mode == SCAN_HEAD_DECAY else 128)


def _scan(mode, seg_info, tokens, token_slot, qn, kn, vv, decay, beta, state, heads, kv_heads, dk, cols, o_raw, fgate=None,
          erase=None, aux_off=0, floor_eps=0.0, den=None) -> None:
    """The recurrence itself: by chunks of sixteen tokens for prompt portions, else token by token."""
    segments = tokens if seg_info is None else seg_info.shape[0]
    if seg_info is not None and mode in CHUNK_MODES and 0 < segments <= 65535 and dk in (64, 128) and cols % 16 == 0 \
            and chunks_pay(mode, segments, tokens, heads, dk, cols):
        # T and Q T of every chunk and head: a chunk of sixteen tokens at most per sixteen rows and one more per portion
        pairs = torch.empty((tokens // 16 + segments) * heads * 512, dtype=torch.float32, device=qn.device)
        _check(lib().tllm_chunk_scan(_p(seg_info), segments, tokens, _p(qn), _p(kn), _p(vv), _p(decay), _p(beta), _p(fgate),
                                     _p(pairs), _p(state), state.stride(0), heads, kv_heads, dk, cols, _p(o_raw), mode, _stream()),
               "chunk_scan", kernels=2)
        return
    _check(lib().tllm_delta_scan(_p(seg_info), segments, tokens, _p(token_slot), _p(qn), _p(kn), _p(vv), _p(decay), _p(beta),
                                 _p(state), state.stride(0), heads, kv_heads, dk, cols, _p(o_raw), mode, _p(fgate), _p(erase),
                                 aux_off, float(floor_eps), _p(den), _stream()), "delta_scan")


INPUT_ACTS = {None: 0, "silu": 1}                     # of q, k and v before a recurrence without a correction
GATE_ACTS = {"sigmoid": 0, "silu": 1}                # what the read-out is multiplied by: act(gate)


def _delta_finish(o_raw, gate, out_weight, weight_per_head, eps, token_slot, tokens, heads, kv_heads, dk, dv, out_dtype,
                  proj, ld, taps, state, den, gate_act):
    out = torch.empty((tokens, heads * dv), dtype=out_dtype, device=o_raw.device)
    assert gate.stride(1) == 1 and gate.dtype in (torch.float32, out_dtype) and out_weight.dtype == torch.float32
    assert out_weight.numel() == (heads * dv if weight_per_head else dv)
    _check(lib().tllm_delta_finish(_p(o_raw), gate.data_ptr(), int(gate.dtype == torch.float32), gate.stride(0), _p(out_weight),
                                   float(eps), _p(token_slot), tokens, heads, kv_heads, dk, dv, _p(out), _dt(out), _p(proj), ld,
                                   taps, _p(state), state.stride(0), _p(den), GATE_ACTS[gate_act],
                                   dv if weight_per_head else 0, _stream()), "delta_finish")
    return out


def delta_rule(proj: torch.Tensor, conv_w: torch.Tensor, taps: int, a: torch.Tensor, dt_bias: torch.Tensor,
               rate: torch.Tensor, gate: torch.Tensor, out_weight: torch.Tensor, eps: float, token_slot: torch.Tensor,
               seg_info: Optional[torch.Tensor], state: torch.Tensor, heads: int, kv_heads: int, dk: int, dv: int,
               q_scale: float, unit_eps: float, out_dtype: torch.dtype, conv_t: Optional[torch.Tensor] = None,
               decay_per_head: bool = False, beta_col: Optional[int] = None, gate_act: str = "sigmoid") -> torch.Tensor:
    """One step of the delta rule for every row of ``proj`` [T, >= channels + heads] = q channels | k channels | v
    channels | ... with the beta logits at column ``beta_col`` (None: right behind the channels), in the storage
    type: convolution with ``conv_w`` [channels, taps] and SiLU, unit q and k, g = exp(-rate_h softplus(a + dt_bias))
    with ``a`` float32 [T, heads * dk] (a decay per head and key channel) or, ``decay_per_head``, [T, heads]; the
    recurrence over each portion's rows from ``state[slot]`` (float32, updated in place), then the read-out divided
    by its root mean square per head, times ``out_weight`` [dv] float32, times ``gate_act``(``gate``) ([T, heads * dv]
    float32 or storage type, rows may be strided).  ``seg_info`` [segments, 4] = slot, first row, length, first
    position; None: every row is a portion of one token.  ``conv_t``: the taps once more as [taps, channels], which
    lets the kernels take eight channels per access.  Returns [T, heads * dv] in ``out_dtype``."""
    _cuda(proj, conv_w, dt_bias, rate, out_weight, token_slot, seg_info, state, conv_t)
    tokens, ld = proj.shape
    assert a.dtype == dt_bias.dtype == rate.dtype == out_weight.dtype == state.dtype == torch.float32
    assert a.stride(1) == 1 and conv_w.dtype == proj.dtype and state.dim() == 2
    assert dt_bias.numel() == (heads if decay_per_head else heads * dk)
    dev = proj.device
    ws = workspace(dev, tokens * (2 * kv_heads * dk + 2 * heads * dv + heads * dk + heads))
    at = 0

    def take(n):
        nonlocal at
        t = ws[at:at + tokens * n]
        at += tokens * n
        return t
    # q, k and the decays first: their rows start on 16-byte boundaries wherever dk is a multiple of four
    qn, kn, decay, vv, o_raw, beta = (take(kv_heads * dk), take(kv_heads * dk), take(heads * dk), take(heads * dv),
                                      take(heads * dv), take(heads))
    _check(lib().tllm_delta_prepare(_p(proj), ld, _dt(proj), _p(conv_w), _p(conv_t), taps, a.data_ptr(), a.stride(0), _p(dt_bias), _p(rate),
                                    _p(token_slot), _p(state), state.stride(0), heads, kv_heads, dk, dv, float(q_scale),
                                    float(unit_eps), _p(qn), _p(kn), _p(vv), _p(decay), _p(beta), tokens,
                                    int(decay_per_head), -1 if beta_col is None else int(beta_col), _stream()),
           "delta_prepare")
    _scan(SCAN_DELTA, seg_info, tokens, token_slot, qn, kn, vv, decay, beta, state, heads, kv_heads, dk, dv, o_raw)
    return _delta_finish(o_raw, gate, out_weight, False, eps, token_slot, tokens, heads, kv_heads, dk, dv, out_dtype,
                         proj, ld, taps, state, None, gate_act)


def erase_delta_rule(proj: torch.Tensor, a_col: int, z: torch.Tensor, z_bias: torch.Tensor, a_bias: torch.Tensor,
                     rate: float, gate: torch.Tensor, gate_act: str, out_weight: torch.Tensor, weight_per_head: bool,
                     eps: float, token_slot: torch.Tensor, seg_info: Optional[torch.Tensor], state: torch.Tensor, heads: int,
                     dk: int, dv: int, unit_eps: float, out_dtype: torch.dtype) -> torch.Tensor:
    """One step of the delta rule with a removal rate per head and key channel, for every row of ``proj`` [T, ...] =
    r | k | v | ... in the storage type with the removal's logits at column ``a_col``: with u = k / sqrt(sum(k^2) +
    ``unit_eps``) per head, w = exp(-``rate`` sigmoid(z + z_bias)) and a = sigmoid(logits + a_bias),
    S <- diag(w) S - (a * u) (u^T S) + k v^T (both terms from the old S), o = S^T r, from ``state[slot]`` (float32,
    updated in place).  ``z`` [T, heads * dk] float32, ``z_bias`` and ``a_bias`` [heads * dk] float32.  The read-out is
    divided by its root mean square per head, times ``out_weight``, times ``gate_act``(``gate``), as in
    ``linear_recurrence``.  Returns [T, heads * dv] in ``out_dtype``."""
    _cuda(proj, z, z_bias, a_bias, out_weight, token_slot, seg_info, state)
    tokens, ld = proj.shape
    assert z.dtype == z_bias.dtype == a_bias.dtype == state.dtype == torch.float32 and state.dim() == 2
    assert z.shape == (tokens, heads * dk) and z_bias.numel() == a_bias.numel() == heads * dk
    assert state.shape[1] == delta_rule_state_floats(heads, heads, dk, dv, 1)
    ws = workspace(proj.device, tokens * heads * (4 * dk + 2 * dv) + 32)
    at = 0

    def take(n):
        nonlocal at
        t = ws[at:at + tokens * n]
        at += -(-tokens * n // 4) * 4
        return t
    qn, kn, decay, erase, vv, o_raw = (take(heads * dk), take(heads * dk), take(heads * dk), take(heads * dk),
                                       take(heads * dv), take(heads * dv))
    _check(lib().tllm_erase_prepare(_p(proj), ld, _dt(proj), int(a_col), _p(z), z.stride(0), _p(z_bias), _p(a_bias), float(rate),
                                    _p(token_slot), heads, dk, dv, float(unit_eps), _p(qn), _p(kn), _p(vv), _p(decay),
                                    _p(erase), tokens, _stream()), "erase_prepare")
    _scan(SCAN_ERASE, seg_info, tokens, token_slot, qn, kn, vv, decay, None, state, heads, heads, dk, dv, o_raw, erase=erase)
    return _delta_finish(o_raw, gate, out_weight, weight_per_head, eps, token_slot, tokens, heads, heads, dk, dv,
                         out_dtype, None, 0, 1, state, None, gate_act)


LINEAR_KINDS = {"channel_decay": 0, "log_gates": 1, "fixed_decay": 2}      # csrc/delta_rule.cu, LinearKind


def linear_recurrence_state_floats(kind: str, heads: int, dk: int, dv: int) -> int:
    """Float32 words of one request's state of ``linear_recurrence``: S of every head in the scan kernel's layout
    (with ``log_gates`` one more column, the normaliser) and, with ``log_gates``, the running maximum per column."""
    cols = dv + 1 if kind == "log_gates" else dv
    s_floats = delta_rule_state_floats(heads, heads, dk, cols, 1)
    return s_floats + (heads * cols if kind == "log_gates" else 0)


def linear_recurrence(proj: torch.Tensor, kind: str, z: Optional[torch.Tensor], z_bias: torch.Tensor, p0: float,
                      gate: torch.Tensor, gate_act: str, out_weight: torch.Tensor, weight_per_head: bool, eps: float,
                      token_slot: torch.Tensor, seg_info: Optional[torch.Tensor], state: torch.Tensor, heads: int,
                      dk: int, dv: int, q_scale: float, out_dtype: torch.dtype, floor_eps: float = 1e-6,
                      input_act: Optional[str] = None, norm_whole: bool = False) -> torch.Tensor:
    """One step of a recurrence S <- decay S + k (w v)^T, o = S^T q per head, for every row of ``proj`` [T, >= heads
    (2 dk + dv)] = q | k | v in the storage type (q is multiplied by ``q_scale``), from ``state[slot]`` (float32,
    updated in place).  ``kind``:

    * ``channel_decay``: a decay per key channel sigmoid(z + z_bias)^p0 with ``z`` [T, heads * dk] float32, w = 1;
    * ``log_gates``: ``z`` [T, 2 heads] float32 = write | keep logits (plus ``z_bias``), each capped as p0 tanh(. /
      p0); with i the capped write logit and f = logsigmoid(capped keep logit), a running maximum m <- max(f + m, i)
      that starts at zero: decay = exp(f + m_before - m), w = exp(i - m); a vector n <- decay n + w k is kept beside
      S and the read-out is S^T q / (max(|n . q|, exp(-m)) + ``floor_eps``);
    * ``fixed_decay``: no ``z``; ``z_bias`` [heads] float32 holds every head's decay itself, w = 1.

    ``input_act`` ``silu``: q (before its scale), k and v are SiLU of what is in ``proj``.  Then the read-out is divided by its root mean square per head (``eps``), times ``out_weight`` ([dv], or [heads *
    dv] with ``weight_per_head``) float32, times ``gate_act``(``gate``) ([T, heads * dv], rows may be strided).
    ``norm_whole``: the root mean square is the one of all heads together (``weight_per_head``, no divisor).  Returns [T, heads * dv] in ``out_dtype``."""
    _cuda(proj, z_bias, out_weight, token_slot, seg_info, state)
    tokens, ld = proj.shape
    assert z_bias.dtype == state.dtype == torch.float32 and state.dim() == 2
    memory, fixed = kind == "log_gates", kind == "fixed_decay"
    if fixed:
        assert z is None and z_bias.numel() == heads
    else:
        assert z.dtype == torch.float32 and z.stride(1) == 1
    cols = dv + 1 if memory else dv
    assert state.shape[1] == linear_recurrence_state_floats(kind, heads, dk, dv)
    dev = proj.device
    ws = workspace(dev, tokens * (3 * heads * dk + heads * (cols + dv) + 3 * heads + 8))
    at = 0

    def take(n):
        nonlocal at
        t = ws[at:at + tokens * n]
        at += -(-tokens * n // 4) * 4
        return t
    qn, kn = take(heads * dk), take(heads * dk)
    decay = None if memory or fixed else take(heads * dk)
    vv, o_raw = take(heads * cols), take(heads * dv)
    wgate, fgate, den = (take(heads), take(heads), take(heads)) if memory else (None, None, None)
    _check(lib().tllm_linear_prepare(_p(proj), ld, _dt(proj), None if fixed else z.data_ptr(), 0 if fixed else z.stride(0), _p(z_bias),
                                     LINEAR_KINDS[kind], INPUT_ACTS[input_act], float(p0), _p(token_slot), heads, dk, dv, float(q_scale), _p(qn), _p(kn), _p(vv),
                                     _p(decay), _p(wgate), _p(fgate), tokens, _stream()), "linear_prepare")
    aux_off = delta_rule_state_floats(heads, heads, dk, cols, 1) if memory else 0
    _scan(SCAN_MEMORY if memory else SCAN_FIXED_DECAY if fixed else SCAN_PLAIN, seg_info, tokens, token_slot, qn, kn, vv, decay,
          wgate, state, heads, heads, dk, cols, o_raw, fgate=z_bias if fixed else fgate, aux_off=aux_off, floor_eps=floor_eps, den=den)
    if norm_whole:
        assert weight_per_head and den is None and gate.stride(1) == 1 and gate.dtype in (torch.float32, out_dtype)
        assert out_weight.dtype == torch.float32 and out_weight.numel() == heads * dv == gate.shape[1]
        out = torch.empty((tokens, heads * dv), dtype=out_dtype, device=dev)
        _check(lib().tllm_whole_finish(_p(o_raw), gate.data_ptr(), int(gate.dtype == torch.float32), gate.stride(0), _p(out_weight),
                                       float(eps), _p(token_slot), tokens, heads * dv, _p(out), _dt(out), GATE_ACTS[gate_act],
                                       _stream()), "whole_finish")
        return out
    return _delta_finish(o_raw, gate, out_weight, weight_per_head, eps, token_slot, tokens, heads, heads, dk, dv,
                         out_dtype, None, 0, 1, state, den, gate_act)


# --------------------------------------------------------------------------- selective state space
def state_space_state_floats(heads: int, groups: int, state: int, head_dim: int, taps: int) -> int:
    """Float32 words of one request's state of ``state_space``: S [state, head_dim] of every head in the scan
    kernel's layout, then the convolution's last ``taps - 1`` inputs over the channels x | B | C."""
    return delta_rule_state_floats(heads, groups, state, head_dim, 1) + (taps - 1) * (heads * head_dim + 2 * groups * state)


def state_space(proj: torch.Tensor, conv_w: torch.Tensor, conv_b: Optional[torch.Tensor], taps: int,
                dt_bias: torch.Tensor, rate: torch.Tensor, skip: torch.Tensor, out_weight: torch.Tensor, eps: float,
                norm_groups: int, token_slot: torch.Tensor, seg_info: Optional[torch.Tensor], state: torch.Tensor,
                heads: int, groups: int, n_state: int, head_dim: int, out_dtype: torch.dtype,
                conv_t: Optional[torch.Tensor] = None) -> torch.Tensor:
    """One step of a selective state space with a decay per head, for every row of ``proj`` [T, >= 2 heads P + 2 G N
    + heads] = z | x | B | C | dt in the storage type (P = ``head_dim``, N = ``n_state``, G = ``groups``): the causal
    convolution ``conv_w`` [channels, taps] with bias ``conv_b`` over x | B | C and SiLU, dt = softplus(dt +
    ``dt_bias``), per head S <- exp(-rate_h dt) S + B (dt x)^T from ``state[slot]`` (float32, updated in place), y =
    S^T C + skip_h x, then y silu(z), an RMS norm over each of ``norm_groups`` equal parts of the row and
    ``out_weight``.  ``dt_bias``, ``rate``, ``skip`` [heads], ``conv_b`` and ``out_weight`` are float32.  ``seg_info``
    as in ``delta_rule``.  ``conv_t``: the taps once more as [taps, channels], which lets the kernels take eight
    channels per access.  Returns [T, heads P] in ``out_dtype``."""
    _cuda(proj, conv_w, conv_b, dt_bias, rate, skip, out_weight, token_slot, seg_info, state, conv_t)
    tokens, ld = proj.shape
    inner, gn = heads * head_dim, groups * n_state
    channels = inner + 2 * gn
    assert dt_bias.dtype == rate.dtype == skip.dtype == out_weight.dtype == state.dtype == torch.float32
    assert conv_w.dtype == proj.dtype and tuple(conv_w.shape) == (channels, taps) and state.dim() == 2
    assert conv_b is None or (conv_b.dtype == torch.float32 and conv_b.numel() == channels)
    assert out_dtype == proj.dtype and state.shape[1] == state_space_state_floats(heads, groups, n_state, head_dim, taps)
    tail_off = delta_rule_state_floats(heads, groups, n_state, head_dim, 1)
    ws = workspace(proj.device, tokens * (2 * gn + 2 * inner + 2 * heads) + 32)
    at = 0

    def take(n):
        nonlocal at
        t = ws[at:at + tokens * n]
        at += -(-tokens * n // 4) * 4
        return t
    qn, kn, decay, step, vv, o_raw = take(gn), take(gn), take(heads), take(heads), take(inner), take(inner)
    _check(lib().tllm_ssd_prepare(_p(proj), ld, _dt(proj), _p(conv_w), _p(conv_t), _p(conv_b), taps, _p(dt_bias), _p(rate),
                                  _p(token_slot), _p(state), state.stride(0), tail_off, heads, groups, n_state, head_dim,
                                  _p(qn), _p(kn), _p(vv), _p(decay), _p(step), tokens, _stream()), "ssd_prepare")
    _scan(SCAN_HEAD_DECAY, seg_info, tokens, token_slot, qn, kn, vv, None, decay, state, heads, groups, n_state, head_dim, o_raw,
          fgate=step)
    out = torch.empty((tokens, inner), dtype=out_dtype, device=proj.device)
    _check(lib().tllm_ssd_finish(_p(o_raw), _p(vv), _p(skip), head_dim, _p(proj), ld, _dt(proj), _p(out_weight), float(eps),
                                 int(norm_groups), _p(token_slot), tokens, inner, channels, taps, _p(state),
                                 state.stride(0), tail_off, _p(out), _stream()), "ssd_finish")
    return out


# --------------------------------------------------------------------------- attention over compressed vectors
def latent_norm_store(proj: torch.Tensor, q_rank: int, rank: int, rot: int, rot_dims: int, q_gain, c_gain,
                      eps: float, freq: torch.Tensor, mag: float, positions, token_slot, block_table,
                      plane: torch.Tensor, page_size: int, store: bool = True,
                      half_pairs: bool = False) -> Optional[torch.Tensor]:
    """Rows of ``proj`` (a view whose rows may be strided) = query latent (q_rank) | key/value latent (rank) |
    shared key part (rot) | anything.  ``half_pairs``: the rotation pairs element i with i + rot_dims / 2 instead of
    its neighbour.
    Returns the query latent divided by its root mean square times ``q_gain`` (None if q_rank is 0) and
    writes [normed latent times ``c_gain`` | rotated key part] of every row into its place of ``plane``
    ([pages, 1, page, rank + rot]).  Gains and ``freq`` [rot_dims / 2] are float32."""
    _cuda(q_gain, c_gain, freq, positions, token_slot, block_table)
    assert proj.is_cuda and proj.stride(1) == 1
    tokens = proj.shape[0]
    cq = torch.empty((tokens, q_rank), dtype=proj.dtype, device=proj.device) if q_rank else None
    pp, stride = _plane(plane)
    assert plane.dtype == proj.dtype and tuple(plane.shape[1:]) == (1, page_size, rank + rot)
    _check(lib().tllm_latent_norm_store(proj.data_ptr(), proj.stride(0), _dt(proj), q_rank, rank, rot, rot_dims, _p(q_gain),
                                        _p(c_gain), float(eps), _p(freq), float(mag), _p(positions), _p(token_slot),
                                        _p(block_table), block_table.shape[1], page_size, pp, stride, _p(cq), int(store),
                                        tokens, int(half_pairs), _stream()), "latent_norm_store")
    return cq


def latent_query(q: torch.Tensor, lat: torch.Tensor, heads: int, plain: int, rot: int, rot_dims: int, rank: int,
                 freq: torch.Tensor, mag: float, positions, token_slot, half_pairs: bool = False) -> torch.Tensor:
    """[T, heads, rank + rot]: per head ``lat`` [heads, T, rank] followed by the rotated last ``rot`` elements
    of the head's query in ``q`` [T, heads * (plain + rot)] (a view whose rows may be strided)."""
    _cuda(lat, freq, positions, token_slot)
    assert q.is_cuda and q.stride(1) == 1
    tokens = q.shape[0]
    assert tuple(lat.shape) == (heads, tokens, rank) and lat.dtype == q.dtype and q.shape[1] == heads * (plain + rot)
    out = torch.empty((tokens, heads * (rank + rot)), dtype=q.dtype, device=q.device)
    _check(lib().tllm_latent_query(q.data_ptr(), q.stride(0), _p(lat), _dt(q), heads, plain, rot, rot_dims, rank, _p(freq), float(mag),
                                   _p(positions), _p(token_slot), tokens, _p(out), int(half_pairs), _stream()), "latent_query")
    return out


def heads_gate(x: torch.Tensor, gate: Optional[torch.Tensor], token_slot=None, per_head: bool = False) -> torch.Tensor:
    """[T, heads * width] = x[h, t, :] * sigmoid(gate[t, h * width + :]) for ``x`` [heads, T, width]; ``gate`` is a
    view whose rows may be strided (None: no gate); with ``per_head`` it is [T, heads], one number per head."""
    _cuda(x, token_slot)
    heads, tokens, width = x.shape
    out = torch.empty((tokens, heads * width), dtype=x.dtype, device=x.device)
    ldg = 0
    if gate is not None:
        assert gate.dtype == x.dtype and gate.stride(1) == 1
        assert tuple(gate.shape) == (tokens, heads if per_head else heads * width)
        ldg = gate.stride(0)
    _check(lib().tllm_heads_gate(_p(x), None if gate is None else gate.data_ptr(), ldg, _dt(x), heads, width, tokens,
                                 _p(token_slot), _p(out), int(per_head), _stream()), "heads_gate")
    return out


# --------------------------------------------------------------------------- mixture of experts
def moe_tile_rows() -> int:
    return int(lib().tllm_moe_tile_rows())


def moe_route(z: torch.Tensor, top: int, softmax_weights: bool = False):
    """(ids [T, top] int32, weights [T, top] float32) from float32 router logits ``z`` [T, E]: the
    ``top`` experts with the largest logits; weight sigmoid(z), or softmax over the chosen ones."""
    _cuda(z)
    assert z.dtype == torch.float32
    tokens, experts = z.shape
    ids = torch.empty((tokens, top), dtype=torch.int32, device=z.device)
    weights = torch.empty((tokens, top), dtype=torch.float32, device=z.device)
    _check(lib().tllm_moe_route(_p(z), tokens, experts, top, int(softmax_weights), _p(ids), _p(weights), _stream()),
           "moe_route")
    return ids, weights


ROUTER_SCORES = {"sigmoid": 0, "softmax": 1}      # scores over all experts (csrc/moe.cu, moe_route_grouped)


def moe_route_grouped(z: torch.Tensor, top: int, scores: str = "softmax", correction: Optional[torch.Tensor] = None,
                      groups: int = 1, keep: int = 1, scale: float = 1.0, experts: Optional[int] = None):
    """(ids [T, top] int32, weights [T, top] float32) from float32 router logits ``z`` [T, E]: scores s over all E
    experts (``softmax`` or ``sigmoid``); the choice goes by s + ``correction`` ([E] float32, if given), within the
    ``keep`` of ``groups`` equal groups of neighbouring experts whose best member scores highest; the weights are
    the chosen experts' s, times ``scale``.  Lowest index first on ties.  ``experts``: how many of the row's columns are
    logits (None: all; others may follow them)."""
    _cuda(z, correction)
    tokens, ldz = z.shape
    experts = ldz if experts is None else int(experts)
    assert z.dtype == torch.float32 and (correction is None or (correction.dtype == torch.float32 and correction.numel() == experts))
    ids = torch.empty((tokens, top), dtype=torch.int32, device=z.device)
    weights = torch.empty((tokens, top), dtype=torch.float32, device=z.device)
    _check(lib().tllm_moe_route_grouped(_p(z), ldz, tokens, experts, top, ROUTER_SCORES[scores], _p(correction), int(groups),
                                        int(keep), float(scale), _p(ids), _p(weights), _stream()), "moe_route_grouped")
    return ids, weights


class MoePlan:
    """Device-side lists that sort a step's (token, choice) assignments by expert, with the rows cut
    into tiles of ``tile_rows`` per expert.  ``real``: experts that have matrices; assignments to later ones
    (identity experts) get rows and no tiles.  ``tensor_memory``: the products over this plan take the tcgen05 kernel
    (None: tiles of 128 rows say so)."""

    def __init__(self, ids: torch.Tensor, experts: int, tile_rows: Optional[int] = None, real: Optional[int] = None,
                 tensor_memory: Optional[bool] = None):
        n = ids.numel()
        self.n, self.experts = n, experts
        self.real = experts if real is None else int(real)
        self.tile_rows = tile_rows or moe_tile_rows()
        self.tensor_memory = self.tile_rows == MOE_TCGEN05_TILE if tensor_memory is None else bool(tensor_memory)
        self.max_tiles = n // self.tile_rows + experts
        ints = torch.empty(experts + 2 + 3 * n + 2 * self.max_tiles, dtype=torch.int32, device=ids.device)
        at = 0

        def take(k):
            nonlocal at
            part = ints[at:at + k]
            at += k
            return part
        self.offsets, self.n_tiles = take(experts + 1), take(1)
        self.row_of, self.src_of, self.expert_of_row = take(n), take(n), take(n)
        self.tile_expert, self.tile_row0 = take(self.max_tiles), take(self.max_tiles)
        _check(lib().tllm_moe_plan(_p(ids), n, experts, self.real, self.tile_rows, _p(self.offsets), _p(self.n_tiles),
                                   _p(self.row_of), _p(self.src_of), _p(self.expert_of_row), _p(self.tile_expert),
                                   _p(self.tile_row0), _stream()), "moe_plan")


MOE_TCGEN05_ROWS = 1        # from this many (token, choice) rows on the experts' products run on tcgen05: all of them (a larger
                            # number sends smaller steps to the mma.sync tiles, to compare the two)
MOE_TCGEN05_TILE = 128
MOE_NARROW_ROWS = 1024      # from this many rows on (and 32 per expert) their results are kept in the storage type


def moe_tcgen05_pays(rows: int, experts: int, n: int, k: int, dtype) -> bool:
    """Whether the experts' products of a step take the tcgen05 kernel: bfloat16 and whole 16-byte pieces."""
    return dtype == torch.bfloat16 and rows >= MOE_TCGEN05_ROWS and k % 8 == 0 and n % 8 == 0


def moe_row_box(rows: int, experts: int) -> int:
    """Rows per tile of a plan for the tcgen05 kernel.  Tiles of 64 leave room for more stages, tiles of 128 read an expert's
    weights once where it has more than 64 rows: with 64 experts of 2048 x 4096 (gate|up + down) 16 rows per expert take 329 + 167
    us with 64 and 331 + 165 with 128, 32 rows 348 + 172 and 345 + 169, 64 rows 364 + 187 and 342 + 179."""
    return 64 if rows <= 24 * experts else MOE_TCGEN05_TILE


def moe_result_dtype(rows: int, experts: int, dtype) -> torch.dtype:
    """How the rows of the experts' last product are kept until they are summed per token: float32 in steps of few rows,
    the storage type where many rows make them a sizeable share of a step's memory traffic."""
    return dtype if rows >= MOE_NARROW_ROWS and rows >= 32 * experts else torch.float32


def moe_grouped(a: torch.Tensor, w: torch.Tensor, plan: MoePlan, top: int, gated: bool, gather: bool,
                weights: Optional[torch.Tensor] = None, act: str = "silu", interleaved: bool = False,
                out_dtype: Optional[torch.dtype] = None, unary: bool = False, consts=None) -> torch.Tensor:
    """Per row r of the plan, A[r] . W[expert of r]^T.  ``w`` is [E, N (or 2 N: gate rows, then up rows, or
    ``interleaved`` by eight), K].  ``gather``: ``a`` is [tokens, K] and a row reads its token, times ``weights``
    [tokens, top] if given.  ``gated``: the result is act(gate) * up [rows, N] in the storage type, else
    [rows, N] float32 (``consts``: constants of ``act``, see ``ACTIVATIONS``), or with ``unary`` act(.) [rows, N] in the storage type (``act`` then one of
    ``ELEMENTWISE_ACTIVATIONS``).  A plan made for it (``plan.tensor_memory``) goes to the tcgen05 product (bfloat16
    in; the gathered rows are laid out by a kernel of their own first; a plain product leaves bfloat16, or float32 with
    ``out_dtype``).  Rows of experts without matrices (``plan.real``) are left unwritten."""
    _cuda(a, w, weights)
    experts, n_total, k = w.shape
    assert a.shape[1] == k and a.dtype == w.dtype and experts == plan.real and not (gated and unary)
    act_code = ELEMENTWISE_ACTIVATIONS[act] if unary else ACTIVATIONS[act] if gated else 0
    limit, slope = _consts(act, consts) if gated else NO_CONSTS
    n = n_total // 2 if gated else n_total
    if plan.tensor_memory:
        assert a.dtype == torch.bfloat16 and (interleaved or not gated)
        if gather:
            xs = torch.empty((plan.n, k), dtype=a.dtype, device=a.device)
            _check(lib().tllm_moe_gather(_p(a), _p(plan.src_of), _p(weights), top, _p(xs), plan.n, k, _stream()),
                   "moe_gather")
            a = xs
        wide = not gated and not unary and out_dtype == torch.float32
        out = torch.empty((plan.n, n), dtype=torch.float32 if wide else torch.bfloat16, device=a.device)
        global tcgen05_calls
        tcgen05_calls += 1
        flags = (1 | 4 | (act_code << 8)) if gated else ((16 | (act_code << 8)) if unary else 32 if wide else 0)
        _check(lib().tllm_moe_tcgen05(
            _p(a), _p(w), _p(out), plan.n, n_total, k, experts, flags, plan.tile_rows, _p(plan.tile_expert), _p(plan.tile_row0),
            _p(plan.n_tiles), _p(plan.offsets), plan.max_tiles, limit, slope, _p(error_word(a.device)), _stream()),
            "moe_tcgen05")
        return out
    out = torch.empty((plan.n, n), dtype=a.dtype if (gated or unary) else torch.float32, device=a.device)
    _check(lib().tllm_moe_grouped(
        _p(a), a.stride(0), _p(plan.src_of), _p(weights), top, _p(w), w.stride(0), _p(plan.tile_expert),
        _p(plan.tile_row0), _p(plan.n_tiles), _p(plan.offsets), _p(plan.expert_of_row), plan.n, plan.max_tiles,
        n, k, _dt(a), 1 if gated else (2 if unary else 0), int(gather), act_code, limit, slope, int(interleaved), plan.real, _p(out),
        _stream()), "moe_grouped")
    return out


def moe_combine(y: torch.Tensor, plan: MoePlan, top: int, shared: Optional[torch.Tensor], dtype: torch.dtype,
                weights: Optional[torch.Tensor] = None, identity_input: Optional[torch.Tensor] = None,
                shared_gate: Optional[torch.Tensor] = None) -> torch.Tensor:
    """out[t] = shared[t] + sum_k (weights[t, k] *) y[row of (t, k)], float32 sums, stored as ``dtype``;
    ``y`` float32 or in the storage type.  ``identity_input`` [T, width] (``dtype``): an assignment to an expert
    without matrices (``plan.real`` or later) adds the token's row of it instead of a row of ``y``.
    ``shared_gate`` [T] float32 (may be strided): the shared unit's output is multiplied by its sigmoid."""
    _cuda(y, shared, weights, identity_input)
    if identity_input is not None:
        assert identity_input.dtype == dtype and tuple(identity_input.shape) == (plan.n // top, y.shape[1])
    tokens, width = plan.n // top, y.shape[1]
    out = torch.empty((tokens, width), dtype=dtype, device=y.device)
    if shared_gate is not None:
        assert shared is not None and shared_gate.dtype == torch.float32 and tuple(shared_gate.shape) == (tokens,)
    if shared is not None:
        assert shared.dtype == dtype and tuple(shared.shape) == (tokens, width)
    _check(lib().tllm_moe_combine(_p(y), _dt(y), _p(plan.row_of), _p(weights), top, _p(shared), _p(out), _DT[dtype],
                                  tokens, width, _p(identity_input), _p(plan.expert_of_row), plan.real,
                                  None if shared_gate is None else shared_gate.data_ptr(),
                                  0 if shared_gate is None else shared_gate.stride(0), _stream()), "moe_combine")
    return out
