"""The operations a decoder step is made of, each a call into a hand-written CUDA kernel.

Tensors are torch tensors on a CUDA device (torch is used for memory and for the library matrix
product only); every function launches on torch's current stream.  There is no CPU implementation and
no fallback: a tensor on another device, a missing compiler or a failed build raises.

Matrix products: float32 runs ``gemm_f32`` (FFMA, no tensor-core mode) and, for a prompt's rows times a large matrix, ``gemm_f32_tc``
(the tensor cores over operands split into three bfloat16 parts, which lose nothing).  bfloat16 runs the weight-streaming
``mma.sync`` kernel up to 8 rows (decode of few sequences) and otherwise the library product (cuBLAS through
``torch.nn.functional.linear``), as the reference does for every linear layer (fms/modules/linear.py:119-156) —
except the gated feed-forward product, which from ``TENSOR_CORE_ROWS_GLU`` (512) rows on, where its tiles of 256
rows fit the number of rows to 6%, takes the tcgen05 kernel
with the tokens on the instruction's rows (prefill; pairs of thread blocks on one tile, the activation in its
epilogue), and the fused projection of queries, keys and values, which from ``TENSOR_CORE_ROWS_QKV`` (2,048) rows
on takes the same kernel with the rotation and the cache write in its epilogue.  The same kernel takes the plain
products from ``FMS_B200_TC_ROWS`` rows on where that is set; measured through whole prefills the library's plain
products are ahead, so by default it is not.
The gated feed-forward product of 9 to 128 rows takes a tcgen05 kernel of this library with the weights on the
instruction's rows and the activation in its epilogue (``gemm_bf16_mid.cu``); the same kernel can take the plain
products and the fused projection up to 256 rows (clusters of blocks share a tile along K; projection + rotation
+ cache write in its epilogue; ``FMS_B200_MID_OPS``), where the library's product is still ahead of it.
"""
from __future__ import annotations

import ctypes
import itertools
import os
from typing import Optional

import torch

from .build import load_launcher, load_library

F32, BF16 = 0, 1
# kinds of parameters: a pointer (a tensor's, an address or None), whole numbers of 32 and 64 bits, a float
_P, _I, _F, _U64, _L = "p", "i", "f", "i", "i"

_SIGNATURES = {
    "fms_embed_rows": [_P, _I, _P, _P, _I, _I, _I, _F, _P, _P],
    "fms_embed_rows_at": [_P, _I, _P, _P, _I, _I, _I, _F, _P, _P, _I, _P, _P],
    "fms_token_gate": [_P, _I, _P, _P, _P, _I, _I, _I, _I, _P],
    "fms_joint_activation": [_P, _P, _I, _I, _I, _P, _I, _I, _I, _I, _I, _I, _I, _I, _P],
    "fms_add_rmsnorm": [_P, _P, _P, _I, _F, _P, _I, _P, _I, _I, _I, _P],
    "fms_gated_activation": [_P, _P, _I, _I, _I, _I, _P],
    "fms_rope_store": [_P, _I, _P, _P, _P, _P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _I, _P, _I, _I, _I, _P],
    "fms_decode_advance": [_P, _P, _P, _P, _P, _I, _I, _P],
    "fms_rotary_table": [_P, _P, _P, _P, _I, _I, _P],
    "fms_gemm_f32": [_P, _P, _P, _P, _I, _I, _I, _P],
    "fms_copy_rows_f32": [_P, _P, _P, _I, _I, _I, _I, _P],
    "fms_gemm_f32_tc": [_P, _P, _P, _P, _P, _L, _I, _I, _I, _P, _P],
    "fms_linear_bf16_skinny": [_P, _P, _P, _P, _I, _I, _I, _I, _P],
    "fms_token_gate_bf16_skinny": [_P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _P],
    "fms_grouped_bf16_skinny": [_P, _P, _P, _P, _I, _I, _I, _I, _F, _F, _P],
    "fms_strided_bf16_skinny": [_P, _P, _P, _I, _I, _I, _I, _L, _L, _L, _L, _L, _P],
    "fms_linear_act_bf16_skinny": [_P, _P, _P, _P, _I, _I, _I, _I, _P],
    "fms_linear_cap_bf16_skinny": [_P, _P, _P, _I, _I, _I, _F, _F, _P],
    "fms_glu_bf16_skinny": [_P, _P, _P, _P, _I, _I, _I, _I, _P],
    "fms_qkv_rope_store_bf16_skinny": [_P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _I, _I, _P,
                                       _I, _I, _I, _P],
    "fms_linear_bf16_mid": [_P, _P, _P, _P, _I, _I, _I, _I, _P, _P],
    "fms_glu_bf16_mid": [_P, _P, _P, _P, _I, _I, _I, _I, _P, _P],
    "fms_qkv_rope_store_bf16_mid": [_P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _I, _I, _P,
                                    _I, _I, _I, _P],
    "fms_gemm_bf16_tc": [_P, _P, _P, _P, _I, _I, _I, _I, _P, _P],
    "fms_linear_act_bf16_tc": [_P, _P, _P, _P, _I, _I, _I, _I, _P, _P],
    "fms_glu_bf16_tc": [_P, _P, _P, _P, _I, _I, _I, _I, _P, _P],
    "fms_qkv_rope_store_bf16_tc": [_P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _I, _I, _P,
                                   _I, _I, _I, _P],
    "fms_embed_pair_hash": [_P, _P, _I, _P, _P, _P, _P, _P, _P, _P, _I, _I, _I, _L, _L, _L, _F, _I, _I, _I, _P, _P],
    "fms_normed_add_rmsnorm": [_P, _P, _I, _P, _F, _F, _P, _F, _F, _I, _P, _I, _P, _I, _I, _I, _P],
    "fms_mingru_scan": [_P, _I, _P, _P, _P, _P, _I, _I, _I, _I, _P, _P, _I, _P, _P],
    "fms_grouped_linear": [_P, _P, _P, _I, _P, _P, _P, _I, _I, _I, _I, _L, _L, _L, _L, _I, _F, _F, _I, _P],
    "fms_route": [_P, _I, _P, _I, _P, _P, _P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _P, _F, _I, _I, _P, _I, _P, _P, _P],
    "fms_route_gather": [_P, _I, _P, _P, _I, _I, _I, _P, _P, _P, _P],
    "fms_relu_squared": [_P, _I, _L, _P],
    "fms_gated_clamped": [_P, _P, _I, _I, _I, _F, _F, _P],
    "fms_latent_attention_prefill_bf16": [_P, _P, _P, _P, _L, _P, _I, _P, _I, _I, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I,
                                          _F, _I, _I, _I, _P, _I, _I, _I, _I, _P, _P, _I, _P],
    "fms_latent_gather": [_P, _I, _P, _I, _I, _P, _P, _P, _I, _P, _I, _I, _I, _P],
    "fms_attention_prefill_rows": [_P, _L, _P, _L, _P, _P, _L, _I, _L, _P, _P, _P, _P, _I, _I, _I, _F, _I, _P, _P, _L, _P, _P],
    "fms_latent_prepare": [_P, _I, _I, _P, _I, _I, _I, _P, _I, _F, _P, _I, _P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _I, _I, _I,
                           _I, _I, _P, _I, _F, _P, _I, _P],
    "fms_latent_query_norm": [_P, _I, _I, _I, _P, _I, _F, _P, _I, _P],
    "fms_latent_attention": [_P, _P, _I, _P, _P, _L, _P, _I, _P, _I, _I, _P, _P, _P, _I, _I, _P, _P, _I, _I, _I, _F, _I,
                             _I, _I, _I, _P],
    "fms_scaled_add_rmsnorm": [_P, _F, _P, _F, _P, _F, _P, _I, _F, _P, _I, _I, _I, _P],
    "fms_cast_rows": [_P, _P, _I, _L, _P],
    "fms_parts_group_rmsnorm": [_P, _P, _F, _P, _F, _P, _F, _P, _F, _P, _P, _F, _I, _P, _P, _I, _P, _I, _I, _I, _P],
    "fms_qk_prepare_store": [_P, _I, _I, _P, _P, _I, _F, _I, _F, _P, _P, _I, _I, _I, _P, _P, _P, _P, _P, _P, _P, _I, _I, _I, _I,
                             _I, _I, _I, _I, _I, _P, _I, _I, _I, _P, _I, _F, _P, _P],
    "fms_sigmoid_gate": [_P, _P, _I, _P, _I, _I, _I, _I, _I, _F, _I, _P],
    "fms_normed_add_norm": [_P, _P, _F, _P, _F, _P, _F, _P, _F, _I, _P, _F, _I, _P, _P, _F, _P, _I, _P, _I, _I, _I, _P],
    "fms_stream_mix_norm": [_P, _I, _P, _P, _P, _P, _P, _F, _P, _I, _P, _I, _I, _I, _I, _P],
    "fms_activation": [_P, _I, _I, _L, _P],
    "fms_scale_cap": [_P, _F, _F, _L, _P],
    "fms_gla_prepare": [_P, _I, _I, _I, _I, _P, _I, _P, _F, _P, _I, _P, _I, _I, _I, _F, _P],
    "fms_gla_chunked": [_P, _I, _I, _I, _I, _P, _I, _P, _F, _F, _P, _P, _I, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _I, _P, _P],
    "fms_gla_decode": [_P, _I, _I, _I, _I, _P, _I, _P, _F, _F, _P, _P, _I, _P, _F, _P, _I, _I, _I, _I, _I, _I, _P],
    "fms_linear_prepare": [_P, _I, _I, _P, _I, _I, _I, _F, _I, _P],
    "fms_exp_gates": [_P, _I, _I, _P, _F, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _P],
    "fms_chunk_scan": [_I, _P, _P, _P, _L, _P, _P, _I, _I, _P, _I, _P, _P, _P, _P, _P, _I, _L, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P,
                       _P, _I, _I, _I, _I, _I, _I, _P],
    "fms_delta_prepare": [_P, _P, _I, _I, _P, _I, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _P],
    "fms_decay_scan": [_P, _P, _I, _I, _P, _F, _P, _P, _P, _P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _I, _P],
    "fms_attention_prefill_sink": [_P, _P, _I, _P, _P, _P, _I, _I, _P, _P, _P, _P, _I, _I, _I, _I, _F, _I, _I, _I, _P, _P,
                                   _P],
    "fms_attention_prefill_masked": [_P, _P, _I, _P, _P, _P, _I, _I, _P, _P, _P, _P, _I, _I, _I, _I, _F, _I, _I, _I, _P, _P,
                                     _I, _F, _P, _L, _P],
    "fms_attention_decode_masked": [_P, _P, _I, _P, _P, _P, _I, _I, _P, _P, _P, _I, _I, _P, _P, _I, _I, _I, _F, _I, _I, _I, _L,
                                    _P, _P, _P, _I, _F, _P, _L, _P],
    "fms_attention_decode_sink": [_P, _P, _I, _P, _P, _P, _I, _I, _P, _P, _P, _I, _I, _P, _P, _I, _I, _I, _F, _I, _I, _I, _L,
                                  _P, _P, _P, _P],
    "fms_causal_conv": [_P, _I, _I, _P, _P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _I, _I, _P],
    "fms_selective_scan": [_P, _P, _I, _I, _P, _P, _P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _I, _P],
    "fms_delta_rule_scan": [_P, _P, _I, _I, _P, _I, _I, _P, _P, _P, _P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _I, _I, _P],
    "fms_gated_group_rmsnorm": [_P, _P, _I, _I, _I, _P, _I, _F, _F, _P, _I, _I, _I, _P],
    "fms_argmax": [_P, _P, _I, _I, _P],
    "fms_sample": [_P, _P, _I, _I, _F, _I, _U64, _P, _I, _P],
    "fms_attention_prefill_f32_split": [_P, _P, _P, _P, _P, _I, _I, _P, _P, _P, _P, _I, _I, _I, _I, _F, _I, _I, _I, _P, _P, _I, _L, _I, _I, _P],
    "fms_attention_prefill": [_P, _P, _I, _P, _P, _P, _I, _I, _P, _P, _P, _P, _I, _I, _I, _I, _F, _I, _I, _I, _P, _P],
    "fms_attention_decode": [_P, _P, _I, _P, _P, _P, _I, _I, _P, _P, _P, _I, _I, _P, _P, _I, _I, _I, _F, _I, _I, _I, _L, _P, _P,
                             _P],
}
_functions = {}
# kernels launched through this module since import (a decode-attention call over several splits launches two)
launches = 0


class KernelError(RuntimeError):
    pass


def _fn(library: str, name: str):
    key = (library, name)
    f = _functions.get(key)
    if f is None:
        lib = load_library(library)
        address = ctypes.cast(getattr(lib, name), ctypes.c_void_p).value
        _functions[key] = f = (load_launcher().entry(address, "".join(_SIGNATURES[name]), KernelError), lib)
    return f


def _call(library: str, name: str, *args):
    """A library's entry.  Tensors stand for their data's address; one that is on the CPU or not contiguous raises."""
    global launches
    f = _functions.get((library, name)) or _fn(library, name)
    launches += 1
    if f[0](*args) != 0:
        raise KernelError(f"{name}: {f[1].fms_last_error().decode(errors='replace')}")


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)
_device = getattr(torch._C, "_cuda_getDevice", torch.cuda.current_device)  # without a look at whether CUDA is initialised: a tensor is there


def _stream() -> int:
    """The current stream's handle (the direct getter where torch has it: a step makes some hundred launches)."""
    if _raw_stream is not None:
        return _raw_stream(_device())
    return torch.cuda.current_stream().cuda_stream


def _code(dtype: torch.dtype) -> int:
    if dtype == torch.float32:
        return F32
    if dtype == torch.bfloat16:
        return BF16
    raise KernelError(f"dtype {dtype} has no kernel: float32 and bfloat16 have")


def _ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    if t is None:
        return None
    if not t.is_cuda:
        raise KernelError("a tensor on the CPU reached a CUDA kernel; this library has no CPU path")
    if not t.is_contiguous():
        raise KernelError("a non-contiguous tensor reached a CUDA kernel")
    return t.data_ptr()


_error_flags = {}


def error_flag(device) -> torch.Tensor:
    """An int32 on the device that kernels set when they meet what the host should have prevented (a token
    id outside the vocabulary, a position without a cache block).  ``check_error_flag`` reads it."""
    flag = _error_flags.get(device)
    return _indexed(_error_flags, device, lambda d: torch.zeros(1, dtype=torch.int32, device=d)) if flag is None else flag


def _indexed(table: dict, device, make):
    """``table``'s entry of a device, which may come as a name or without an index; the keys are devices with one."""
    device = torch.device(device)
    if device.index is None:
        device = torch.device(device.type, torch.cuda.current_device())
    if device not in table:
        table[device] = make(device)
    return table[device]


_work_counters = {}
WORK_COUNTERS = 4096


def _work_counter(device) -> int:
    """The address of an int32 on the device that is 0 between launches: the persistent decode-attention kernel's warps
    draw their units from it, and the kernel that merges the splits puts it back.  Every call hands out the next of
    4,096, so that launches in flight at the same time (other streams, the launches inside captured graphs) do
    not share one."""
    entry = _work_counters.get(device)
    if entry is None:
        entry = _indexed(_work_counters, device, lambda d: [torch.zeros(WORK_COUNTERS, dtype=torch.int32, device=d), 0])
    entry[1] = at = (entry[1] + 1) % WORK_COUNTERS
    return entry[0].data_ptr() + 4 * at


def check_error_flag(device) -> None:
    """Raises if a kernel met something the host should have prevented; in a bounds-checked build
    (FMS_B200_DEBUG_BOUNDS=1) also if any kernel computed an index outside its array.  Synchronises."""
    flag = error_flag(device)
    v = int(flag.item())
    from .build import bounds_violations

    outside = bounds_violations()
    if outside:
        raise KernelError("bounds-checked build: " + "; ".join(outside))
    if v:
        flag.zero_()
        raise KernelError({1: "a token id outside the vocabulary reached the embedding",
                           2: "a token's position has no cache block",
                           4: "a kernel gave up waiting for a copy or for the tensor cores",
                           8: "decode attention was launched with fewer key splits than a sequence's length needs",
                           16: "a kernel's bounds check met an index outside its array",
                           32: "a position outside the table of learned positions reached the embedding"}.get(v, f"device error flag {v}"))


# ---- embedding ---------------------------------------------------------------------------------------
def embed(table: torch.Tensor, tokens: torch.Tensor, scale: float = 1.0) -> torch.Tensor:
    """Float32 rows of ``table`` at ``tokens``, times ``scale``: the start of the residual stream."""
    n, dim = tokens.shape[0], table.shape[1]
    out = torch.empty((n, dim), dtype=torch.float32, device=table.device)
    _call("elementwise", "fms_embed_rows", table, _code(table.dtype), tokens, out, n, dim,
          table.shape[0], float(scale), error_flag(table.device), _stream())
    return out


def embed_at(table: torch.Tensor, positions_table: torch.Tensor, batch, scale: float = 1.0) -> torch.Tensor:
    """Float32 rows ``scale`` * table[token] + positions_table[position] of a step's tokens; a row's position is
    ``batch.position_ids`` where the batch has them, else its place in the cache."""
    n, dim = batch.tokens.shape[0], table.shape[1]
    if positions_table.dtype != table.dtype or positions_table.shape[1] != dim:
        raise KernelError("embed_at: the table of positions has the token table's dtype and width")
    ids = getattr(batch, "position_ids", None)
    out = torch.empty((n, dim), dtype=torch.float32, device=table.device)
    _call("elementwise", "fms_embed_rows_at", table, _code(table.dtype), batch.tokens, out, n, dim,
          table.shape[0], float(scale), positions_table, batch.positions if ids is None else ids,
          positions_table.shape[0], error_flag(table.device), _stream())
    return out


def embed_pair_hash(table: torch.Tensor, pairs: torch.Tensor, batch, last_token: torch.Tensor, buckets: int,
                    mul_prev: int, mul_cur: int, scale: float = 1.0) -> torch.Tensor:
    """Float32 rows table[token] + pairs[(previous * mul_prev + token * mul_cur) mod buckets] (pairs[buckets] for the
    token at place 0 of its sequence), times ``scale``.  ``last_token`` [slots, 1] int32 is each sequence's last
    token so far: read for a step's first row, then set to the step's last token."""
    n, dim = batch.tokens.shape[0], table.shape[1]
    if pairs.dtype != table.dtype or pairs.shape != (buckets + 1, dim) or last_token.dtype != torch.int32:
        raise KernelError("embed_pair_hash: the pair table has the token table's dtype and buckets + 1 rows of its width; "
                          "the state is int32")
    out = torch.empty((n, dim), dtype=torch.float32, device=table.device)
    _call("elementwise", "fms_embed_pair_hash", table, pairs, _code(table.dtype), batch.tokens,
          batch.positions, batch.token_seq, batch.first_row, batch.slots, last_token,
          out, n, dim, table.shape[0], int(buckets), int(mul_prev), int(mul_cur), float(scale), 1,
          batch.slots.shape[0], last_token.shape[0], error_flag(table.device), _stream())
    return out


# ---- norm --------------------------------------------------------------------------------------------
def normed_add_rmsnorm(residual: torch.Tensor, delta: Optional[torch.Tensor], post, gain, out_dtype: torch.dtype,
                       rows: Optional[torch.Tensor] = None) -> torch.Tensor:
    """residual (float32, in place) += post_norm(delta); returns norm(residual) in ``out_dtype``.  ``post`` and ``gain``
    are (vector or None, number, eps): an RMS norm's gain as a vector of the row's width or as one number.  ``post``
    None adds delta as it is.  With ``rows`` only those rows are computed and the residual is not written."""
    dim = residual.shape[1]
    n = rows.shape[0] if rows is not None else residual.shape[0]
    if residual.dtype != torch.float32:
        raise KernelError("the residual stream is float32")
    if delta is not None and delta.dtype != out_dtype:
        raise KernelError(f"sublayer output is {delta.dtype}, compute dtype is {out_dtype}")
    post_vec, post_num, post_eps = post if post is not None else (None, 1.0, 0.0)
    gain_vec, gain_num, eps = gain
    vecs = [v for v in (post_vec, gain_vec) if v is not None]
    if len({v.dtype for v in vecs}) > 1:
        raise KernelError("normed_add_rmsnorm: the two gain vectors differ in dtype")
    out = torch.empty((n, dim), dtype=out_dtype, device=residual.device)
    _call("elementwise", "fms_normed_add_rmsnorm", residual, delta, 0 if post is None else 1, post_vec,
          float(post_num), float(post_eps), gain_vec, float(gain_num), float(eps),
          _code(vecs[0].dtype) if vecs else F32, out, _code(out_dtype), rows, n, dim, residual.shape[0],
          _stream())
    return out


NORM_NONE, NORM_RMS, NORM_LAYER = 0, 1, 2


def normed_add_norm(residual: torch.Tensor, delta, post, out_norm, out_dtype: torch.dtype,
                    rows: Optional[torch.Tensor] = None, want_out: bool = True,
                    bias: Optional[torch.Tensor] = None) -> Optional[torch.Tensor]:
    """residual (float32, in place) += post(delta); returns out_norm(residual) in ``out_dtype``.  ``post`` and
    ``out_norm`` are (mode, gain, eps) with mode ``NORM_NONE`` (the rows as they are), ``NORM_RMS`` or ``NORM_LAYER``
    (the mean taken off, the variance the mean of the squared deviations) and gain a float32 vector of the
    row's width (None with ``NORM_NONE``); ``bias`` (float32, or None) is added to the result.  ``delta`` may also be a
    list of up to four (delta, factor), whose weighted sum is added (with no ``post``).  With ``rows`` only those rows
    are computed and the residual is not written.  ``want_out`` False: only the sum is wanted and nothing is returned."""
    dim = residual.shape[1]
    n = rows.shape[0] if rows is not None else residual.shape[0]
    if residual.dtype != torch.float32:
        raise KernelError("the residual stream is float32")
    parts = list(delta) if isinstance(delta, (list, tuple)) else ([] if delta is None else [(delta, 1.0)])
    if len(parts) > 4 or any(d.dtype != out_dtype or tuple(d.shape) != tuple(residual.shape) for d, _ in parts):
        raise KernelError(f"normed_add_norm: up to four sublayer outputs of the stream's shape in the compute dtype, {out_dtype}")
    post_mode, post_gain, post_eps = post if post is not None else (NORM_NONE, None, 0.0)
    if post_mode != NORM_NONE and len(parts) > 1:
        raise KernelError("normed_add_norm: one output is normed on its way, not several")
    out_mode, gain, eps = out_norm if out_norm is not None else (NORM_NONE, None, 0.0)
    flat = []
    for i in range(4):
        flat += [_ptr(parts[i][0]), float(parts[i][1])] if i < len(parts) else [None, 0.0]
    for g in (post_gain, gain, bias):
        if g is not None and (g.dtype != torch.float32 or g.shape[0] != dim):
            raise KernelError("normed_add_norm: gains are float32 vectors of the row's width")
    out = torch.empty((n, dim), dtype=out_dtype, device=residual.device) if want_out else None
    _call("elementwise", "fms_normed_add_norm", residual, *flat, int(post_mode), post_gain, float(post_eps),
          int(out_mode), gain, bias, float(eps), out, _code(out_dtype), rows, n, dim, residual.shape[0], _stream())
    return out


def add_rmsnorm(residual: torch.Tensor, delta: Optional[torch.Tensor], gain: torch.Tensor, eps: float,
                out_dtype: torch.dtype, rows: Optional[torch.Tensor] = None) -> torch.Tensor:
    """residual (float32, in place) += delta; returns gain * rmsnorm(residual) in ``out_dtype``.  With
    ``rows`` only those rows are computed and the residual is not written."""
    dim = residual.shape[1]
    n = rows.shape[0] if rows is not None else residual.shape[0]
    if residual.dtype != torch.float32:
        raise KernelError("the residual stream is float32")
    if delta is not None and delta.dtype != out_dtype:
        raise KernelError(f"sublayer output is {delta.dtype}, compute dtype is {out_dtype}")
    out = torch.empty((n, dim), dtype=out_dtype, device=residual.device)
    _call("elementwise", "fms_add_rmsnorm", residual, delta, gain, _code(gain.dtype), float(eps),
          out, _code(out_dtype), rows, n, dim, residual.shape[0], _stream())
    return out


def scaled_add_rmsnorm(residual: torch.Tensor, alpha: float, parts, gain: torch.Tensor, eps: float,
                       out_dtype: torch.dtype) -> Optional[torch.Tensor]:
    """The norm that follows the residual sum: residual (float32, in place) = gain * rmsnorm(alpha * residual +
    sum of factor * delta over ``parts``, a list of one or two (delta, factor)).  Returns the new rows in ``out_dtype``
    too, or None where that is float32 (the stream itself then serves)."""
    n, dim = residual.shape
    if residual.dtype != torch.float32:
        raise KernelError("the residual stream is float32")
    if not 1 <= len(parts) <= 2 or any(d.dtype != out_dtype or tuple(d.shape) != (n, dim) for d, _ in parts):
        raise KernelError("scaled_add_rmsnorm: one or two sublayer outputs of the stream's shape, in the compute dtype")
    (da, sa), (db, sb) = parts[0], (parts[1] if len(parts) > 1 else (None, 0.0))
    copy = None if out_dtype == torch.float32 else torch.empty((n, dim), dtype=out_dtype, device=residual.device)
    _call("elementwise", "fms_scaled_add_rmsnorm", residual, float(alpha), da, float(sa), db, float(sb),
          gain, _code(gain.dtype), float(eps), copy, _code(out_dtype), n, dim, _stream())
    return copy


def parts_group_rmsnorm(residual: torch.Tensor, parts, gains, eps: float, groups: int, out_dtype: torch.dtype,
                        rows: Optional[torch.Tensor] = None):
    """residual (float32, in place) += sum of factor * delta over ``parts`` (up to four (delta, factor), deltas in
    ``out_dtype``); then the row in ``groups`` equal consecutive runs, each divided by its own root mean square, and
    one output per entry of ``gains`` (one or two float32 vectors of the row's width): the normed row times that gain,
    in ``out_dtype``.  Two norms of the same stream so share one pass and one set of statistics.  With ``rows`` only
    those rows are computed and the residual is not written.  Returns the list of outputs."""
    dim = residual.shape[1]
    n = rows.shape[0] if rows is not None else residual.shape[0]
    parts = [(d, float(f)) for d, f in (parts or []) if d is not None]
    if residual.dtype != torch.float32:
        raise KernelError("the residual stream is float32")
    if len(parts) > 4 or any(d.dtype != out_dtype or tuple(d.shape) != tuple(residual.shape) for d, _ in parts):
        raise KernelError("parts_group_rmsnorm: up to four sublayer outputs of the stream's shape, in the compute dtype")
    if not 1 <= len(gains) <= 2 or any(g.dtype != torch.float32 or g.shape[0] != dim for g in gains):
        raise KernelError("parts_group_rmsnorm: one or two float32 gains of the row's width")
    outs = [torch.empty((n, dim), dtype=out_dtype, device=residual.device) for _ in gains]
    flat = []
    for i in range(4):
        flat += [_ptr(parts[i][0]), parts[i][1]] if i < len(parts) else [None, 0.0]
    _call("elementwise", "fms_parts_group_rmsnorm", residual, *flat, gains[0],
          gains[1] if len(gains) > 1 else None, float(eps), int(groups), outs[0],
          outs[1] if len(outs) > 1 else None, _code(out_dtype), rows, n, dim, residual.shape[0], _stream())
    return outs


def stream_mix_norm(streams, delta: Optional[torch.Tensor], on: Optional[torch.Tensor], w_in: torch.Tensor,
                    gain: Optional[torch.Tensor], eps: float, out_dtype: torch.dtype,
                    rows: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Several residual streams X_s a token (a ``parts.streams.StreamSet``, float32).  First X_t becomes
    sum_s mix[s, t] X_s + w_out[t] * delta, in place, where there is a ``delta`` [tokens, dim] in the compute dtype
    (``on`` float32: mix [streams, streams], from and to, then w_out [streams]); then returns u / sqrt(mean(u^2) + eps) *
    gain for u = sum_s w_in[s] X_s in ``out_dtype`` (``gain`` float32 [dim]; None: u).  With ``rows`` only those tokens are
    computed and the streams are not written."""
    start, n_streams = streams.start, streams.streams
    n_all, dim = start.shape
    n = rows.shape[0] if rows is not None else n_all
    if start.dtype != torch.float32 or (delta is not None and (delta.dtype != out_dtype or tuple(delta.shape) != (n_all, dim))):
        raise KernelError(f"stream_mix_norm: the streams are float32, a sublayer's output {out_dtype} [{n_all}, {dim}]")
    if w_in.dtype != torch.float32 or w_in.shape[0] != n_streams or (gain is not None and (gain.dtype != torch.float32 or gain.shape[0] != dim)) \
            or (delta is not None and (on is None or on.dtype != torch.float32 or on.numel() != n_streams * (n_streams + 1))):
        raise KernelError(f"stream_mix_norm: float32 weights of {n_streams} streams and a gain of {dim}")
    src, src_streams = (start, 1) if streams.rows is None else (streams.rows, n_streams)
    dst = None
    if delta is not None and rows is None:
        if streams.rows is None:
            streams.rows = torch.empty((n_all, n_streams, dim), dtype=torch.float32, device=start.device)
        dst = streams.rows
    out = torch.empty((n, dim), dtype=out_dtype, device=start.device)
    _call("elementwise", "fms_stream_mix_norm", src, src_streams, dst, delta, on, w_in, gain,
          float(eps), out, _code(out_dtype), rows, n, dim, n_streams, n_all, _stream())
    return out


def cast_rows(x: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    """Float32 rows in ``dtype`` (the same tensor where that is float32)."""
    if dtype == torch.float32:
        return x
    out = torch.empty(x.shape, dtype=dtype, device=x.device)
    _call("elementwise", "fms_cast_rows", x, out, _code(dtype), x.numel(), _stream())
    return out


# ---- linear ------------------------------------------------------------------------------------------
# Tokens of a sequence from which the float32 products of its rows go to the tensor cores (gemm_f32_tc.cu: operands in three bfloat16
# parts), by the matrix' values.  The sequence's own tokens decide, and what a row gets there does not depend on the other
# rows, so that a sequence's results do not depend on what else is in the step.  CUDA cores / tensor cores in us, by rows: w of 28,672 x
# 4,096 17 240 / 183, 64 645 / 200, 256 1,260 / 335; 4,096 x 14,336 17 121 / 91, 256 700 / 165; 4,096 x 4,096 16 33 / 34, 17 43 / 36;
# 2,048 x 2,048 17 18 / 22, 33 37 / 24; 1,536 x 1,536 33 23 / 22, 257 50 / 40; 1,024 x 1,024 257 31 / 22, 2,048 111 / 54.  A step with
# sequences on both sides reads the matrix twice, so from the line on a long sequence has to gain what some short ones beside it
# lose: 257 tokens and 1 of 1,536 x 1,536 49 / 46, between eight and eight of 1 50 / 58 (33 and 1 23 / 28, 40 between eight and eight
# 23 / 42); 2,000 between four and four of 1,024 x 1,024 111 / 87 (four of 200 and four of 300 in turn 111 / 189).  Larger
# matrices: 33 and 1 of 2,048 x 2,048 37 / 30, 40 between eight and eight 37 / 48; of 28,672 x 4,096 17 and seven of 1 244 / 286, fifteen
# of 17 and one of 16 1,570 / 501.
F32_SPLIT_LINES = ((12 << 20, 17), (4 << 20, 33), (2 << 20, 257), (0, 1025))
F32_SPLIT_MOST_K = 1 << 18  # terms of a sum, whose operands of up to 2^30 are split times 2^24
F32_SPLIT_BYTES = 256 << 20  # of scratch that a product takes at a time for the parts of its rows (2,816 rows of 14,336 values)


def f32_split_tokens(weight: torch.Tensor) -> int:
    """Tokens from which a sequence's rows go to the tensor cores; 0: never."""
    n, k = weight.shape
    if min(n, k) < 1024 or k > F32_SPLIT_MOST_K:
        return 0
    return next(tokens for size, tokens in F32_SPLIT_LINES if n * k >= size)


def _linear_f32(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], sequences) -> torch.Tensor:
    m, (n, k) = x.shape[0], weight.shape
    y = torch.empty((m, n), dtype=torch.float32, device=x.device)
    batch = sequences if hasattr(sequences, "num_new") else None
    if batch is not None:
        sequences = None if batch.decode else batch.num_new or None
    least = f32_split_tokens(weight) if sequences else 0
    if not least or max(sequences) < least or sum(sequences) != m:
        _call("gemm_f32", "fms_gemm_f32", x, weight, bias, y, m, n, k, _stream())
        return y
    if min(sequences) >= least:
        _split_product(x, weight, bias, y)
        return y
    # Either side is one product over its rows, brought together where they do not lie so: one for every run of neighbours would read
    # the matrix as often as there are runs (eight sequences of 16 and eight of 17 tokens in turn, w of 28,672 x 4,096: 2,699 us; two
    # products 1,036, one on the CUDA cores 1,569).  A capture brings no new places to the device and takes the runs.
    capturing = torch.cuda.is_current_stream_capturing()
    if batch is not None:
        sides = batch.row_sides(least, capturing)
    else:
        from ..engine.batch import row_sides

        sides = row_sides(sequences, least, x.device, capturing)
    for many, first, rows, places in sides:
        if places is None:
            xs, ys = x[first:first + rows], y[first:first + rows]
        else:
            xs, ys = x.new_empty((rows, k)), y.new_empty((rows, n))
            _call("gemm_f32_tc", "fms_copy_rows_f32", x, xs, places, rows, k, m, 0, _stream())
        if many:
            _split_product(xs, weight, bias, ys)
        else:
            _call("gemm_f32", "fms_gemm_f32", xs, weight, bias, ys, rows, n, k, _stream())
        if places is not None:
            _call("gemm_f32_tc", "fms_copy_rows_f32", ys, y, places, rows, n, m, 1, _stream())
    return y


def _split_product(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], y: torch.Tensor) -> None:
    """y = x weight^T (+ bias) on the tensor cores, some rows at a time: a row's result does not depend on those beside it.  Where the
    memory does not hold the scratch for as many rows, fewer are taken at a time."""
    global launches
    m, (n, k) = x.shape[0], weight.shape
    size = (k + 63) // 64 * 64 * 6 + 1  # of a row of x in its parts
    step = max(256, F32_SPLIT_BYTES // size // 256 * 256)
    while True:
        try:
            scratch = torch.empty((min(m, step) * size + n,), dtype=torch.uint8, device=x.device)
            break
        except torch.OutOfMemoryError:
            if step <= 32:
                raise
            step = (min(m, step) // 2 + 31) // 32 * 32
    for first in range(0, m, step):
        some = min(step, m - first)
        _call("gemm_f32_tc", "fms_gemm_f32_tc", x[first:first + some], weight, bias, y[first:first + some], scratch, scratch.numel(),
              some, n, k, error_flag(x.device), _stream())
        launches += 1  # the kernel that splits the rows


def linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None,
           out_dtype: Optional[torch.dtype] = None, sequences=None) -> torch.Tensor:
    """x [rows, in] times weight [out, in] transposed (+ bias).  ``out_dtype`` defaults to x's dtype.  ``sequences``: the rows'
    ``Batch`` or how many rows each sequence has, one behind the other (a large float32 product chooses its kernel by it); None:
    every row stands alone."""
    out_dtype = out_dtype or x.dtype
    _ptr(x), _ptr(weight)
    if weight.dtype == torch.float32:
        # true float32: also taken by a float32-stored matrix inside a bfloat16 model
        x32 = x if x.dtype == torch.float32 else x.float()
        b32 = None if bias is None else (bias if bias.dtype == torch.float32 else bias.float())
        y = _linear_f32(x32, weight, b32, sequences)
        return y if out_dtype == torch.float32 else y.to(out_dtype)
    if weight.dtype != torch.bfloat16 or x.dtype != torch.bfloat16:
        raise KernelError(f"linear: x {x.dtype}, weight {weight.dtype}")
    if x.shape[0] <= SKINNY_ROWS and weight.shape[1] % 8 == 0 and (bias is None or bias.dtype == torch.bfloat16):
        # few rows (decode): the weight-streaming tensor-core kernel
        y = torch.empty((x.shape[0], weight.shape[0]), dtype=out_dtype, device=x.device)
        _call("gemm_bf16_skinny", "fms_linear_bf16_skinny", x, weight, bias, y, _code(out_dtype),
              x.shape[0], weight.shape[0], weight.shape[1], _stream())
        return y
    if _mid_fits(x, weight, bias):
        y = torch.empty((x.shape[0], weight.shape[0]), dtype=out_dtype, device=x.device)
        _call("gemm_bf16_mid", "fms_linear_bf16_mid", x, weight, bias, y, _code(out_dtype),
              x.shape[0], weight.shape[0], weight.shape[1], error_flag(x.device), _stream())
        return y
    if _tensor_core_fits(x, weight, bias):
        return linear_tensor_core(x, weight, bias, out_dtype)
    if out_dtype == torch.float32:
        y = torch.mm(x, weight.t(), out_dtype=torch.float32)
        return y if bias is None else y + bias.float()
    b = None if bias is None else bias.to(torch.bfloat16)
    return torch.nn.functional.linear(x, weight, b)


def capped_logits(x: torch.Tensor, weight: torch.Tensor, scale: float, cap: float) -> torch.Tensor:
    """Float32 logits cap * tanh(scale * x weight^T / cap) (``cap`` 0: without the cap): for a few bfloat16 rows in the
    product's epilogue, else a pass over the product's results."""
    if x.dtype == weight.dtype == torch.bfloat16 and x.shape[0] <= SKINNY_ROWS and weight.shape[1] % 8 == 0:
        y = torch.empty((x.shape[0], weight.shape[0]), dtype=torch.float32, device=x.device)
        _call("gemm_bf16_skinny", "fms_linear_cap_bf16_skinny", x, weight, y, x.shape[0], weight.shape[0],
              weight.shape[1], float(scale), float(cap), _stream())
        return y
    y = linear(x, weight, None, torch.float32)
    _call("elementwise", "fms_scale_cap", y, float(scale), float(cap), y.numel(), _stream())
    return y


# Rows from which the tcgen05 kernel with the tokens on the instruction's rows (gemm_bf16_tc.cu) is used instead of the
# library's product.  Measured through whole prefills at the 8B sizes (ms; library for everything / own gated product
# only / own for everything).  The policies taking turns in one warmed-up process: 1,100 tokens 15.4 / 16.4 / 19.6;
# 2,048 tokens 27.5 / 27.5 / 27.5; 4,096 tokens 56.0 / 54.8 / 54.9.  Each in a process of its own: 512 tokens 8.0 /
# 7.8 / 7.8; 1,024 tokens 14.8 / 12.8 / -; 1,280 tokens 17.7 / 17.6 / 19.1; 8,192 tokens 117.0 / 118.7 / 123.2.  The
# own kernel works on tiles of 256 rows, so it loses where the last tile is mostly padding (1,100 rows: a sixth is).
# So the gated product, whose activation the own kernel has in its epilogue, takes the own kernel from 512 rows on
# where at most 6% of the computed rows are padding, and everything else stays with the library unless
# FMS_B200_TC_ROWS / FMS_B200_TC_ROWS_GLU / FMS_B200_TC_MAX_PADDING say otherwise (both row limits were 1,024 once, which
# cost prompts of 1,025 to 1,800 tokens up to a quarter of their time).
TENSOR_CORE_ROWS = int(os.environ.get("FMS_B200_TC_ROWS", str(1 << 30)))
TENSOR_CORE_ROWS_GLU = int(os.environ.get("FMS_B200_TC_ROWS_GLU", "512"))
# The projection with the rotation and the cache write in the own kernel's epilogue, against the library's product and
# the rotation kernel after it, whole prefills in processes of their own (ms, fused / two kernels): 1,024 tokens 14.5 /
# 14.1; 2,048 tokens 26.5 / 26.6; 3,000 tokens 40.0 / 41.0; 4,096 tokens 53.3 / 54.3; 8,192 tokens 121.2 / 120.1.
TENSOR_CORE_ROWS_QKV = int(os.environ.get("FMS_B200_TC_ROWS_QKV", "2048"))
TENSOR_CORE_MAX_PADDING = float(os.environ.get("FMS_B200_TC_MAX_PADDING", "1.06"))  # rows computed over rows asked for
USE_TENSOR_CORE_GEMM = os.environ.get("FMS_B200_TC_GEMM", "1") != "0"


# The tcgen05 kernel with the weights on the instruction's rows (gemm_bf16_mid.cu), for SKINNY_ROWS + 1 to MID_ROWS
# rows.  By default it takes the gated feed-forward product up to 128 rows, where it is ahead of the library's
# product followed by the activation kernel (a decode step of batch 16 at the 8B sizes: 3.75 against 3.86 ms; batch 32:
# 4.59 against 4.66; batch 64: at par; batch 96: 6.80 against 6.90; batch 128: 7.89 against 7.93; batch 256: 13.70
# against 12.99, hence no further).  The plain products and the fused projection, whose matrices have too few
# rows for one block a tile and so run as clusters that add their sums, are 3 to 9 us a product behind the library
# (batch 16: 4.02 ms with them, batch 64: 6.47) and stay with it unless FMS_B200_MID_OPS names them
# ("linear,glu,qkv"; FMS_B200_MID_ROWS up to 256; FMS_B200_MID_GEMM=0 turns the kernel off).
MID_ROWS = min(256, int(os.environ.get("FMS_B200_MID_ROWS", "128")))
USE_MID_GEMM = os.environ.get("FMS_B200_MID_GEMM", "1") != "0"
MID_OPS = os.environ.get("FMS_B200_MID_OPS", "glu").split(",")


def _mid_fits(x, weight, bias, op: str = "linear") -> bool:
    return (USE_MID_GEMM and op in MID_OPS and SKINNY_ROWS < x.shape[0] <= MID_ROWS and weight.shape[1] % 8 == 0
            and x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16
            and (bias is None or bias.dtype == torch.bfloat16))


def _tensor_core_fits(x, weight, bias, rows_from: Optional[int] = None) -> bool:
    rows_from = TENSOR_CORE_ROWS if rows_from is None else rows_from
    return (USE_TENSOR_CORE_GEMM and x.shape[0] >= rows_from and weight.shape[1] % 8 == 0
            and x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16
            and (bias is None or bias.dtype == torch.bfloat16))


def linear_tensor_core(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None,
                       out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    """The product on the tcgen05 tensor cores (TMA-fed, accumulator in tensor memory): bfloat16 in, bfloat16 or
    float32 out.  K must be a multiple of 8."""
    out_dtype = out_dtype or x.dtype
    y = torch.empty((x.shape[0], weight.shape[0]), dtype=out_dtype, device=x.device)
    _call("gemm_bf16_tc", "fms_gemm_bf16_tc", x, weight, bias, y, _code(out_dtype), x.shape[0],
          weight.shape[0], weight.shape[1], error_flag(x.device), _stream())
    return y


def gated_linear_tensor_core(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor],
                             activation: int) -> torch.Tensor:
    """act(x Wg^T) * (x Wu^T) in one tcgen05 kernel: gate and up rows share a tile, the epilogue multiplies."""
    hidden = weight.shape[0] // 2
    y = torch.empty((x.shape[0], hidden), dtype=torch.bfloat16, device=x.device)
    _call("gemm_bf16_tc", "fms_glu_bf16_tc", x, weight, bias, y, x.shape[0], hidden,
          weight.shape[1], int(activation), error_flag(x.device), _stream())
    return y


SKINNY_ROWS = 8  # rows up to which the weight-streaming kernels are used (more rows re-read x too often)


# ---- feed-forward ------------------------------------------------------------------------------------
def gated_linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], activation: int,
                 sequences=None) -> torch.Tensor:
    """act(x Wg^T) * (x Wu^T) for weight = [Wg; Wu]: one kernel for few bfloat16 rows, else the product
    followed by ``gated_activation``."""
    hidden = weight.shape[0] // 2
    if (x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and x.shape[0] <= SKINNY_ROWS
            and weight.shape[1] % 8 == 0 and (bias is None or bias.dtype == torch.bfloat16)):
        _ptr(x), _ptr(weight)
        y = torch.empty((x.shape[0], hidden), dtype=torch.bfloat16, device=x.device)
        _call("gemm_bf16_skinny", "fms_glu_bf16_skinny", x, weight, bias, y, x.shape[0], hidden,
              weight.shape[1], int(activation), _stream())
        return y
    if _mid_fits(x, weight, bias, "glu"):
        _ptr(x), _ptr(weight)
        y = torch.empty((x.shape[0], hidden), dtype=torch.bfloat16, device=x.device)
        _call("gemm_bf16_mid", "fms_glu_bf16_mid", x, weight, bias, y, x.shape[0], hidden,
              weight.shape[1], int(activation), error_flag(x.device), _stream())
        return y
    # the own kernel works on tiles of 256 rows: where the last one would be mostly padding, the library is ahead
    if (_tensor_core_fits(x, weight, bias, TENSOR_CORE_ROWS_GLU)
            and (x.shape[0] + 255) // 256 * 256 <= TENSOR_CORE_MAX_PADDING * x.shape[0]):
        return gated_linear_tensor_core(x, weight, bias, activation)
    return gated_activation(linear(x, weight, bias, None, sequences), activation)


def activated_linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], activation: int,
                     sequences=None) -> torch.Tensor:
    """act(x weight^T + bias): the first product of an ungated feed-forward.  A few bfloat16 rows: the weight-streaming kernel
    with the activation in its epilogue; many, where its tiles fit (as for the gated product): the tcgen05 kernel with
    the activation in its epilogue; else the product and then the activation in place."""
    own = x.dtype == weight.dtype == torch.bfloat16 and weight.shape[1] % 8 == 0 and (bias is None or bias.dtype == torch.bfloat16) \
        and activation <= 3
    if own and x.shape[0] <= SKINNY_ROWS:
        y = x.new_empty((x.shape[0], weight.shape[0]))
        _call("gemm_bf16_skinny", "fms_linear_act_bf16_skinny", x, weight, bias, y, x.shape[0],
              weight.shape[0], weight.shape[1], int(activation), _stream())
        return y
    if (own and _tensor_core_fits(x, weight, bias, TENSOR_CORE_ROWS_GLU)
            and (x.shape[0] + 255) // 256 * 256 <= TENSOR_CORE_MAX_PADDING * x.shape[0]):
        y = x.new_empty((x.shape[0], weight.shape[0]))
        _call("gemm_bf16_tc", "fms_linear_act_bf16_tc", x, weight, bias, y, x.shape[0], weight.shape[0],
              weight.shape[1], int(activation), error_flag(x.device), _stream())
        return y
    y = linear(x, weight, bias, None, sequences)
    _call("elementwise", "fms_activation", y, _code(y.dtype), int(activation), y.numel(), _stream())
    return y


def gated_activation(gate_up: torch.Tensor, activation: int) -> torch.Tensor:
    """act(gate) * up for rows [gate | up]."""
    n, two_f = gate_up.shape
    hidden = two_f // 2
    out = gate_up.new_empty((n, hidden))
    _call("elementwise", "fms_gated_activation", gate_up, out, _code(gate_up.dtype), n, hidden,
          int(activation), _stream())
    return out


def token_gated_linear(x: torch.Tensor, weight: torch.Tensor, table: torch.Tensor, tokens: torch.Tensor,
                       activation: int) -> torch.Tensor:
    """act(x weight^T) * table[tokens]: one kernel for a few bfloat16 rows, else the product and ``token_gate``."""
    if (x.dtype == weight.dtype == table.dtype == torch.bfloat16 and x.shape[0] <= SKINNY_ROWS and weight.shape[1] % 8 == 0
            and activation <= 3 and table.shape[1] == weight.shape[0]):
        y = x.new_empty((x.shape[0], weight.shape[0]))
        _call("gemm_bf16_skinny", "fms_token_gate_bf16_skinny", x, weight, table, tokens, y,
              x.shape[0], weight.shape[0], weight.shape[1], table.shape[0], int(activation), _stream())
        return y
    return token_gate(linear(x, weight), table, tokens, activation)


def token_gate(z: torch.Tensor, table: torch.Tensor, tokens: torch.Tensor, activation: int) -> torch.Tensor:
    """act(z[t]) * table[tokens[t]]: rows of a table, one a token, gated by ``z`` [tokens, dim]."""
    n, dim = z.shape
    if table.dtype != z.dtype or table.shape[1] != dim:
        raise KernelError(f"token_gate: z {z.dtype} {tuple(z.shape)}, table {table.dtype} {tuple(table.shape)}")
    out = torch.empty_like(z)
    _call("elementwise", "fms_token_gate", z, _code(z.dtype), table, tokens, out, n, dim, table.shape[0],
          int(activation), _stream())
    return out


def joint_activation(o: torch.Tensor, proj: torch.Tensor, gate_col: int, ff_col: int, nheads: int, vdim: int, pad: int,
                     hidden: int, activation: int, gated: bool) -> torch.Tensor:
    """[tokens, nheads * vdim + hidden]: the heads' results ``o`` (heads of ``pad`` values, of which ``vdim`` count) times
    sigmoid of ``proj``'s columns from ``gate_col`` on (negative: no gate), then the feed-forward's hidden values,
    act(proj[:, ff_col:]) or, ``gated``, act of the first ``hidden`` columns times the next ``hidden``."""
    n = o.shape[0]
    if proj.dtype != o.dtype or proj.shape[0] != n or o.shape[1] != nheads * pad \
            or proj.shape[1] < max(gate_col + nheads * vdim, ff_col + hidden * (2 if gated else 1) if hidden else 0):
        raise KernelError(f"joint_activation: o {o.dtype} {tuple(o.shape)}, proj {proj.dtype} {tuple(proj.shape)}")
    out = o.new_empty((n, nheads * vdim + hidden))
    _call("elementwise", "fms_joint_activation", o, proj, proj.shape[1], int(gate_col), int(ff_col), out,
          _code(o.dtype), n, nheads, vdim, pad, hidden, int(activation), 1 if gated else 0, _stream())
    return out


# ---- attention ---------------------------------------------------------------------------------------
def rope_store(qkv: torch.Tensor, inv_freq: Optional[torch.Tensor], batch, view, nheads: int, kvheads: int,
               head_dim: int, writes_cache: bool = True) -> torch.Tensor:
    """Rotates q and k of ``qkv`` [tokens, (nheads + 2 kvheads) head_dim] by each token's position, writes k
    and v into the cache at the token's slot and place, returns the rotated q [tokens, nheads head_dim].  The
    rotation sees ``batch.position_ids`` where the batch has them (sequences that did not start at position 0),
    else the token's place in the cache, ``batch.positions``; ``inv_freq`` None rotates nothing."""
    n = qkv.shape[0]
    if view.keys.dtype != qkv.dtype:
        raise KernelError(f"cache is {view.keys.dtype}, activations are {qkv.dtype}")
    q = qkv.new_empty((n, nheads * head_dim))
    _call("elementwise", "fms_rope_store", qkv, _code(qkv.dtype), q, inv_freq, batch.positions,
          getattr(batch, "position_ids", None), batch.token_seq, batch.slots, view.keys,
          view.values, view.table,
          view.table.shape[1], view.block_tokens, n, nheads, kvheads, head_dim, 1 if writes_cache else 0,
          error_flag(qkv.device), batch.slots.shape[0], view.table.shape[0], view.keys.shape[0], _stream())
    return q


FUSE_QKV_ROPE = os.environ.get("FMS_B200_FUSE_QKV_ROPE", "1") != "0"


def rotary_table(inv_freq: torch.Tensor, batch) -> torch.Tensor:
    """[tokens, head_dim / 2, 2] float32: (sin, cos) of every token's rotation angles, made once a step and kept
    with the batch (``batch.scratch``, which the decoder empties when a step starts) for every layer that rotates by
    the same frequencies."""
    scratch = getattr(batch, "scratch", None)
    key = ("rotary_table", inv_freq.data_ptr())
    if scratch is not None and key in scratch:
        return scratch[key]
    n, half = batch.positions.shape[0], inv_freq.shape[0]
    out = torch.empty((n, half, 2), dtype=torch.float32, device=inv_freq.device)
    _call("elementwise", "fms_rotary_table", inv_freq, batch.positions, getattr(batch, "position_ids", None),
          out, n, half, _stream())
    if scratch is not None:
        scratch[key] = out
    return out


def qkv_rope_store(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], inv_freq: Optional[torch.Tensor],
                   batch, view, nheads: int, kvheads: int, head_dim: int, writes_cache: bool = True) -> torch.Tensor:
    """An attention layer's fused projection and what follows it: qkv = x weight^T (+ bias), q and k rotated by each
    token's position, k and v written into the cache, the rotated q returned.  For a few bfloat16 rows (a decode
    step) this is one kernel, the weight-streaming product with the rotation and the cache write in its epilogue;
    else the product and ``rope_store`` one after the other."""
    if (FUSE_QKV_ROPE and x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and x.shape[0] <= SKINNY_ROWS
            and weight.shape[1] % 8 == 0 and head_dim % 2 == 0 and (bias is None or bias.dtype == torch.bfloat16)
            and view.keys.dtype == torch.bfloat16 and weight.shape[0] == (nheads + 2 * kvheads) * head_dim):
        n = x.shape[0]
        q = x.new_empty((n, nheads * head_dim))
        _call("gemm_bf16_skinny", "fms_qkv_rope_store_bf16_skinny", x, weight, bias, q,
              inv_freq, batch.positions, getattr(batch, "position_ids", None), batch.token_seq,
              batch.slots, view.keys, view.values, view.table, view.table.shape[1],
              view.block_tokens, n, weight.shape[1], nheads,
              kvheads, head_dim, 1 if writes_cache else 0, error_flag(x.device), batch.slots.shape[0],
              view.table.shape[0], view.keys.shape[0], _stream())
        return q
    if (FUSE_QKV_ROPE and _mid_fits(x, weight, bias, "qkv") and head_dim % 2 == 0 and view.keys.dtype == torch.bfloat16
            and weight.shape[0] == (nheads + 2 * kvheads) * head_dim):
        n = x.shape[0]
        q = x.new_empty((n, nheads * head_dim))
        _call("gemm_bf16_mid", "fms_qkv_rope_store_bf16_mid", x, weight, bias, q, inv_freq,
              batch.positions, getattr(batch, "position_ids", None), batch.token_seq, batch.slots,
              view.keys, view.values, view.table, view.table.shape[1], view.block_tokens, n,
              weight.shape[1], nheads, kvheads, head_dim, 1 if writes_cache else 0, error_flag(x.device),
              batch.slots.shape[0], view.table.shape[0], view.keys.shape[0], _stream())
        return q
    if (FUSE_QKV_ROPE and _tensor_core_fits(x, weight, bias, TENSOR_CORE_ROWS_QKV) and head_dim % 16 == 0
            and (x.shape[0] + 255) // 256 * 256 <= TENSOR_CORE_MAX_PADDING * x.shape[0]
            and view.keys.dtype == torch.bfloat16 and weight.shape[0] == (nheads + 2 * kvheads) * head_dim):
        # many tokens: the tcgen05 product with the rotation and the cache write in its epilogue; the angles' sines and
        # cosines come from a table that the step's first such layer makes for all layers with the same frequencies
        n = x.shape[0]
        q = x.new_empty((n, nheads * head_dim))
        table = None if inv_freq is None else rotary_table(inv_freq, batch)
        _call("gemm_bf16_tc", "fms_qkv_rope_store_bf16_tc", x, weight, bias, q, table,
              batch.positions, batch.token_seq, batch.slots,
              view.keys, view.values, view.table, view.table.shape[1], view.block_tokens, n,
              weight.shape[1], nheads, kvheads, head_dim, 1 if writes_cache else 0, error_flag(x.device),
              batch.slots.shape[0], view.table.shape[0], view.keys.shape[0], _stream())
        return q
    if weight.dtype == torch.float32 and f32_split_tokens(weight):
        qkv = linear(x, weight, bias, sequences=batch)
    else:
        qkv = linear(x, weight, bias)
    return rope_store(qkv, inv_freq, batch, view, nheads, kvheads, head_dim, writes_cache)


def _attention_library(head_dim: int) -> str:
    return f"attention_hd{head_dim}"


_attn_constants = {}


def attention_constants(head_dim: int, dtype: torch.dtype, nheads: int, kvheads: int):
    """(keys per decode split, positions per prefill tile) of the library built for this head size."""
    key = (head_dim, dtype, nheads, kvheads)
    if key not in _attn_constants:
        lib = load_library(_attention_library(head_dim))
        _attn_constants[key] = (int(lib.fms_attn_split_tokens()),
                                int(lib.fms_attn_prefill_tile_positions(_code(dtype), nheads, kvheads)))
    return _attn_constants[key]


ROTARY_TABLE_ROWS = 256  # rows of a step from which ``qk_prepare_store`` reads the step's table of sines and cosines


def qk_prepare_store(proj: torch.Tensor, inv_freq: Optional[torch.Tensor], rot: int, qk_norm: bool, eps: float, batch,
                     view, nheads: int, kvheads: int, dim: int, vdim: int, pad: int,
                     writes_cache: bool = True, norm_first: bool = False, q_gain: Optional[torch.Tensor] = None,
                     k_gain: Optional[torch.Tensor] = None, halves: bool = False, values_are_keys: bool = False,
                     rot_mult: float = 1.0, q_in_place: bool = False, first_values=None, v_mix: float = 0.0) -> Optional[torch.Tensor]:
    """From rows [q: nheads x dim | k: kvheads x dim | v: kvheads x vdim | ...] of ``proj``: rotates the first ``rot``
    values of every q and k head by the row's position (adjacent pairs; with ``halves`` value i with value i + rot / 2),
    divides q and k by their root mean square over ``dim`` where ``qk_norm`` (after the rotation; with ``norm_first``
    before it, and then times ``q_gain`` / ``k_gain``, float32 [dim], where given), writes k and v into the cache (heads
    of ``pad`` values there, zeros beyond dim and vdim) and returns q [tokens, nheads * pad], padded alike.
    ``values_are_keys``: the rows have no v columns; a value is its key as projected, before norm and rotation.
    ``rot_mult`` multiplies the rotation's sines and cosines (stretched frequencies come with such a constant).
    ``q_in_place``: the queries need nothing (no rotation, no norm, no padding) and are left where they are; returns None.
    ``first_values`` (matrix, column): the values become (1 - v_mix) v + v_mix first, mixed in float32, with first the
    kvheads * vdim columns of that matrix from that column on."""
    n = proj.shape[0]
    first_ptr = first_stride = None
    if first_values is not None:
        first, col = first_values
        if first.dtype != proj.dtype or first.shape[0] != n or first.shape[1] < col + kvheads * vdim:
            raise KernelError(f"qk_prepare_store: the values to mix in are {first.dtype} {tuple(first.shape)} from column {col}")
        first_ptr, first_stride = _ptr(first) + col * first.element_size(), first.shape[1]
    if q_in_place and (rot or qk_norm or pad != dim):
        raise KernelError("qk_prepare_store: queries that are rotated, normed or padded are not left in place")
    for g in (q_gain, k_gain):
        if g is not None and (g.dtype != torch.float32 or g.shape[0] != dim):
            raise KernelError("qk_prepare_store: gains are float32 vectors of the head's size")
    if view.keys.dtype != proj.dtype or view.keys.shape[-1] != pad:
        raise KernelError(f"cache is {view.keys.dtype} with heads of {view.keys.shape[-1]}, activations are {proj.dtype}, "
                          f"heads of {pad}")
    q = None if q_in_place else proj.new_empty((n, nheads * pad))
    # many tokens: the angles' sines and cosines come from a table that all layers with the same frequencies share
    table = rotary_table(inv_freq, batch) if rot and n >= ROTARY_TABLE_ROWS and getattr(batch, "scratch", None) is not None else None
    _call("elementwise", "fms_qk_prepare_store", proj, _code(proj.dtype), proj.shape[1], q, inv_freq,
          int(rot), float(rot_mult), 1 if qk_norm else 0, float(eps), q_gain, k_gain, 1 if norm_first else 0,
          1 if halves else 0,
          1 if values_are_keys else 0, batch.positions, getattr(batch, "position_ids", None),
          batch.token_seq, batch.slots, view.keys, view.values, view.table,
          view.table.shape[1], view.block_tokens, n, nheads, kvheads, dim, vdim, pad, 1 if writes_cache else 0,
          error_flag(proj.device), batch.slots.shape[0], view.table.shape[0], view.keys.shape[0], first_ptr,
          first_stride or 0, float(v_mix), table, _stream())
    return q


def sigmoid_gate(o: torch.Tensor, gate: Optional[torch.Tensor], gate_offset: int, nheads: int, vdim: int, pad: int,
                 factor: float = 1.0, per_head: bool = False) -> torch.Tensor:
    """out[t, h, :vdim] = factor * o[t, h, :vdim] * sigmoid(gate[t, gate_offset + h * vdim + :vdim]) for o with heads
    of ``pad`` values; ``gate`` is a matrix whose columns from ``gate_offset`` on hold the gates' logits (None: no
    gate, only the padding is dropped).  ``per_head``: one gate a head, sigmoid(gate[t, gate_offset + h])."""
    n = o.shape[0]
    out = o.new_empty((n, nheads * vdim))
    gate_ptr = None if gate is None else _ptr(gate) + gate_offset * gate.element_size()
    _call("elementwise", "fms_sigmoid_gate", o, gate_ptr, 0 if gate is None else gate.shape[1], out,
          _code(o.dtype), n, nheads, vdim, pad, float(factor), 1 if per_head else 0, _stream())
    return out


# Tokens of a sequence from which its float32 prefill attention goes to the tensor cores (attention_f32_tc.cuh); its own tokens decide.
# CUDA cores / tensor cores in us, 32 heads of 128 over 8: 16 tokens onto 1,000 cached ones 97 / 119 (tiles of up to 16 rows take a
# shorter walk there), 17 onto 1,000 236 / 119, 17 alone 29 / 27, 128 alone 39 / 29, three prompts of 1,100 tokens together 207 / 95.
F32_SPLIT_ATTENTION_TOKENS = 17
_f32_split_takes = {}


def _f32_split_attention(head_dim: int, nheads: int, kvheads: int) -> bool:
    key = (head_dim, nheads, kvheads)
    if key not in _f32_split_takes:
        _f32_split_takes[key] = bool(load_library(_attention_library(head_dim)).fms_attn_f32_split_takes(nheads, kvheads))
    return _f32_split_takes[key]


def attention(q: torch.Tensor, batch, view, nheads: int, kvheads: int, head_dim: int, scale: float,
              window: int, sink: Optional[torch.Tensor] = None, chunk: int = 0, softcap: float = 0.0,
              distance: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Causal softmax attention of the step's queries over the cache (which already holds the step's own
    keys and values).  One query per sequence takes the split-key decode kernels, else the prefill kernel.
    ``sink`` [nheads] float32: a term exp(sink[h]) in every row's denominator that belongs to no key.
    ``chunk`` > 0: the positions of a sequence are cut into runs of ``chunk``, counted from its position 0, and a query
    sees the keys of its own run only (not together with a window).  ``softcap`` > 0: a score s becomes
    softcap * tanh(s / softcap) after the scale.  ``distance`` [nheads, 2] float32, pairs (r1, r2): then
    r1 * ln(1 + r2 * (query position - key position)) is taken off the score.  The queries are the first nheads *
    head_dim columns of ``q``, which may be wider."""
    wide = q.shape[1] != nheads * head_dim
    masked = bool(chunk) or bool(softcap) or distance is not None or wide
    if distance is not None and (distance.dtype != torch.float32 or tuple(distance.shape) != (nheads, 2)):
        raise KernelError("attention: the distance term is float32, two numbers a head")
    if chunk < 0 or softcap < 0 or (chunk and window):
        raise KernelError(f"attention: chunk {chunk}, window {window}, softcap {softcap}")
    if sink is not None and (sink.dtype != torch.float32 or sink.shape[0] != nheads):
        raise KernelError("attention: the sinks are float32, one per head")
    out = q.new_empty((q.shape[0], nheads * head_dim))
    lib = _attention_library(head_dim)
    split, tile_rows = attention_constants(head_dim, q.dtype, nheads, kvheads)
    common = (q, out, _code(q.dtype), view.keys, view.values, view.table,
              view.table.shape[1], view.block_tokens, batch.slots, batch.first_row, batch.len_after)
    if batch.decode:
        n_splits = (batch.max_len_after + split - 1) // split
        # a split's results [head_dim] of all, then their maxima and sums [2]
        parts = torch.empty((batch.n_seqs * nheads * n_splits * (head_dim + 2),), dtype=torch.float32, device=q.device)
        part_o = parts.data_ptr()
        part_ml = part_o + batch.n_seqs * nheads * n_splits * head_dim * 4
        # total_len (what the host knows of the sequences' lengths) chooses between the two bfloat16 decode kernels
        tail = (sink, int(chunk), float(softcap), distance, q.shape[1]) if masked else \
            (() if sink is None else (sink,))
        _call(lib, "fms_attention_decode_masked" if masked else
              ("fms_attention_decode" if sink is None else "fms_attention_decode_sink"), *common, batch.n_seqs,
              n_splits, part_o, part_ml, nheads,
              kvheads, head_dim, float(scale), int(window), view.keys.shape[0], view.table.shape[0],
              int(getattr(batch, "total_len", 0)),
              _work_counter(q.device), error_flag(q.device), *tail, _stream())
        if n_splits > 1 or q.dtype == torch.float32:
            global launches
            launches += 1  # the kernel that merges the splits
    else:
        members = None
        if q.dtype == torch.float32 and not softcap and distance is None and _f32_split_attention(head_dim, nheads, kvheads):
            long = [i for i, n in enumerate(batch.num_new) if n >= F32_SPLIT_ATTENTION_TOKENS]
            if long:
                tiles = batch.query_tiles(tile_rows, long)
                _call(lib, "fms_attention_prefill_f32_split", q, out, view.keys, view.values, view.table, view.table.shape[1], view.block_tokens,
                      batch.slots, batch.first_row, batch.len_after, tiles, tiles.shape[0], nheads, kvheads, head_dim, float(scale), int(window),
                      view.keys.shape[0], view.table.shape[0], error_flag(q.device), sink, int(chunk), q.shape[1], batch.n_seqs, q.shape[0], _stream())
                if len(long) == batch.n_seqs:
                    return out
                members = [i for i, n in enumerate(batch.num_new) if 0 < n < F32_SPLIT_ATTENTION_TOKENS]
        tiles = batch.query_tiles(tile_rows, members)
        tail = (sink, int(chunk), float(softcap), distance, q.shape[1]) if masked else \
            (() if sink is None else (sink,))
        _call(lib, "fms_attention_prefill_masked" if masked else
              ("fms_attention_prefill" if sink is None else "fms_attention_prefill_sink"), *common, tiles,
              tiles.shape[0], nheads, kvheads, head_dim, float(scale), int(window), view.keys.shape[0],
              view.table.shape[0], error_flag(q.device), *tail, _stream())
    return out


def attention_stream_launches(head_dim: int) -> int:
    """How often this process has launched (or captured) the streaming decode-attention kernel of a head size."""
    lib = load_library(f"attention_hd{head_dim}")
    lib.fms_attn_stream_launches.restype = ctypes.c_long
    return int(lib.fms_attn_stream_launches())


def decode_advance(positions: torch.Tensor, lengths: torch.Tensor, offsets: Optional[torch.Tensor] = None,
                   position_ids: Optional[torch.Tensor] = None, slots: Optional[torch.Tensor] = None,
                   spare_slot: int = -1) -> None:
    """positions[i] = lengths[i]; lengths[i] += 1 — the bookkeeping of a decode step, on the device.  With
    ``offsets`` (sequences that did not start at position 0) also position_ids[i] = positions[i] + offsets[i].
    With ``slots``: a row in ``spare_slot`` (one that only fills the step up to a captured size) restarts at
    position 0 every step."""
    _call("elementwise", "fms_decode_advance", positions, lengths, offsets, position_ids,
          slots, int(spare_slot), positions.shape[0], _stream())


# ---- recurrence --------------------------------------------------------------------------------------
_recurrent_chunk = None
SCAN_CHUNKS_FROM = 192  # tokens of a sequence in one step from which its scan runs chunk by chunk


def mingru_scan(proj: torch.Tensor, state: torch.Tensor, batch, width: int, writes_state: bool = True) -> torch.Tensor:
    """The minGRU recurrence over a step's rows.  ``proj`` [tokens, 3 width] = [z logits | u | g]; ``state``
    [slots, width] float32 is read for every sequence of the batch and, with ``writes_state``, left at its value after
    the step's last token.  Returns S_t * silu(g) [tokens, width] in proj's dtype."""
    global _recurrent_chunk
    n = proj.shape[0]
    if proj.shape[1] != 3 * width or state.dtype != torch.float32 or state.shape[1] != width:
        raise KernelError("mingru_scan: proj is [tokens, 3 width], the state float32 [slots, width]")
    y = proj.new_empty((n, width))
    chunk_rows = first_chunk = ab = None
    n_chunks = 0
    if batch.max_new >= SCAN_CHUNKS_FROM:
        if _recurrent_chunk is None:
            _recurrent_chunk = int(load_library("recurrent").fms_recurrent_chunk_tokens())
        chunk_rows, first_chunk = batch.row_chunks(_recurrent_chunk)
        n_chunks = chunk_rows.shape[0]
        ab = torch.empty((n_chunks, 2, width), dtype=torch.float32, device=proj.device)
    _call("recurrent", "fms_mingru_scan", proj, _code(proj.dtype), state, y, batch.first_row,
          batch.slots, batch.n_seqs, width, state.shape[0], 1 if writes_state else 0, chunk_rows,
          first_chunk, n_chunks, ab, _stream())
    global launches
    launches += 2 if n_chunks else 0
    return y


# ---- state matrices carried from token to token -----------------------------------------------------
def causal_conv(x: torch.Tensor, offset: int, channels: int, weight: torch.Tensor, bias: Optional[torch.Tensor],
                tail: torch.Tensor, batch, activation: bool = True, writes_state: bool = True) -> torch.Tensor:
    """A short causal convolution per channel over each sequence's rows, then silu (``activation``).  The convolved
    channels are columns ``offset .. offset + channels`` of ``x``; ``weight`` [channels, taps] float32 (its last column
    multiplies the current row), ``bias`` [channels] float32 or None; ``tail`` [slots, taps - 1, channels] float32 holds
    each sequence's last taps - 1 inputs and, with ``writes_state``, is left at those after this step.  Returns float32
    [tokens, channels]."""
    n, taps = x.shape[0], weight.shape[1]
    if weight.dtype != torch.float32 or tuple(weight.shape) != (channels, taps) or tail.dtype != torch.float32 \
            or tuple(tail.shape[1:]) != (taps - 1, channels) or (bias is not None and bias.dtype != torch.float32):
        raise KernelError("causal_conv: weight [channels, taps], bias and tail [slots, taps - 1, channels] are float32")
    out = torch.empty((n, channels), dtype=torch.float32, device=x.device)
    decode = batch.decode and n == batch.n_seqs and n <= 65535  # as many rows as sequences alone may be two of one and none of another
    _call("state_scan", "fms_causal_conv", _ptr(x) + offset * x.element_size(), _code(x.dtype), x.shape[1], weight,
          bias, tail, batch.token_seq, batch.first_row, batch.slots, out, n,
          batch.n_seqs, channels, taps, 1 if activation else 0, 1 if writes_state else 0, tail.shape[0],
          1 if decode else 0, _stream())
    global launches
    launches += 1 if writes_state and taps > 1 and not decode else 0  # the tails' kernel (a decode step's does both)
    return out


CHUNK_STATE_BYTES = 64 << 20  # states of the runs of one pass (they are read back soon: within the second-level cache)
# A sequence goes run by run through a scan under one decay a head from so many tokens of a step on: its own tokens decide, so that
# its results do not depend on what else is in the step.  Whole layers, all walk / all by runs in us, under exponential gates with a
# normalizer, fixed decays, state space with heads of 64, delta rule of 16 heads of 128: one prompt of 200 tokens 156 / 140, 125 / 137,
# 192 / 178, 140 / 160; of 256 183 / 142, 140 / 140, 219 / 179, 165 / 158; of 512 329 / 201, 240 / 183, 389 / 245, 295 / 199; of 2,048
# 1,327 / 607, 891 / 574, 1,455 / 782, 1,110 / 462; eight of 131 to 392 693 / 673, 598 / 652, 868 / 891, 566 / 468.  The walk takes a sequence's
# tokens one after the other, but many sequences fill the multiprocessors all the same, and a step that mixes both forms pays for both
# (eight of 131 to 392, those of 256 and more by runs: fixed decays 613, state space 902): so the lines lie where a mixed step seldom
# takes longer than its walk, for the kinds whose runs gain least highest.
CHUNK_SCAN_FROM = {"gated": 256, "fixed": 512, "space": 384, "delta": 256}


def chunk_scan_pays(n: int, kind: str) -> bool:
    """Whether a sequence's ``n`` tokens of a step go run by run (``fms_chunk_scan``) or token by token."""
    return n >= CHUNK_SCAN_FROM[kind]


class _Runs:
    """The sequences of a step that go run by run."""

    def __init__(self, rows: torch.Tensor, first: torch.Tensor, whole: bool) -> None:
        self.rows, self.first = rows, first  # as ``Batch.row_chunks``
        self.whole = whole  # every sequence of the step is among them


def _chunk_scan_runs(batch, dim: int, vdim: int, heads: int, key_heads: int, rows: torch.Tensor, kind: str) -> Optional[_Runs]:
    """The step's rows as runs for ``fms_chunk_scan``, or None where it takes none of them: other head sizes, rows
    that do not lie on 16 bytes, decode steps and short prompts (which go token by token), a capture that has not seen the batch
    before (the runs come from the host)."""
    if batch.decode or not batch.num_new:
        return None
    chosen = [chunk_scan_pays(n, kind) for n in batch.num_new]
    if not any(chosen):
        return None
    if _ptr(rows) & 15 or rows.shape[1] % 4 or batch.n_seqs > 65535:
        return None
    lib = load_library("chunk_scan")
    if not lib.fms_chunk_scan_takes(int(dim), int(vdim), heads // key_heads):
        return None
    chunk = int(lib.fms_chunk_scan_tokens())
    if batch.row_chunks_key(chunk, chosen) not in batch._tiles and torch.cuda.is_current_stream_capturing():
        return None
    return _Runs(*batch.row_chunks(chunk, chosen), all(chosen))


def _chunk_scan(kind: int, q: int, k: int, v: int, row: int, plan: _Runs, batch, state: torch.Tensor, o: torch.Tensor, heads: int,
                key_heads: int, dim: int, vdim: int, writes_state: bool, decay=None, gates=None, norm_in=None, norm_state=None,
                dt_raw: Optional[int] = None, dt_dtype: int = F32, dt_stride: int = 0, dt_bias=None, a_log=None, d_skip=None) -> None:
    """``fms_chunk_scan`` with its scratch; q, k, v, dt_raw: addresses."""
    global launches
    runs, first_run = plan.rows, plan.first
    n, chunk, dev = runs.shape[0], 64, state.device
    per_pass = max(1, min(n, CHUNK_STATE_BYTES // (heads * vdim * dim * 4)))
    new = lambda *shape: torch.empty(shape, dtype=torch.float32, device=dev)  # noqa: E731
    scores, states, totals = new(per_pass, key_heads, chunk, chunk), new(per_pass, heads, vdim, dim), new(per_pass, heads)
    factors, flags = new(per_pass, heads, 4, chunk), torch.empty((per_pass, heads), dtype=torch.int32, device=dev)
    norms = new(per_pass, heads, dim) if kind == 1 else None
    carry = new(2, heads, vdim, dim) if per_pass < n else None
    _call("chunk_scan", "fms_chunk_scan", kind, q, k, v, row, runs, first_run, n, per_pass, batch.slots, batch.n_seqs,
          decay, gates, norm_in, norm_state, dt_raw, dt_dtype, dt_stride, dt_bias, a_log, d_skip,
          state, carry, scores, factors, totals, states, norms, new(per_pass, heads, chunk, chunk) if kind == 3 else None, flags, o,
          heads, key_heads, dim, vdim, 1 if writes_state else 0, state.shape[0], _stream())
    launches += (4 if kind == 3 else 3) * ((n + per_pass - 1) // per_pass) - 1


def selective_scan(xbc: torch.Tensor, proj: torch.Tensor, dt_offset: int, dt_bias: torch.Tensor, a_log: torch.Tensor,
                   d_skip: torch.Tensor, state: torch.Tensor, batch, heads: int, vdim: int, n_state: int, groups: int,
                   writes_state: bool = True) -> torch.Tensor:
    """Per head, S = exp(-exp(a_log) dt) S + dt B x^T and y = S^T C + d_skip x over each sequence's rows, with
    dt = softplus(proj[:, dt_offset + head] + dt_bias).  ``xbc`` float32 [tokens, heads * vdim + 2 groups * n_state] =
    [x | B | C]; ``state`` float32 [slots, heads, vdim, n_state].  Returns y float32 [tokens, heads * vdim]."""
    n = xbc.shape[0]
    if xbc.dtype != torch.float32 or state.dtype != torch.float32 or xbc.shape[1] != heads * vdim + 2 * groups * n_state \
            or tuple(state.shape[1:]) != (heads, vdim, n_state):
        raise KernelError("selective_scan: xbc float32 [tokens, x | B | C], state float32 [slots, heads, vdim, state]")
    y = torch.empty((n, heads * vdim), dtype=torch.float32, device=xbc.device)
    plan = _chunk_scan_runs(batch, n_state, vdim, heads, groups, xbc, "space")
    if plan is not None:
        x, b = _ptr(xbc), _ptr(xbc) + heads * vdim * 4
        _chunk_scan(2, b + groups * n_state * 4, b, x, xbc.shape[1], plan, batch, state, y, heads, groups, n_state, vdim, writes_state,
                    dt_raw=_ptr(proj) + dt_offset * proj.element_size(), dt_dtype=_code(proj.dtype), dt_stride=proj.shape[1],
                    dt_bias=dt_bias, a_log=a_log, d_skip=d_skip)
        if plan.whole:
            return y
    _call("state_scan", "fms_selective_scan", xbc, _ptr(proj) + dt_offset * proj.element_size(), _code(proj.dtype),
          proj.shape[1], dt_bias, a_log, d_skip, state, y, batch.first_row, None if plan is None else plan.first,
          batch.slots, batch.n_seqs, heads, vdim, n_state, groups, 1 if writes_state else 0, state.shape[0],
          _stream())
    return y


def delta_rule_scan(qkv: torch.Tensor, proj: torch.Tensor, beta_offset: int, a_raw: Optional[torch.Tensor],
                    dt_bias: torch.Tensor, a_log: torch.Tensor, state: torch.Tensor, batch, heads: int, kvheads: int,
                    dim: int, vdim: int, writes_state: bool = True, decay_offset: Optional[int] = None) -> torch.Tensor:
    """Per head, S = diag(g) S; u = beta (v - S^T k); S += k u^T; o = S^T q over each sequence's rows.  ``qkv`` float32
    [tokens, 2 kvheads * dim + heads * vdim] = [q | k | v]; beta = sigmoid(proj[:, beta_offset + head]);
    g = exp(-exp(a_log[head]) softplus(a_raw + dt_bias)), [heads * dim] a row; ``state`` float32 [slots, heads, vdim, dim].
    q and k of ``qkv`` are made unit vectors in place on the way.  Returns o float32 [tokens, heads * vdim].
    ``decay_offset`` (with ``a_raw`` None): one decay a head instead of one a key channel (many tokens then go run by run),
    g = exp(-exp(a_log[head]) softplus(proj[:, decay_offset + head] + dt_bias[head])), dt_bias [heads]."""
    n = qkv.shape[0]
    per_head = decay_offset is not None
    if qkv.dtype != torch.float32 or state.dtype != torch.float32 or qkv.shape[1] != 2 * kvheads * dim + heads * vdim \
            or tuple(state.shape[1:]) != (heads, vdim, dim):
        raise KernelError("delta_rule_scan: qkv float32 [tokens, q | k | v], state float32 [slots, heads, vdim, dim]")
    if per_head:
        if a_raw is not None or dt_bias.shape[0] != heads or proj.shape[1] < decay_offset + heads:
            raise KernelError("delta_rule_scan: one decay a head reads its logits from proj and a bias a head")
        a_ptr, a_stride = _ptr(proj) + decay_offset * proj.element_size(), proj.shape[1]
    else:
        if tuple(a_raw.shape) != (n, heads * dim) or a_raw.dtype != proj.dtype or dt_bias.shape[0] != heads * dim:
            raise KernelError("delta_rule_scan: decays' logits [tokens, heads * dim] in the projection's dtype")
        a_ptr, a_stride = _ptr(a_raw), heads * dim
    o = torch.empty((n, heads * vdim), dtype=torch.float32, device=qkv.device)
    plan = _chunk_scan_runs(batch, dim, vdim, heads, kvheads, qkv, "delta") if per_head and vdim == 128 else None
    # decays [tokens, heads * dim] where a sequence walks, then betas and, where one goes run by run, decays [tokens, heads]
    walks = plan is None or not plan.whole
    scratch = torch.empty((n * heads * ((dim if walks else 0) + (1 if plan is None else 2)),), dtype=torch.float32, device=qkv.device)
    channels = scratch.data_ptr() if walks else None
    beta = scratch.data_ptr() + (4 * n * heads * dim if walks else 0)
    if plan is not None:
        decay = beta + 4 * n * heads
        _call("state_scan", "fms_delta_prepare", qkv, _ptr(proj) + beta_offset * proj.element_size(), _code(proj.dtype), proj.shape[1],
              a_ptr, a_stride, dt_bias, a_log, channels, decay, beta, n, heads, kvheads, dim, vdim, _stream())
        q = _ptr(qkv)
        _chunk_scan(3, q, q + kvheads * dim * 4, q + 2 * kvheads * dim * 4, qkv.shape[1], plan, batch, state, o, heads, kvheads, dim,
                    vdim, writes_state, decay=decay, gates=beta)
        if not walks:
            return o
    _call("state_scan", "fms_delta_rule_scan", qkv, _ptr(proj) + beta_offset * proj.element_size(),
          _code(proj.dtype), proj.shape[1], a_ptr, a_stride, 1 if per_head else 0, dt_bias, a_log, channels, beta, state, o,
          batch.first_row, None if plan is None else plan.first, batch.slots, n,
          batch.n_seqs, heads, kvheads, dim, vdim, 1 if writes_state else 0, state.shape[0], _stream())
    global launches
    launches += 1 if plan is None else 0  # the kernel that makes q, k, the decays and the betas ready
    return o


GLA_CHUNKS_FROM = 32  # tokens of a sequence in one step from which its scan runs chunk by chunk
_gla_chunk = None


def gla_scan(proj: torch.Tensor, state: torch.Tensor, batch, heads: int, dim: int, vdim: int, rank_offset: int,
             decay_weight: torch.Tensor, decay_bias: torch.Tensor, tau: float, q_scale: float,
             writes_state: bool = True) -> torch.Tensor:
    """A state matrix per head with one decay a token and key channel, over each sequence's rows: S = diag(a) S + k v^T;
    o = S^T (q_scale q), a = sigmoid(decay_weight u + decay_bias)^(1 / tau).  The columns of ``proj`` are [q: heads x dim |
    k: heads x dim | v: heads x vdim | ...], u its columns ``rank_offset .. rank_offset + rank``; ``decay_weight``
    [heads * dim, rank], ``decay_bias`` float32 [heads * dim]; ``state`` float32 [slots, heads, vdim, dim].  Returns o float32
    [tokens, heads * vdim].  Steps that bring ``GLA_CHUNKS_FROM`` tokens or more of a sequence run in chunks of tokens, others
    token by token."""
    global _gla_chunk, launches
    n = proj.shape[0]
    cols, channels = heads * (2 * dim + vdim), heads * dim
    rank = decay_weight.shape[1]
    if state.dtype != torch.float32 or tuple(state.shape[1:]) != (heads, vdim, dim) or proj.shape[1] < max(cols, rank_offset + rank):
        raise KernelError("gla_scan: proj [tokens, q | k | v | ... | u ...], state float32 [slots, heads, vdim, dim]")
    if decay_weight.shape[0] != channels or decay_bias.dtype != torch.float32 or decay_bias.shape[0] != channels:
        raise KernelError("gla_scan: a row of the decays' matrix and a float32 bias for every head and key channel")
    o = torch.empty((n, heads * vdim), dtype=torch.float32, device=proj.device)
    if batch.max_new >= GLA_CHUNKS_FROM:
        lib = load_library("gated_linear")
        if _gla_chunk is None:
            lib.fms_gla_record_floats.restype = ctypes.c_long
            _gla_chunk = int(lib.fms_gla_chunk_tokens())
        chunk_rows, first_chunk = batch.row_chunks(_gla_chunk)
        n_chunks = chunk_rows.shape[0]
        records = torch.empty((n_chunks * heads * int(lib.fms_gla_record_floats(dim, vdim)),), dtype=torch.float32, device=proj.device)
        _call("gated_linear", "fms_gla_chunked", proj, _code(proj.dtype), proj.shape[1], int(rank_offset), rank, decay_weight,
              _code(decay_weight.dtype), decay_bias, float(tau), float(q_scale), chunk_rows, first_chunk, n_chunks,
              records, state, o, batch.slots, n, batch.n_seqs, heads, dim, vdim, 1 if writes_state else 0,
              state.shape[0], error_flag(proj.device), _stream())
        launches += 1
        return o
    qkv = torch.empty((n, cols), dtype=torch.float32, device=proj.device)
    decay = torch.empty((n, channels), dtype=torch.float32, device=proj.device)
    _call("state_scan", "fms_gla_prepare", proj, _code(proj.dtype), proj.shape[1], int(rank_offset), rank, decay_weight,
          _code(decay_weight.dtype), decay_bias, float(tau), decay, channels, qkv, n, cols, channels,
          float(q_scale), _stream())
    _call("state_scan", "fms_decay_scan", qkv, None, _code(proj.dtype), 0, None, 0.0, decay, None, None, state,
          None, o, batch.first_row, None, batch.slots, n, batch.n_seqs, heads, dim, vdim,
          1 if writes_state else 0, state.shape[0], _stream())
    return o


def gla_read_out(proj: torch.Tensor, state: torch.Tensor, batch, heads: int, dim: int, vdim: int, rank_offset: int,
                 decay_weight: torch.Tensor, decay_bias: torch.Tensor, tau: float, q_scale: float, gate_offset: int, norm: torch.Tensor,
                 eps: float, writes_state: bool = True) -> torch.Tensor:
    """``gla_scan`` and what follows it: every head divided by its root mean square, times ``norm`` (float32 [vdim]), times
    silu of ``proj``'s columns from ``gate_offset`` on; [tokens, heads * vdim] in proj's dtype.  A decode step (one token of
    every sequence) is one kernel, else the scan and ``gated_group_rmsnorm``."""
    n = proj.shape[0]
    if batch.decode and dim % 4 == 0 and vdim <= 4096 and n == batch.n_seqs:
        rank = decay_weight.shape[1]
        if state.dtype != torch.float32 or tuple(state.shape[1:]) != (heads, vdim, dim) or norm.dtype != torch.float32 or norm.shape[0] != vdim \
                or proj.shape[1] < max(heads * (2 * dim + vdim), rank_offset + rank, gate_offset + heads * vdim) \
                or decay_weight.shape[0] != heads * dim or decay_bias.dtype != torch.float32 or decay_bias.shape[0] != heads * dim:
            raise KernelError("gla_read_out: proj [tokens, q | k | v | ...], state float32 [slots, heads, vdim, dim], norm float32 [vdim]")
        out = proj.new_empty((n, heads * vdim))
        _call("gated_linear", "fms_gla_decode", proj, _code(proj.dtype), proj.shape[1], int(rank_offset), rank, decay_weight,
              _code(decay_weight.dtype), decay_bias, float(tau), float(q_scale), state, batch.slots, int(gate_offset),
              norm, float(eps), out, n, heads, dim, vdim, 1 if writes_state else 0, state.shape[0], _stream())
        return out
    o = gla_scan(proj, state, batch, heads, dim, vdim, rank_offset, decay_weight, decay_bias, tau, q_scale, writes_state)
    return gated_group_rmsnorm(o, proj, gate_offset, GATE_SILU_AFTER, norm, eps, vdim, proj.dtype)


ACT_NONE, ACT_SILU = 0, 1


def decay_scan(proj: torch.Tensor, state: torch.Tensor, batch, heads: int, dim: int, vdim: int, activation: int = ACT_NONE,
               q_scale: float = 1.0, decay: Optional[torch.Tensor] = None, gate_offset: int = 0,
               gate_bias: Optional[torch.Tensor] = None, gate_cap: float = 0.0, norm_state: Optional[torch.Tensor] = None,
               writes_state: bool = True) -> torch.Tensor:
    """A state matrix per head under scalar decays, over each sequence's rows.  The first columns of ``proj`` are
    [q: heads x dim | k: heads x dim | v: heads x vdim]; they are taken in float32 through ``activation`` (``ACT_SILU``
    or none), q times ``q_scale``.  ``state`` float32 [slots, heads, vdim, dim].

    With ``decay`` (float32 [heads]): S = decay_h S + k v^T; o = S^T q.

    With ``gate_bias`` (float32 [2 heads]: the input gates' biases, then the forget gates'): columns ``gate_offset + h``
    and ``gate_offset + heads + h`` of ``proj`` are head h's gates before their biases, i = cap tanh((. + b) / cap),
    f = logsigmoid(cap tanh((. + b) / cap)); with the running maximum m' = max(f + m, i): S = exp(f + m - m') S +
    exp(i - m') k v^T, n likewise with k alone, o = S^T q / (max(|n.q|, exp(-m')) + 1e-6).  ``norm_state`` float32
    [slots, heads, dim + 1] holds n and then m (zeros for a new sequence).

    Returns o float32 [tokens, heads * vdim]."""
    n = proj.shape[0]
    cols = heads * (2 * dim + vdim)
    gated = gate_bias is not None
    if state.dtype != torch.float32 or tuple(state.shape[1:]) != (heads, vdim, dim) or proj.shape[1] < cols:
        raise KernelError("decay_scan: proj [tokens, q | k | v | ...], state float32 [slots, heads, vdim, dim]")
    if gated == (decay is not None):
        raise KernelError("decay_scan: either one decay a head or the gates' biases")
    if gated and (norm_state is None or norm_state.dtype != torch.float32 or tuple(norm_state.shape[1:]) != (heads, dim + 1)
                  or gate_bias.dtype != torch.float32 or gate_bias.shape[0] != 2 * heads
                  or proj.shape[1] < gate_offset + 2 * heads or norm_state.shape[0] != state.shape[0]):
        raise KernelError("decay_scan: gate biases float32 [2 heads], norm_state float32 [slots, heads, dim + 1]")
    if not gated and (decay.dtype != torch.float32 or decay.shape[0] != heads):
        raise KernelError("decay_scan: decays float32 [heads]")
    qkv = torch.empty((n, cols), dtype=torch.float32, device=proj.device)
    _call("state_scan", "fms_linear_prepare", proj, _code(proj.dtype), proj.shape[1], qkv, n, cols, heads * dim,
          float(q_scale), int(activation), _stream())
    o = torch.empty((n, heads * vdim), dtype=torch.float32, device=proj.device)
    gates = torch.empty((n, heads, 3), dtype=torch.float32, device=proj.device) if gated else None
    norm_in = torch.empty((batch.n_seqs, heads, dim), dtype=torch.float32, device=proj.device) if gated else None
    gate_ptr = _ptr(proj) + gate_offset * proj.element_size() if gated else None
    plan = _chunk_scan_runs(batch, dim, vdim, heads, heads, qkv, "gated" if gated else "fixed") if vdim == 128 else None
    if plan is not None:
        if gated:
            _call("state_scan", "fms_exp_gates", gate_ptr, _code(proj.dtype), proj.shape[1], gate_bias, float(gate_cap),
                  norm_state, norm_in, gates, batch.first_row, batch.slots, n, batch.n_seqs, heads, dim,
                  1 if writes_state else 0, state.shape[0], _stream())
        q = _ptr(qkv)
        _chunk_scan(1 if gated else 0, q, q + heads * dim * 4, q + 2 * heads * dim * 4, cols, plan, batch, state, o, heads, heads, dim, vdim,
                    writes_state, decay=decay, gates=gates, norm_in=norm_in, norm_state=norm_state)
        if plan.whole:
            return o
    _call("state_scan", "fms_decay_scan", qkv, gate_ptr, _code(proj.dtype), proj.shape[1], gate_bias,
          float(gate_cap), gates, norm_in, decay, state, norm_state, o, batch.first_row, None if plan is None else plan.first,
          batch.slots, n, batch.n_seqs, heads, dim, vdim, 1 if writes_state else 0, state.shape[0], _stream())
    global launches
    launches += 1 if gated and plan is None else 0  # the kernel that walks the gates
    return o


GATE_NONE, GATE_SILU_BEFORE, GATE_SIGMOID_AFTER, GATE_SILU_AFTER = 0, 1, 2, 3


def gated_group_rmsnorm(x: torch.Tensor, gate: Optional[torch.Tensor], gate_offset: int, gate_mode: int,
                        weight: torch.Tensor, eps: float, group_size: int, out_dtype: torch.dtype,
                        factor: float = 1.0) -> torch.Tensor:
    """Rows of ``x`` (float32) cut into groups of ``group_size``, each divided by its root mean square, times
    ``weight`` (float32; repeated along the row where it is shorter), times ``factor``.  ``gate``: a matrix whose
    columns from ``gate_offset`` on are the gates' logits: ``GATE_SILU_BEFORE`` multiplies x by silu(gate) before the
    norm, ``GATE_SIGMOID_AFTER`` the normed and weighted values by sigmoid(gate), ``GATE_SILU_AFTER`` by silu(gate)."""
    n, width = x.shape
    if x.dtype != torch.float32 or weight.dtype != torch.float32 or width % weight.shape[0]:
        raise KernelError("gated_group_rmsnorm: x and weight are float32, the weight's length divides the row's")
    if gate is not None and gate.dtype != out_dtype:
        raise KernelError(f"gated_group_rmsnorm: gate {gate.dtype}, compute dtype {out_dtype}")
    out = torch.empty((n, width), dtype=out_dtype, device=x.device)
    gate_ptr = None if gate is None else _ptr(gate) + gate_offset * gate.element_size()
    _call("state_scan", "fms_gated_group_rmsnorm", x, gate_ptr, _code(out_dtype), 0 if gate is None else gate.shape[1],
          int(gate_mode) if gate is not None else GATE_NONE, weight, weight.shape[0], float(eps), float(factor),
          out, n, width, int(group_size), _stream())
    return out


# ---- groups of rows, each with a matrix of its own ---------------------------------------------------
ROUTE_FEW_ROWS = 64  # rows of a step up to which the routing kernel makes the router's product itself
GROUPED_FEW_ROWS = 32  # rows of a step up to which the grouped products walk each group's rows (a decode step)
# FMS_B200_GROUPED_LIBRARY=0: the own float32-sum kernel for the ragged products of many bfloat16 rows too
USE_LIBRARY_GROUPED = os.environ.get("FMS_B200_GROUPED_LIBRARY", "1") != "0" and hasattr(torch.nn.functional, "grouped_mm")


def grouped_linear(x: torch.Tensor, weight: torch.Tensor, groups: int, rows: int, n_out: int, k: int, x_row_stride: int,
                   x_group_offset: int, y: torch.Tensor, y_row_stride: int, y_group_offset: int) -> torch.Tensor:
    """Uniform groups: for every group g, y[r, g * y_group_offset + :n_out] = x[r, g * x_group_offset + :k] . weight[g]^T
    for r < rows (x and y are walked by their row strides; weight [groups, n_out, k])."""
    if weight.dtype != x.dtype or y.dtype != x.dtype or tuple(weight.shape) != (groups, n_out, k):
        raise KernelError(f"grouped_linear: x {x.dtype}, weight {weight.dtype} {tuple(weight.shape)}, y {y.dtype}")
    _ptr(x), _ptr(weight), _ptr(y)
    if USE_LIBRARY_GROUPED and x.dtype == torch.bfloat16 and rows > GROUPED_FEW_ROWS:
        # many bfloat16 rows: the library's batched product over strided views of x and y (no copy of either)
        xv = torch.as_strided(x, (groups, rows, k), (x_group_offset, x_row_stride, 1), x.storage_offset())
        yv = torch.as_strided(y, (groups, rows, n_out), (y_group_offset, y_row_stride, 1), y.storage_offset())
        torch.bmm(xv, weight.transpose(1, 2), out=yv)
        return y
    if x.dtype == torch.bfloat16 and rows <= SKINNY_ROWS and k % 8 == 0 and x_row_stride % 8 == 0 and x_group_offset % 8 == 0 \
            and (_ptr(x) | _ptr(weight)) % 16 == 0 and groups <= 65535:
        # a decode step of few rows: the weight-streaming kernel, a block per group and run of its matrix's rows (8 rows, 32
        # groups of 512 x 96: 4.7 us, of 128 x 512: 3.5; the two 27 with a warp a row of the matrix)
        _call("gemm_bf16_skinny", "fms_strided_bf16_skinny", x, weight, y, rows, groups, n_out, k, x_row_stride,
              x_group_offset, y_row_stride, y_group_offset, y.numel(), _stream())
        return y
    _call("grouped", "fms_grouped_linear", x, weight, y, _code(x.dtype), None, None, None, groups, rows,
          n_out, k, x_row_stride, x_group_offset, y_row_stride, y_group_offset, 0, 0.0, 0.0,
          1 if rows <= GROUPED_FEW_ROWS else 0, _stream())
    return y


class Routing:
    """What ``route`` leaves on the device: each pair's expert and weight, the experts' row ranges in the sorted
    matrix, and the sorted, weighted rows themselves."""

    __slots__ = ("expert", "weight", "offsets", "tile_first", "row_of_pair", "group_of_row", "rows", "top", "experts",
                 "weights_on_output", "side")


ROUTE_SIGMOID, ROUTE_SOFTMAX, ROUTE_SIGMOID_GROUPS, ROUTE_SOFTMAX_CHOSEN = 0, 1, 2, 3


def route(x: torch.Tensor, router: torch.Tensor, top: int, mode: int = ROUTE_SIGMOID,
          correction: Optional[torch.Tensor] = None, route_scale: float = 1.0, groups: int = 1, keep: int = 1,
          bias: Optional[torch.Tensor] = None, side: bool = False, experts: Optional[int] = None) -> Routing:
    """``ROUTE_SIGMOID``: scores sigmoid(x router^T) in float32; every token's ``top`` best experts; rows
    weight * x[token] sorted by expert.  ``ROUTE_SOFTMAX``: scores softmax(x router^T) over all experts; the ``top``
    experts with the largest score + ``correction`` [experts] (float32, or None) are the token's; its weights are their
    scores over their sum (+ 1e-20), times ``route_scale``; the sorted rows are the tokens' as they are and
    ``route_gather`` multiplies the experts' results by the weights.  ``ROUTE_SIGMOID_GROUPS``: scores sigmoid(x
    router^T); the choice is by score + ``correction`` among the experts of the ``keep`` best of ``groups`` equal groups of
    neighbours (a group's score: the sum of its two largest choice scores); the weights are the chosen scores (without
    the correction) times ``route_scale``, and multiply the results as with ``ROUTE_SOFTMAX``.  ``ROUTE_SOFTMAX_CHOSEN``: the
    ``top`` largest logits are chosen, the weights are the softmax over those alone times ``route_scale``, and multiply the
    results.  ``bias`` [experts] float32 is added to the logits first.  ``side``: the router's matrix has a row behind the
    experts' (``experts`` says how many those are where further rows follow) and ``Routing.side`` [tokens] float32 = sigmoid(x . that row), which ``route_gather`` takes for a unit that
    every token uses."""
    experts = int(experts) if experts is not None else router.shape[0] - (1 if side else 0)
    if experts + (1 if side else 0) > router.shape[0]:
        raise KernelError(f"route: {experts} experts and {router.shape[0]} rows of the router")
    if bias is not None and (bias.dtype != torch.float32 or bias.shape[0] != experts):
        raise KernelError("route: the bias is float32, one number an expert")
    if correction is not None and (correction.dtype != torch.float32 or correction.shape[0] != experts):
        raise KernelError("route: the correction is float32, one number an expert")
    n, dim = x.shape
    dev = x.device
    r = Routing()
    r.top, r.experts = top, experts
    r.weights_on_output = mode != ROUTE_SIGMOID
    ints = torch.empty((n * top * 3 + 3 * (experts + 1),), dtype=torch.int32, device=dev)
    r.expert = ints[: n * top].view(n, top)
    r.row_of_pair = ints[n * top: 2 * n * top]
    r.group_of_row = ints[2 * n * top: 3 * n * top]
    o = 3 * n * top
    counts = ints[o: o + experts + 1]
    r.offsets = ints[o + experts + 1: o + 2 * (experts + 1)]
    r.tile_first = ints[o + 2 * (experts + 1): o + 3 * (experts + 1)]
    r.weight = torch.empty((n, top), dtype=torch.float32, device=dev)
    r.side = torch.empty((n,), dtype=torch.float32, device=dev) if side else None
    r.rows = torch.empty((n * top, dim), dtype=x.dtype, device=dev)
    # many bfloat16 rows: the logits from the library's product with float32 results (bfloat16 factors are exact in it)
    logits = None
    if x.dtype == router.dtype == torch.bfloat16 and n > ROUTE_FEW_ROWS and 8 * 4 * (2 * experts + groups) <= 48 * 1024:
        _ptr(x), _ptr(router)
        logits = torch.mm(x, router.t(), out_dtype=torch.float32)
    _call("grouped", "fms_route", x, _code(x.dtype), router, _code(router.dtype), r.expert,
          r.weight, counts, r.offsets, r.tile_first, r.row_of_pair, r.group_of_row,
          r.rows, n, dim, experts, top, int(mode), correction, float(route_scale), int(groups), int(keep),
          logits, router.shape[0], bias, r.side, _stream())
    global launches
    launches += 2
    return r


def routed_linear(rows: torch.Tensor, weight: torch.Tensor, routing: Routing, glu: bool = False, limit: float = 0.0,
                  alpha: float = 1.0, relu_squared: bool = False, silu: bool = False) -> torch.Tensor:
    """Ragged groups: y[r] = rows[r] . weight[expert of r]^T; with ``glu`` weight[e] = [gate; up] and
    y = g * sigmoid(alpha g) * (u + 1) for g = min(gate, limit), u = clamp(up, -limit, limit), or, with ``silu`` too,
    y = silu(gate) * up; with ``relu_squared`` y = max(y, 0)^2."""
    n, k = rows.shape
    n_out = weight.shape[1] // (2 if glu else 1)
    if weight.dtype != rows.dtype or weight.shape[0] != routing.experts or weight.shape[2] != k:
        raise KernelError(f"routed_linear: rows {rows.dtype} {tuple(rows.shape)}, weight {weight.dtype} {tuple(weight.shape)}")
    if (USE_LIBRARY_GROUPED and rows.dtype == torch.bfloat16 and n > max(GROUPED_FEW_ROWS, SKINNY_ROWS * routing.top)
            and k % 8 == 0 and weight.shape[1] % 8 == 0):
        # many bfloat16 rows: the library's grouped product (it takes the groups' ends from the device, as the
        # own kernels do), as the plain products of many rows take the library's; the gated unit is a kernel after it
        _ptr(rows), _ptr(weight)
        y = torch.nn.functional.grouped_mm(rows, weight.transpose(1, 2), offs=routing.offsets[1:])
        if relu_squared and not glu:
            _call("grouped", "fms_relu_squared", y, _code(y.dtype), y.numel(), _stream())
        if not glu:
            return y
        if silu:
            return gated_activation(y, 0)
        out = rows.new_empty((n, n_out))
        _call("grouped", "fms_gated_clamped", y, out, _code(y.dtype), n, n_out, float(limit), float(alpha),
              _stream())
        return out
    y = rows.new_empty((n, n_out))
    if rows.dtype == torch.bfloat16 and n <= SKINNY_ROWS * routing.top and k % 8 == 0 and (_ptr(rows) | _ptr(weight)) % 16 == 0:
        # up to eight tokens, so up to eight rows an expert: the weight-streaming kernel, a block per group and run of rows
        # (the clamped unit of eight tokens over 16 experts of 3,584: 120 us; the kernel below 236)
        _call("gemm_bf16_skinny", "fms_grouped_bf16_skinny", rows, weight, y, routing.offsets,
              routing.experts, n_out, k, (3 if silu else 1) if glu else (2 if relu_squared else 0), float(limit), float(alpha), _stream())
        return y
    _call("grouped", "fms_grouped_linear", rows, weight, y, _code(rows.dtype), routing.offsets,
          routing.tile_first, routing.group_of_row, routing.experts, n, n_out, k, k, 0, n_out, 0,
          (3 if silu else 1) if glu else (2 if relu_squared else 0), float(limit), float(alpha), 1 if n <= GROUPED_FEW_ROWS else 0, _stream())
    return y


def route_gather(ys: torch.Tensor, routing: Routing, every: Optional[torch.Tensor] = None) -> torch.Tensor:
    """out[token] = the sum of its pairs' rows of ``ys`` (each times its weight where the routing left the weights for
    the experts' results), float32, in the order of its choices; plus the token's row of ``every`` [tokens, dim], times
    ``routing.side`` where the routing has it."""
    if every is not None and (every.dtype != ys.dtype or tuple(every.shape) != (ys.shape[0] // routing.top, ys.shape[1])):
        raise KernelError(f"route_gather: rows {ys.dtype} {tuple(ys.shape)} of {routing.top} a token, beside {every.dtype} {tuple(every.shape)}")
    n = ys.shape[0] // routing.top
    out = ys.new_empty((n, ys.shape[1]))
    _call("grouped", "fms_route_gather", ys, _code(ys.dtype), routing.row_of_pair, out, n, ys.shape[1],
          routing.top, routing.weight if routing.weights_on_output else None, every,
          routing.side if every is not None else None, _stream())
    return out


# ---- attention over cached latents -------------------------------------------------------------------
_latent_split = None
# Keys of a split of the tensor-core kernel in a decode step: LATENT_SHORT_SPLIT for a row that sees up to LATENT_SHORT_UP_TO, in steps
# of more than LATENT_FEW_ROWS rows up to LATENT_SHORT_UP_TO_MANY, else 256.  A block walks its split's keys one tile after the other
# (0.15 us a key), so short splits end sooner, but each costs its partial result.  Whole layers, splits of 256 / of 64 in us: 8
# rows of 1,000 keys 111 / 62, 32 186 / 168, 64 109 / 131, 128 164 / 203; 64 of 250 85 / 72.
LATENT_SHORT_SPLIT, LATENT_SHORT_UP_TO, LATENT_SHORT_UP_TO_MANY, LATENT_FEW_ROWS = 64, 2048, 512, 32
USE_LATENT_MMA = os.environ.get("FMS_B200_LATENT_MMA", "1") != "0"  # 0: a prompt's rows through the float32 kernel too


def latent_prepare(proj: torch.Tensor, q_full: torch.Tensor, c_gain: torch.Tensor, eps: float, inv_freq: torch.Tensor,
                   rot_dims: int, batch, view, heads: int, dim: int, rot: int, rank: int, writes_cache: bool = True,
                   halves: bool = False, rot_mult: float = 1.0, kv: Optional[torch.Tensor] = None, own_space: bool = False) -> None:
    """From the fused projection [q heads (dim + rot each) | c (rank) | kr (rot) | ...] of a step's rows: norms c,
    rotates kr and every head's rot part by the row's position, writes [c | kr] into the cache at the row's place and
    the rotated query parts into q_full[:, h, rank:].  ``kv``: [c | kr] are the first columns of this matrix instead
    (queries that come from a projection of their own; ``proj`` then holds the query heads only).  ``halves``: value i
    of a rotated run turns with value i + rot_dims / 2 instead of its neighbour; ``rot_mult`` multiplies sines and cosines.
    ``own_space``: ``q_full`` is [tokens, heads, dim + rot] and takes every head's whole query, its rot part turned."""
    q_width = (dim if own_space else rank) + rot
    if q_full.numel() != proj.shape[0] * heads * q_width:
        raise KernelError(f"latent_prepare: queries {tuple(q_full.shape)} for {heads} heads of {dim} + {rot}, rank {rank}")
    if kv is not None and (kv.dtype != proj.dtype or kv.shape[0] != proj.shape[0] or kv.shape[1] < rank + rot):
        raise KernelError("latent_prepare: the latent's matrix has the projection's dtype and rows, and rank + rot columns")
    if view.keys.dtype != proj.dtype or q_full.dtype != proj.dtype:
        raise KernelError(f"cache is {view.keys.dtype}, activations are {proj.dtype}")
    _call("latent_attention", "fms_latent_prepare", proj, _code(proj.dtype), proj.shape[1], q_full,
          q_width, dim if own_space else rank, 1 if own_space else 0, c_gain, _code(c_gain.dtype), float(eps), inv_freq, int(rot_dims), batch.positions,
          getattr(batch, "position_ids", None), batch.token_seq, batch.slots, view.keys,
          view.table, view.table.shape[1], view.block_tokens, proj.shape[0], heads, dim, rot, rank,
          1 if writes_cache else 0, batch.slots.shape[0], view.table.shape[0], view.keys.shape[0],
          error_flag(proj.device), 1 if halves else 0, float(rot_mult), kv, 0 if kv is None else kv.shape[1],
          _stream())


def latent_query_norm(proj: torch.Tensor, offset: int, n: int, gain: torch.Tensor, eps: float) -> torch.Tensor:
    """Columns ``offset .. offset + n`` of ``proj``, each row divided by its root mean square over them, times ``gain``
    [n]: the query's latent on its way to the projection that makes the heads' queries of it."""
    if proj.shape[1] < offset + n or gain.shape[0] != n:
        raise KernelError("latent_query_norm: the columns lie inside the rows and the gain has their number")
    out = proj.new_empty((proj.shape[0], n))
    _call("latent_attention", "fms_latent_query_norm", _ptr(proj) + offset * proj.element_size(), _code(proj.dtype),
          proj.shape[1], n, gain, _code(gain.dtype), float(eps), out, proj.shape[0], _stream())
    return out


# Bytes that ``latent_attention_expanded`` takes at a time for gathered rows and the keys and values made of them: sequences, and
# then heads, are taken a few at a time beyond it, and a sequence whose rows with one head's keys and values are more than that stays
# in the latent's space.  Room for 8,192 rows of 32 heads of 128 at once (in two passes eight sequences of 8 tokens onto 1,024 cached
# ones each took 178 instead of 146 us a layer); in the latent's space a prompt of 2,500 tokens takes as much for its queries and results.
LATENT_EXPANDED_BYTES = 160 << 20
# What decides between the two forms of a prompt's latent attention, a sequence at a time: its own tokens and whether the step has more
# than LATENT_FEW_SEQS sequences, not what the others bring.  In the latent's space a block walks a sequence's keys at LATENT_WALK ns a
# value of a key's two products, and a (query, key) pair of a head takes LATENT_PAIR ns a value where all multiprocessors are busy;
# making a key and a value of a head takes LATENT_MAKE ns a multiply-add, once for all queries: with heads of 96 + 32 over a latent of
# 512 160, 0.02 and 0.44 ns.  So up to 8 sequences of 32 heads are made sooner than one is walked, and of more sequences those that bring
# 23 tokens or more (32 sequences of 8 tokens onto 1,000 cached ones each would take three times as long).  Whole layers, latent's space /
# heads' space in us: a prompt of 40 tokens 51 / 46, 16 tokens onto 1,024 cached ones 252 / 70, two prompts of 2,048 together
# 852 / 183, 64 tokens of eight sequences onto 8,192 230 / 146, 256 of eight 310 / 152.
LATENT_WALK, LATENT_PAIR, LATENT_MAKE = 160.0 / (2 * 512 + 32), 0.02 / (2 * 512 + 32), 0.44 / (128 * (512 + 32))
LATENT_FEW_SEQS = 8


_rows_tiles = {}


def _rows_tile(head_dim: int) -> int:
    """Positions of a tile of the prefill kernel over rows of a matrix; 0: there is none for this head size, or it is switched off."""
    if head_dim not in _rows_tiles:
        _rows_tiles[head_dim] = int(load_library(_attention_library(head_dim)).fms_attn_rows_tile_positions())
    return _rows_tiles[head_dim]


def latent_prefers_expanded(batch, n: int, seen: int, heads: int, head_dim: int, rank: int, rot: int) -> bool:
    """Whether a sequence that brings ``n`` tokens, which see ``seen`` cached rows, attends over keys and values made of the
    cached latents (``latent_attention_expanded``) rather than in the latent's space: unless their making does not pay, its rows are
    too many (LATENT_EXPANDED_BYTES), or the tensor-core kernels of either form are switched off (FMS_B200_LATENT_MMA,
    FMS_B200_ATTN_TC)."""
    if batch.decode or not USE_LATENT_MMA or not _rows_tile(head_dim) or seen * (rank + rot + 2 * head_dim) * 2 > LATENT_EXPANDED_BYTES:
        return False
    make, values = LATENT_MAKE * head_dim * (rank + rot), 2 * rank + rot
    if batch.n_seqs <= LATENT_FEW_SEQS and LATENT_FEW_SEQS * heads * make < LATENT_WALK * values:
        return True
    return n * LATENT_PAIR * values > make


def latent_expanded_members(batch, window: int, heads: int, head_dim: int, rank: int, rot: int):
    """The sequences of a step that ``latent_prefers_expanded`` sends into the heads' own space (none of a batch whose lengths the
    host does not know)."""
    if batch.decode or getattr(batch, "len_before_host", None) is None:
        return []
    return [i for i, n in enumerate(batch.num_new) if n > 0 and
            latent_prefers_expanded(batch, n, batch.rows_seen(i, window), heads, head_dim, rank, rot)]


def latent_attention_expanded(q: torch.Tensor, batch, view, expand: torch.Tensor, sink: Optional[torch.Tensor], heads: int,
                              head_dim: int, scale: float, window: int = 0, gate: Optional[torch.Tensor] = None,
                              gate_offset: int = 0, members=None, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """The same attention in the heads' own space, for steps of many tokens: the cached rows [c | kr] that the step sees
    are gathered, every head's keys and values made of them in one product, and the tcgen05 prefill kernel runs over those.
    ``q`` [tokens, heads, head_dim]; ``expand`` [heads, 2 * head_dim, rank + rot]: head h's matrix that makes [key | value] of
    a cached row; ``sink`` float32 or None; ``gate`` as in ``latent_attention``; ``members``: the sequences whose rows are made
    (default: all), the others' rows of ``out`` being left as they are.  Returns [tokens, heads * head_dim]."""
    n, width = q.shape[0], expand.shape[2]
    if tuple(expand.shape[:2]) != (heads, 2 * head_dim) or view.keys.shape[-1] != width or q.dtype != torch.bfloat16 \
            or (sink is not None and sink.dtype != torch.float32) or (gate is not None and gate.dtype != q.dtype):
        raise KernelError(f"latent_attention_expanded: {heads} heads of {head_dim}, matrices {tuple(expand.shape)}, rows of {view.keys.shape[-1]}")
    if not _rows_tile(head_dim):
        raise KernelError(f"latent_attention_expanded: no tcgen05 prefill kernel for heads of {head_dim}, or it is switched off")
    out = q.new_empty((n, heads * head_dim)) if out is None else out
    size, lib = q.element_size(), _attention_library(head_dim)
    gate_ptr = None if gate is None else _ptr(gate) + gate_offset * gate.element_size()
    for some in batch.key_passes(window, LATENT_EXPANDED_BYTES // ((width + 2 * head_dim) * size), members):
        start, first, base, rows = batch.key_rows(window, some)
        tiles = batch.query_tiles(_rows_tile(head_dim), some)
        cached = q.new_empty((rows, width))
        _call("latent_attention", "fms_latent_gather", view.keys, width * size, view.table, view.table.shape[1],
              view.block_tokens, batch.slots, start, first, batch.n_seqs, cached, rows, view.table.shape[0],
              view.keys.shape[0], _stream())
        step = max(1, min(heads, (LATENT_EXPANDED_BYTES - rows * width * size) // (rows * 2 * head_dim * size)))
        step = -(-heads // -(-heads // step))  # as many heads in the last pass as in the others, or nearly
        for h in range(0, heads, step):
            m = min(step, heads - h)
            kv = linear(cached, expand[h:h + m].view(m * 2 * head_dim, width))
            at = h * head_dim * size
            _call(lib, "fms_attention_prefill_rows", _ptr(q) + at, heads * head_dim, _ptr(out) + at, heads * head_dim, kv,
                  _ptr(kv) + head_dim * size, kv.shape[1], 2 * head_dim, rows, base, batch.first_row,
                  batch.len_after, tiles, tiles.shape[0], m, head_dim, float(scale), int(window),
                  None if sink is None else _ptr(sink) + h * 4, None if gate is None else gate_ptr + h * gate.element_size(),
                  0 if gate is None else gate.shape[1], error_flag(q.device), _stream())
            del kv  # before the next ones are made
        del cached
    return out


def latent_attention(q_full: torch.Tensor, batch, view, gate: Optional[torch.Tensor], gate_offset: int,
                     sink: Optional[torch.Tensor], heads: int, rank: int, rot: int, scale: float,
                     window: int = 0, members=None) -> torch.Tensor:
    """Causal softmax attention of the step's rows over the cached latent rows [c | kr] (which already hold the step's
    own), with a per-head sink in the denominator and a per-head sigmoid gate on the result.  ``gate``: the matrix
    whose column ``gate_offset + h`` holds head h's gate logit of each row (None: no gate); ``sink`` None: no sink;
    ``window`` > 0: the row at position p sees the keys p - window + 1 .. p only.  ``members``: the sequences whose rows are
    wanted (default: all; the others' rows may hold anything).  Returns [tokens, heads, rank]."""
    global _latent_split, launches
    n = q_full.shape[0]
    out = q_full.new_empty((n, heads, rank))
    if _latent_split is None:
        _latent_split = int(load_library("latent_attention").fms_latent_split_tokens())
    if (USE_LATENT_MMA and q_full.dtype == torch.bfloat16 and rank % 64 == 0 and rank <= 512
            and (rank + rot) % 32 == 0 and (gate is None or gate.dtype == torch.bfloat16)):
        # both products on the tensor cores, 32 rows a block: a prompt's rows as tokens x heads over all their keys; a
        # decode step's as one token's heads over one split of the keys, merged afterwards
        n_splits, part_o, part_ml, split, short = 1, None, None, _latent_split, 0
        if batch.decode:
            heads_per_block = 32
            # two at least: the merge rounds its results its own way, and the longest row must not decide for the others
            short = LATENT_SHORT_UP_TO if n <= LATENT_FEW_ROWS else LATENT_SHORT_UP_TO_MANY
            n_splits = max(2, -(-min(batch.max_len_after, short) // LATENT_SHORT_SPLIT), -(-batch.max_len_after // split))
            parts = torch.empty((n * heads * n_splits * (rank + 2),), dtype=torch.float32, device=q_full.device)
            part_o = parts.data_ptr()  # [rank] of every split, then its maxima and sums [2]
            part_ml = part_o + n * heads * n_splits * rank * 4
        else:
            heads_per_block = 1
            while heads_per_block < min(32, heads):
                heads_per_block *= 2
        tile_tokens = 32 // heads_per_block
        tiles = batch.query_tiles(tile_tokens, members)
        gate_ptr = None if gate is None else _ptr(gate) + gate_offset * gate.element_size()
        _call("latent_attention", "fms_latent_attention_prefill_bf16", q_full, out, view.keys, gate_ptr,
              0 if gate is None else gate.shape[1], sink, _code(sink.dtype) if sink is not None else F32,
              view.table, view.table.shape[1], view.block_tokens, batch.slots, batch.first_row,
              batch.positions, tiles, tiles.shape[0], tile_tokens, heads_per_block, heads, rank, rot,
              float(scale), batch.slots.shape[0], view.table.shape[0], view.keys.shape[0], batch.token_seq, n_splits, split,
              LATENT_SHORT_SPLIT, short, part_o, part_ml, int(window), _stream())
        if n_splits > 1:
            launches += 1
        return out
    n_splits, part_o, part_ml = 1, None, None
    if batch.decode:
        n_splits = max(1, (batch.max_len_after + _latent_split - 1) // _latent_split)
        if n_splits > 1:
            part_o = torch.empty((n, heads, n_splits, rank), dtype=torch.float32, device=q_full.device)
            part_ml = torch.empty((n, heads, n_splits, 2), dtype=torch.float32, device=q_full.device)
    gate_ptr = None if gate is None else _ptr(gate) + gate_offset * gate.element_size()
    _call("latent_attention", "fms_latent_attention", q_full, out, _code(q_full.dtype), view.keys, gate_ptr,
          0 if gate is None else gate.shape[1], sink, _code(sink.dtype) if sink is not None else F32,
          view.table, view.table.shape[1], view.block_tokens, batch.slots, batch.token_seq,
          batch.positions, n, n_splits, part_o, part_ml, heads, rank, rot, float(scale),
          batch.slots.shape[0], view.table.shape[0], view.keys.shape[0], int(window), _stream())
    if n_splits > 1:
        launches += 1
    return out


# ---- sampling ----------------------------------------------------------------------------------------
def argmax(logits: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    rows, vocab = logits.shape
    if logits.dtype != torch.float32:
        raise KernelError("logits are float32")
    out = out if out is not None else torch.empty((rows,), dtype=torch.int32, device=logits.device)
    _call("sampling", "fms_argmax", logits, out, rows, vocab, _stream())
    return out


def sample(logits: torch.Tensor, temperature: float, top_k: int, seed: int, requests: torch.Tensor, step: int,
           out: Optional[torch.Tensor] = None) -> torch.Tensor:
    rows, vocab = logits.shape
    if logits.dtype != torch.float32:
        raise KernelError("logits are float32")
    out = out if out is not None else torch.empty((rows,), dtype=torch.int32, device=logits.device)
    _call("sampling", "fms_sample", logits, out, rows, vocab, float(temperature), int(top_k),
          int(seed) & 0xFFFFFFFFFFFFFFFF, requests, int(step), _stream())
    return out
