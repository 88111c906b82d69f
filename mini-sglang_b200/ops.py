"""Python face of the engine's CUDA kernels.

Every function here launches hand-written sm_100a kernels from `csrc/` on the current CUDA
stream of torch and returns torch tensors.  There is no other implementation behind them: a
tensor that is not on a CUDA device, a missing compiler or an unsupported size raises.
Matrix products with more than a few rows are the one exception to "hand-written": `linear` then calls
the library GEMM that torch binds (cuBLAS), in bfloat16 with float32 accumulation or in true float32
(TF32 off), as the reference does for every projection (F.linear in mini_sglang/layers/linear.py).  Float32 products of more than a few rows and
of weights that are not small go to this engine's float32 kernel on the tensor cores.  Up to
SMALL_M_MAX rows go to this engine's weight-streaming kernels, and the gated products and output heads of larger decode batches to
its decode-batch kernel.  The reference's own kernels for the
other operations come from sgl_kernel / flash-attn (mini_sglang/layers/layernorm.py:39-50,
mini_sglang/layers/rotary_embedding.py, mini_sglang/layers/attn/fa3_attn_backend.py).
"""

from __future__ import annotations

import ctypes
import os
from typing import Optional, Sequence, Tuple

import torch

from .csrc import build as _build

_DT = {torch.float32: 0, torch.bfloat16: 1}
_ERR = {1: "element type not handled", 2: "size not supported by the kernel", 3: "kernel launch failed",
        4: "pointer not aligned"}

c_void_p, c_int, c_float, c_ll, c_ull = ctypes.c_void_p, ctypes.c_int, ctypes.c_float, ctypes.c_longlong, ctypes.c_ulonglong


class KernelError(RuntimeError):
    pass


LAUNCHES = 0      # kernels of this engine launched (or recorded into a graph) so far


def _check(code: int, what: str) -> None:
    global LAUNCHES
    LAUNCHES += 1
    if code != 0:
        detail = ""
        if code == 3:
            detail = f" ({torch.cuda.get_device_name()}: the kernels are built for sm_100a only)"
        raise KernelError(f"{what}: {_ERR.get(code, f'error {code}')}{detail}")


def _ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    if t is None:
        return None
    return t.data_ptr()


def _need_cuda(*tensors: Optional[torch.Tensor]) -> None:
    for t in tensors:
        if t is not None and not t.is_cuda:
            raise KernelError("the engine's kernels run on a CUDA device only; got a tensor on " + str(t.device))


def _stream() -> int:
    # the handle alone: the Stream object costs a microsecond a launch, which prompt steps of a few tokens wait for
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def _dt(t: torch.Tensor) -> int:
    try:
        return _DT[t.dtype]
    except KeyError:
        raise KernelError(f"dtype {t.dtype} is not handled; the engine computes in bfloat16 or float32") from None


_common = None
_attn = {}


def _lib():
    global _common
    if _common is None:
        lib = _build.common_library()
        lib.msgl_embedding.argtypes = [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_void_p]
        lib.msgl_resolve_ids.argtypes = [c_void_p, c_void_p, c_int, c_int, c_void_p]
        lib.msgl_table_delta.argtypes = [c_void_p, c_int, c_void_p, c_int, c_void_p]
        lib.msgl_decode_meta.argtypes = [c_void_p] * 4 + [c_int, c_int, c_void_p, c_int, c_int, c_int, c_int] + [c_void_p] * 9 + [c_int, c_int, c_void_p, c_void_p, c_void_p, c_int,
                                         c_void_p]
        lib.msgl_rmsnorm.argtypes = [c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_float, c_int, c_void_p,
                                     c_int, c_int, c_int, c_void_p, c_void_p]
        lib.msgl_qknorm_rope_kvwrite.argtypes = [c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_void_p, c_int,
                                                 c_float, c_void_p, c_int, c_int, c_void_p, c_void_p, c_void_p,
                                                 c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_void_p]
        lib.msgl_swiglu.argtypes = [c_void_p, c_void_p, c_int, c_int, c_int, c_void_p]
        lib.msgl_cast_from_f32.argtypes = [c_void_p, c_void_p, c_ll, c_int, c_void_p]
        lib.msgl_gemm_small_m.argtypes = [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_ll, c_ll, c_int,
                                          c_int, c_void_p, c_ll, c_void_p]
        lib.msgl_gemm_stream.argtypes = [c_void_p] * 4 + [c_int] * 3 + [c_ll, c_ll, c_int, c_int, c_void_p, c_void_p]
        lib.msgl_gemm_tc.argtypes = [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_ll, c_ll, c_int, c_void_p,
                                     c_void_p]
        lib.msgl_gemm_tc2.argtypes = lib.msgl_gemm_tc.argtypes
        lib.msgl_gemm_tc2_splitk.argtypes = [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_ll, c_ll, c_int, c_int,
                                             c_void_p, c_void_p, c_void_p]
        lib.msgl_gemm_tc2_splits.argtypes = [c_int, c_int, c_int, c_int]
        lib.msgl_gemm_tc2_splits.restype = c_int
        lib.msgl_gemm_rows.argtypes = [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_ll, c_ll, c_int, c_int, c_float, c_int,
                                       c_void_p, c_int, c_int, c_int, c_void_p, c_void_p]
        lib.msgl_gemm_rows_apart.argtypes = [c_void_p] + lib.msgl_gemm_rows.argtypes
        lib.msgl_gemm_rows_plain.argtypes = [c_void_p] * 4 + [c_int] * 3 + [c_ll, c_ll, c_int, c_void_p, c_void_p]
        lib.msgl_gemm_f32.argtypes = [c_void_p] * 4 + [c_int] * 3 + [c_ll, c_ll, c_void_p, c_void_p]
        lib.msgl_tensor_maps.argtypes = []
        lib.msgl_tensor_maps.restype = c_int
        lib.msgl_sample.argtypes = [c_void_p, c_int, c_int, c_ll, c_void_p, c_void_p, c_void_p, c_ull, c_void_p,
                                    c_void_p, c_void_p, c_void_p, c_int, c_void_p]
        _common = lib
    return _common


def _attn_lib(head_dim: int):
    hd = head_dim if head_dim in _build.MMA_HEAD_DIMS else 128
    lib = _attn.get(hd)
    if lib is None:
        lib = _build.attention_library(hd)
        lib.msgl_attention.argtypes = [c_void_p] * 10 + [c_int] * 9 + [c_float] + [c_int] * 6 + [c_void_p, c_void_p, c_int, c_void_p, c_void_p,
                                       c_ll, c_int, c_int, c_float, c_float, c_float, c_void_p]
        lib.msgl_attention_window.argtypes = [c_void_p] * 10 + [c_int] * 9 + [c_float] + [c_int] * 6 + [c_void_p, c_int, c_void_p, c_int, c_void_p]
        lib.msgl_attention_combine.argtypes = [c_void_p] * 5 + [c_int] * 5 + [c_void_p, c_void_p, c_ll, c_void_p]
        lib.msgl_attention_tc.argtypes = [c_void_p] * 7 + [c_int] * 8 + [c_float] + [c_int] * 5 + [c_void_p, c_int, c_void_p, c_int, c_void_p,
                                         c_void_p, c_ll, c_int, c_int, c_float, c_float, c_float, c_int, c_int, c_int, c_int, c_void_p, c_void_p, c_void_p, c_void_p]
        lib.msgl_attention_combine_diff.argtypes = [c_void_p] * 5 + [c_int, c_void_p] + [c_int] * 5 + [c_float, c_float, c_float, c_void_p]
        lib.msgl_attention_combine_range.argtypes = [c_void_p] * 4 + [c_int] * 9 + [c_void_p, c_void_p, c_ll, c_void_p]
        lib.msgl_attention_head_dim.restype = c_int
        if hd == 128:
            lib.msgl_attention_decode_runs.argtypes = [c_void_p] * 10 + [c_int] * 6 + [c_float, c_int, c_void_p]
        _attn[hd] = lib
    return lib


def warm_up(head_dims=()) -> None:
    """Build and load the libraries a model needs (compiles at the first call)."""
    _lib()
    for hd in head_dims:
        _attn_lib(hd)


# ---------------------------------------------------------------------------------------

def embedding(ids: torch.Tensor, table: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """ids int32 [T], table [V, H] -> float32 [T, H] (the residual stream starts in float32)."""
    _need_cuda(ids, table)
    T, (V, H) = ids.numel(), table.shape
    assert ids.dtype == torch.int32 and table.is_contiguous()
    if out is None:
        out = torch.empty((T, H), dtype=torch.float32, device=table.device)
    _check(_lib().msgl_embedding(_ptr(ids), _ptr(table), _ptr(out), T, H, V, _dt(table), _stream()), "embedding")
    return out


def resolve_ids(ids: torch.Tensor, prev: torch.Tensor) -> None:
    """In place: ids[t] = prev[-1 - ids[t]] where ids[t] < 0 (int32, on the device)."""
    _need_cuda(ids, prev)
    assert ids.dtype == torch.int32 and prev.dtype == torch.int32 and ids.is_contiguous() and prev.is_contiguous()
    _check(_lib().msgl_resolve_ids(_ptr(ids), _ptr(prev), ids.numel(), prev.numel(), _stream()), "resolve_ids")


def table_delta(deltas: torch.Tensor, n_records: int, table: torch.Tensor) -> None:
    """Rows of the device copy of a cache group's block tables, brought up to date: deltas = [n, (slot, count, offset) x n,
    page ids ...] int32 on the device; table int32 [slots, pages per request]."""
    _need_cuda(deltas, table)
    assert deltas.dtype == torch.int32 and table.dtype == torch.int32 and table.is_contiguous()
    _check(_lib().msgl_table_delta(_ptr(deltas), n_records, _ptr(table), table.shape[1], _stream()), "table_delta")


def decode_meta(ids: torch.Tensor, slots_in: torch.Tensor, pos: torch.Tensor, nsplit_in: torch.Tensor, B: int, b: int,
                table: torch.Tensor, page_size: int, mp: int, common: bool, *, input_ids, positions, token_req, q_start, kv_len,
                slots, out_loc, nsplit, block_table, order, window: int = 0, chunk: int = 0, even_in: Optional[torch.Tensor] = None,
                even_out: Optional[torch.Tensor] = None) -> None:
    """The step fields of a decode batch of B requests (captured size b) written on the device from (token id, slot,
    position) per request and the device copy of the block tables; see csrc/elementwise.cu.  `order` receives the rows
    by falling number of keys per kv split (what the attention launch walks first); `even_in` (the even cut of the step's
    keys, made by the host) is copied to `even_out` as it is."""
    _need_cuda(ids, slots_in, pos, nsplit_in, table, input_ids, block_table)
    code = _lib().msgl_decode_meta(_ptr(ids), _ptr(slots_in), _ptr(pos), _ptr(nsplit_in), B, b, _ptr(table), table.shape[1], page_size,
                                   mp, int(common), _ptr(input_ids), _ptr(positions), _ptr(token_req), _ptr(q_start), _ptr(kv_len),
                                   _ptr(slots), _ptr(out_loc), _ptr(nsplit), _ptr(block_table), int(window), int(chunk), _ptr(order),
                                   _ptr(even_in), _ptr(even_out), even_in.numel() if even_in is not None else 0, _stream())
    _check(code, "decode_meta")


def rmsnorm(weight: torch.Tensor, eps: float, *, x: Optional[torch.Tensor] = None,
            residual: Optional[torch.Tensor] = None, residual_out: Optional[torch.Tensor] = None,
            rows: Optional[torch.Tensor] = None, out_dtype: Optional[torch.dtype] = None,
            out: Optional[torch.Tensor] = None, center: bool = False, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """y = rmsnorm(residual + x) * weight, the sum and the norm in float32; with `center` the row's mean is taken off first
    (a layer norm: the variance is the mean of the squared deviations).  bias (float32 [H] or None) is added last.

    x: float32 or activation dtype [N, H] or None; residual: float32 [N, H] or None; residual_out: float32
    buffer that receives the sum (may be `residual` itself when `rows` is None);
    rows: int32 [R] picks input rows (outputs are then [R, H]).  Returns y in `out_dtype`
    (default: x's dtype)."""
    _need_cuda(weight, x, residual, residual_out, rows, bias)
    assert bias is None or (bias.dtype == torch.float32 and bias.numel() == weight.numel() and bias.is_contiguous())
    src = x if x is not None else residual
    assert src is not None and src.dim() == 2 and src.is_contiguous()
    H = src.shape[1]
    n_out = rows.numel() if rows is not None else src.shape[0]
    if out_dtype is None:
        out_dtype = x.dtype if x is not None else torch.float32
    if x is not None:
        assert x.dtype in (out_dtype, torch.float32) and x.is_contiguous()
    if residual is not None:
        assert residual.dtype == torch.float32 and residual.shape[1] == H
    assert weight.numel() == H and weight.dtype in (torch.float32, torch.bfloat16)
    if out is None:
        out = torch.empty((n_out, H), dtype=out_dtype, device=src.device)
    x_f32 = int(x is not None and x.dtype == torch.float32)
    code = _lib().msgl_rmsnorm(_ptr(x), x_f32, _ptr(residual), _ptr(residual_out), _ptr(rows), _ptr(weight),
                               int(weight.dtype == torch.float32), float(eps), int(bool(center)), _ptr(out), n_out, H, _DT[out_dtype],
                               _ptr(bias), _stream())
    _check(code, "layernorm" if center else "rmsnorm")
    return out


def qknorm_rope_kvwrite(qkv: torch.Tensor, positions: torch.Tensor, n_q: int, n_kv: int, d: int, *,
                        q_weight: Optional[torch.Tensor], k_weight: Optional[torch.Tensor], eps: float,
                        rope_table: Optional[torch.Tensor], out_loc: Optional[torch.Tensor],
                        k_cache: Optional[torch.Tensor], v_cache: Optional[torch.Tensor], page_size: int,
                        q_out: Optional[torch.Tensor] = None, interleaved: bool = False, attention_next: bool = False) -> torch.Tensor:
    """Per-head RMSNorm of q and k (if weights are given), rotary encoding from `rope_table`
    [max_pos, rot] float32 = cos | sin (if given; the first `rot` elements of a head are rotated in halves, element i
    against i + rot/2, or with `interleaved` in neighbouring pairs 2p, 2p+1), k and v written to the paged cache at token
    slots `out_loc` (if a cache is given), q returned as [T, n_q, d].  attention_next: the caller's next launch is decode attention over this step's fields, which may then set
    itself up beside this kernel and the one ahead of it."""
    _need_cuda(qkv, positions, q_weight, k_weight, rope_table, out_loc, k_cache, v_cache)
    T = qkv.shape[0]
    assert qkv.dim() == 2 and qkv.stride(1) == 1 and qkv.shape[1] == (n_q + 2 * n_kv) * d
    assert positions.numel() == T and positions.dtype == torch.int32
    if out_loc is not None:
        assert out_loc.numel() == T and out_loc.dtype == torch.int32, "one cache slot per token"
    if q_out is None:
        q_out = torch.empty((T, n_q, d), dtype=qkv.dtype, device=qkv.device)
    w_f32 = 0
    if q_weight is not None:
        assert k_weight is not None and q_weight.dtype == k_weight.dtype
        w_f32 = int(q_weight.dtype == torch.float32)
    rot, max_pos = (rope_table.shape[1], rope_table.shape[0]) if rope_table is not None else (0, 0)
    if rope_table is not None:
        assert rope_table.dtype == torch.float32 and rope_table.is_contiguous()
    if k_cache is not None:
        assert k_cache.dtype == qkv.dtype and v_cache.dtype == qkv.dtype
    code = _lib().msgl_qknorm_rope_kvwrite(_ptr(qkv), qkv.stride(0), _ptr(positions), _ptr(out_loc), _ptr(q_weight),
                                           _ptr(k_weight), w_f32, float(eps), _ptr(rope_table), rot, max_pos,
                                           _ptr(q_out), _ptr(k_cache), _ptr(v_cache), page_size, n_q, n_kv, d, T,
                                           _dt(qkv), int(bool(interleaved)), int(attention_next), _stream())
    _check(code, f"qknorm_rope_kvwrite (head size {d})")
    return q_out


def swiglu(gate_up: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """[T, 2I] (gate first) -> [T, I] = silu(gate) * up."""
    _need_cuda(gate_up)
    assert gate_up.dim() == 2 and gate_up.is_contiguous() and gate_up.shape[1] % 2 == 0
    T, I = gate_up.shape[0], gate_up.shape[1] // 2
    if out is None:
        out = torch.empty((T, I), dtype=gate_up.dtype, device=gate_up.device)
    _check(_lib().msgl_swiglu(_ptr(gate_up), _ptr(out), T, I, _dt(gate_up), _stream()), "swiglu")
    return out


def cast_from_f32(x: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    _need_cuda(x)
    assert x.dtype == torch.float32 and x.is_contiguous()
    out = torch.empty(x.shape, dtype=dtype, device=x.device)
    _check(_lib().msgl_cast_from_f32(_ptr(x), _ptr(out), x.numel(), _DT[dtype], _stream()), "cast")
    return out


_sample_scratch = {}          # per device: (part, row_max, tickets)
_sm_counts = {}


def sm_count(device) -> int:
    """Number of SMs of a CUDA device (asked once)."""
    dev = torch.device(device)
    idx = dev.index if dev.index is not None else torch.cuda.current_device()
    if idx not in _sm_counts:
        _sm_counts[idx] = int(torch.cuda.get_device_properties(idx).multi_processor_count)
    return _sm_counts[idx]



def _sample_buffers(device, rows: int, slices: int):
    """Scratch of the sampling kernels, kept per device and grown on demand.  The tickets are zero between calls:
    the block that takes a row's last ticket puts it back to zero."""
    key = (device.type, device.index if device.index is not None else torch.cuda.current_device())
    part, row_max, tickets = _sample_scratch.get(key, (None, None, None))
    if part is None or part.numel() < rows * slices * 2 or tickets.numel() < rows:
        n_rows = max(rows, 256, tickets.numel() if tickets is not None else 0)
        part = torch.empty(max(rows * slices * 2, 256 * 64 * 2), dtype=torch.float32, device=device)
        row_max = torch.empty(n_rows, dtype=torch.float32, device=device)
        tickets = torch.zeros(n_rows, dtype=torch.int32, device=device)
        _sample_scratch[key] = (part, row_max, tickets)
    return part, row_max, tickets


def sample(logits: torch.Tensor, temperatures: Optional[torch.Tensor], row_keys: Optional[torch.Tensor],
           steps: Optional[torch.Tensor], seed: int, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """float32 logits [N, V] -> int32 token ids [N]; greedy where temperature is 0."""
    _need_cuda(logits, temperatures, row_keys, steps)
    assert logits.dim() == 2 and logits.dtype == torch.float32 and logits.stride(1) == 1
    N, V = logits.shape
    if out is None:
        out = torch.empty((N,), dtype=torch.int32, device=logits.device)
    if N == 0:
        return out
    if temperatures is not None:
        assert temperatures.dtype == torch.float32 and row_keys.dtype == torch.int32 and steps.dtype == torch.int32
    # blocks per row: about four blocks an SM over all rows, but no slice below 2,048 entries
    sms = sm_count(logits.device)
    slices = max(1, min(-(-4 * sms // N), V // 2048, 64))
    part, row_max, tickets = _sample_buffers(logits.device, N, slices)
    code = _lib().msgl_sample(_ptr(logits), N, V, logits.stride(0), _ptr(temperatures), _ptr(row_keys), _ptr(steps),
                              seed & 0xFFFFFFFFFFFFFFFF, _ptr(out), _ptr(part), _ptr(row_max), _ptr(tickets), slices, _stream())
    _check(code, "sample")
    if temperatures is not None:
        global LAUNCHES
        LAUNCHES += 1            # the race is a kernel of its own
    return out


# ---------------------------------------------------------------------------------------
# attention
# ---------------------------------------------------------------------------------------
VARIANT_SIMT, VARIANT_MMA_ROWS, VARIANT_MMA_DECODE, VARIANT_TC = 0, 1, 2, 3
TC_ROWS = 128                     # query rows per block of the tcgen05 prefill kernel
USE_TC_ATTENTION = os.environ.get("MSGL_NO_TC_ATTENTION", "") == ""
_status = None                    # device int32[64]: word 0 tcgen05 attention, word 1 delta rule in chunks, word 2 tcgen05 GEMM, word 3 decode-step kernel; words 4..: debug counters
_status_host = None               # its pinned mirror, refreshed by poll_status()
_status_event = None


def _status_tensor(device) -> torch.Tensor:
    global _status, _status_host
    if _status is None:
        _status = torch.zeros(64, dtype=torch.int32, device=device)
        _status_host = torch.zeros(64, dtype=torch.int32).pin_memory()
    return _status


def _status_words(device) -> Optional[torch.Tensor]:
    """The status words, or None in a stream capture that comes before they exist: made there they would lie in the graph's memory and be cleared
    by every replay.  For calls that have another way."""
    if _status is None and torch.cuda.is_current_stream_capturing():
        return None
    return _status_tensor(device)


def poll_status() -> None:
    """Queue a copy of the kernels' status words to the host (no synchronisation).  Not inside a stream capture."""
    global _status_event
    if _status is None:
        return
    _status_host.copy_(_status, non_blocking=True)
    _status_event = torch.cuda.Event()
    _status_event.record()


def raise_if_failed(wait: bool = False) -> None:
    """Raise if a kernel with bounded waits gave up in a launch that the last finished poll_status() saw."""
    if _status_event is None:
        return
    if wait:
        _status_event.synchronize()
    elif not _status_event.query():
        return
    if int(_status_host[0]) != 0:
        raise KernelError("tcgen05 attention: a block timed out waiting for the tensor core; results are invalid")
    if int(_status_host[1]) != 0:
        raise KernelError("delta rule: a block timed out waiting for a chunk's operands; results are invalid")
    if int(_status_host[2]) != 0:
        raise KernelError("tcgen05 GEMM: a block timed out waiting for its pipeline; results are invalid")
    if int(_status_host[3]) != 0:
        raise KernelError("decode step: a block timed out at a grid barrier; results are invalid")


def tc_supported(head_dim: int, dtype: torch.dtype, group: int) -> bool:
    """The tcgen05 prefill attention kernels take bfloat16, head size 128, up to 128 query heads per kv head."""
    return USE_TC_ATTENTION and dtype == torch.bfloat16 and head_dim == 128 and 1 <= group <= TC_ROWS


def check_kernel_status() -> None:
    """Raise if a block of a kernel with bounded waits ever gave up waiting (synchronises)."""
    poll_status()
    raise_if_failed(wait=True)


TC_VERSION = int(os.environ.get("MSGL_TC_VERSION", "2"))      # 2: two query tiles per block in ping-pong (needs TMA page sizes); 1: one tile
_tc2_usable = True


def attention_tc(q: torch.Tensor, out: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, *,
                 q_start: torch.Tensor, kv_len: torch.Tensor, block_table: torch.Tensor, n_kv: int, page_size: int,
                 window: int, scale: float, qlen_min: int, qlen_max: int, q_lens: Sequence[int], keep_first: int = 0,
                 bias_log2: Optional[torch.Tensor] = None, null_log2: Optional[torch.Tensor] = None,
                 gate: Optional[torch.Tensor] = None, chunk: int = 0, diff: Optional[Tuple[float, float, float]] = None,
                 kv_lens: Optional[Sequence[int]] = None, workspace=None, beside=None) -> bool:
    """Prefill attention on tcgen05 tensor cores for the requests with q_len in [qlen_min, qlen_max];
    q_lens: the host's copy of every request's number of query tokens (to size the grid).  keep_first, bias_log2: as in
    `attention`; they are taken by the kernel on pairs of query tiles only (TMA page sizes), and the call returns False,
    having launched nothing, where that kernel cannot run.  null_log2, gate, chunk: as in `attention`, taken by both kernels;
    diff: as there, by the kernel on pairs of query tiles only.  With kv_lens (the host's copy of kv_len) and a workspace
    query tiles with far more keys than the launch's mean are cut into pieces (`plan_tc_pieces`) and merged here.
    beside: called behind the tiles' launch, ahead of the merges: for launches that run beside the tiles."""
    global _tc2_usable
    gate_stride = _attention_extras(q, null_log2, gate)
    _need_cuda(q, out, k_cache, v_cache, q_start, kv_len, block_table)
    T, n_q, d = q.shape
    B = kv_len.numel()
    assert q.is_contiguous() and out.is_contiguous() and block_table.stride(1) == 1 and q.dtype == torch.bfloat16
    assert tuple(out.shape) == (T, n_q if diff is None else n_q // 2, d) and q_start.numel() == B + 1 and block_table.shape[0] == B
    status = _status_tensor(q.device)
    group = n_q // n_kv
    whole = k_cache.is_contiguous() and v_cache.is_contiguous() and k_cache.shape == v_cache.shape
    pages = k_cache.shape[0] if whole else 0
    tma_pages = whole and page_size >= 8 and (page_size & (page_size - 1)) == 0
    versions = [2, 1] if (TC_VERSION == 2 and _tc2_usable and tma_pages) else [1]
    ext = bool(keep_first) or bias_log2 is not None or diff is not None
    if ext:
        _need_cuda(bias_log2)
        if versions[0] != 2:
            return False
        versions = [2]
        if bias_log2 is not None:
            assert bias_log2.dtype == torch.float32 and bias_log2.dim() == 2 and bias_log2.shape[0] == n_q and bias_log2.is_contiguous()
    for version in versions:
        rows = TC_ROWS * version
        qt = rows // group if group <= TC_ROWS else version
        grid_x = sum(-(-n // qt) for n in q_lens if qlen_min <= n <= qlen_max)
        cut = None
        # the plan is made in Python: two bounds on the key tiles, the cheap one first, keep it out of launches that the rule leaves whole
        if version == 2 and kv_lens is not None and workspace is not None and not (window or chunk or ext) and \
                (longest := max(kv_lens)) > 128 * (TC_PIECE_MIN + TC_PIECE_GAIN - 1) and \
                (T // qt + B) * (longest // 128 + 1) * n_kv >= (enough := TC_PIECE_MEAN * sm_count(q.device)) and \
                sum((n // qt + 1) * (kv // 128 + 1) for n, kv in zip(q_lens, kv_lens) if n >= qlen_min) * n_kv >= enough:
            cut = plan_tc_pieces(q_lens, kv_lens, qlen_min=qlen_min, qlen_max=qlen_max, tile_tokens=qt, heads=n_kv * (1 if group <= TC_ROWS else -(-group // TC_ROWS)),
                                 sms=sm_count(q.device), bytes_per_piece=T * n_q * d * 4)
        part_o = part_ml = tok_pieces = None
        lo = plane = 0
        if cut is not None:                   # rows for the tokens from the first cut one to the last, in buffers that no decode graph knows
            lo, plane = cut[2][0][0], cut[2][-1][0] + cut[2][-1][1] - cut[2][0][0]
            part_o = workspace.get("attn_piece_o", cut[1] * plane * n_q * d, torch.float32)
            part_ml = workspace.get("attn_piece_ml", cut[1] * plane * n_q * 2, torch.float32)
            tok_pieces = workspace.get("attn_tok_pieces", T, torch.int32)
        code = _attn_lib(d).msgl_attention_tc(
            _ptr(q), _ptr(out), _ptr(k_cache), _ptr(v_cache), _ptr(q_start), _ptr(kv_len), _ptr(block_table), B, T, n_q,
            n_kv, d, page_size, block_table.stride(0), window, float(scale), qlen_min, qlen_max, grid_x, pages, version,
            _ptr(status), int(keep_first), _ptr(bias_log2), bias_log2.shape[1] if bias_log2 is not None else 0, _ptr(null_log2), _ptr(gate),
            gate_stride, int(chunk), int(diff is not None), *(diff or (0.0, 0.0, 0.0)), *(cut[:2] if cut else (0, 0)), lo, plane, _ptr(part_o),
            _ptr(part_ml), _ptr(tok_pieces), _stream())
        if code == 2 and version == 2:        # no tensor maps here (driver without the encoder, unaligned cache): one-tile kernel
            _tc2_usable = False
            if ext:
                return False
            continue
        _check(code, "attention_tc")
        if beside is not None:
            beside()
        for tok0, n in cut[2] if cut is not None else ():
            _check(_attn_lib(d).msgl_attention_combine_range(_ptr(part_o), _ptr(part_ml), _ptr(tok_pieces), _ptr(out), T, lo, plane, tok0, n, n_q, d, cut[1],
                                                             _dt(out), _ptr(null_log2), _ptr(gate), gate_stride, _stream()), "attention_combine_range")
        return True
    return False


# The tcgen05 kernel walks a query tile's key tiles (128 keys) one after the other, about 2.6 us each, one block an SM.  Cutting a tile's keys
# costs some 7.5 us (three key tiles: the merge's launches and the pieces' starts) and 2.1 us a megabyte of partial results (their float32 rows out
# and in), so a launch is cut where its longest tile gets shorter by more key tiles than that, and by TC_PIECE_GAIN at least.  Fitted to
# attention layers at 8B widths, us whole / cut: 65 + 1,500 tokens behind 3,000 + 100 keys (11 tiles, 2 MB) 190 / 173; six portions of 100, three of them behind
# 4,000 (16 tiles, 15 MB) 138 / 121; 600 + 64 + 64 behind 0 + 9,000 + 9,000 (57 tiles, 17 MB) 238 / 119; 300 x 4 behind 100, 2,000, 3,000, 10 (8 tiles,
# 10 MB) 152 / 160: not cut.  Launches of fewer than TC_PIECE_MEAN key tiles an SM stay whole whatever that says: a cautious bound from when small prompt steps
# waited for the host's launches.  Cut, 64 tokens behind 8,192 take 70 us and not 189, 100 behind 3,000 64 and not 95, 700 + 65 behind 100 + 3,000
# 99 and not 124.
TC_PIECE_MIN, TC_PIECE_MEAN, TC_PIECE_GAIN, TC_PIECE_MAX, TC_PIECE_BYTES = 4, 8, 8, 8, 1 << 28
TC_PIECE_COST, TC_PIECE_TILE_BYTES = 3, 1_250_000          # key tiles that a cut launch costs, and how many bytes of partial results cost another


def plan_tc_pieces(q_lens: Sequence[int], kv_lens: Sequence[int], *, qlen_min: int, qlen_max: int, tile_tokens: int, heads: int, sms: int,
                   bytes_per_piece: int) -> Optional[Tuple[int, int, Tuple[Tuple[int, int], ...]]]:
    """(key tiles a piece, most pieces of a query tile, (first token, tokens) of every run of tokens whose tiles are cut) of a tcgen05 prefill
    launch, or None if its tiles stay whole.  A piece gets about the key tiles that every SM would have if they were dealt out
    evenly; tiles with up to 1.5 times that stay whole.  At most TC_PIECE_BYTES of partial results if all tokens were cut."""
    total, tiles, first = 0, [], 0
    for n, kv in zip(q_lens, kv_lens):
        if qlen_min <= n <= qlen_max:
            for t in range(0, n, tile_tokens):
                m = min(tile_tokens, n - t)
                k = (kv - n + t + m - 1) // 128 + 1
                total += k
                tiles.append((k, first + t, m))
        first += n
    if not tiles:
        return None
    longest, per = max(t[0] for t in tiles), max(TC_PIECE_MIN, -(-total * heads // sms))
    pieces = min(-(-longest // per), TC_PIECE_MAX, TC_PIECE_BYTES // max(bytes_per_piece, 1))
    if total * heads < TC_PIECE_MEAN * sms or 2 * longest <= 3 * per or pieces < 2:
        return None
    runs, cut, whole = [], 0, 0
    for k, at, m in tiles:                  # the rule of the kernel: a tile is cut if it has more than 1.5 times `per`
        if 2 * k > 3 * per:
            cut += m
            if runs and runs[-1][0] + runs[-1][1] == at:
                runs[-1][1] += m
            else:
                runs.append([at, m])
        else:
            whole = max(whole, k)
    saved = longest - max(-(-longest // pieces), per, whole)
    if saved < TC_PIECE_GAIN or saved < TC_PIECE_COST + bytes_per_piece * pieces * cut / first / TC_PIECE_TILE_BYTES:
        return None
    return per, pieces, tuple((a, m) for a, m in runs)


def attention_tile_tokens(variant: int, group: int, head_dim: int = 128) -> int:
    """Tokens per query tile of a kernel variant for a given group size (q heads per kv head)."""
    if variant == VARIANT_MMA_DECODE:
        lib = _attn_lib(head_dim)
        lib.msgl_attention_decode_tile_tokens.restype = c_int
        return int(lib.msgl_attention_decode_tile_tokens(int(group)))
    rows = {VARIANT_MMA_ROWS: 64, VARIANT_TC: TC_ROWS}.get(variant, 16)
    return rows // group if group <= rows else 1


def decode_blocks_per_sm(head_dim: int, dtype: torch.dtype, group: int = 1) -> int:
    """Blocks of the decode attention kernel that fit one SM (used to choose the kv splits)."""
    if not mma_supported(head_dim, dtype):
        return 4
    lib = _attn_lib(head_dim)
    lib.msgl_attention_decode_blocks_per_sm.restype = c_int
    return int(lib.msgl_attention_decode_blocks_per_sm(int(group)))


def even_cut_size(B: int, n_blocks: int) -> int:
    """int32 words of the even cut of a decode step of B requests over n_blocks blocks per kv head: blocks in use, start
    unit of every block [n_blocks + 1], first request of every block [n_blocks], first unit of every request [B + 1], first
    block of every request [B]."""
    return 1 + (n_blocks + 1) + n_blocks + (B + 1) + B


def decode_even_ok(head_dim: int, dtype: torch.dtype, group: int = 1) -> bool:
    """Whether the decode attention launch for this head size takes an even cut of the keys (`attention(even=...)`)."""
    if not mma_supported(head_dim, dtype):
        return False
    lib = _attn_lib(head_dim)
    lib.msgl_attention_decode_even_ok.restype = c_int
    return bool(lib.msgl_attention_decode_even_ok(int(group)))


def window_bias_supported(head_dim: int, dtype: torch.dtype, group: int) -> bool:
    """Whether `attention(keep_first=..., bias_log2=...)` takes this geometry: bfloat16, head sizes in steps of 32 (the mma
    prefill kernel and the transposed decode kernel), up to 16 query heads a kv head."""
    return mma_supported(head_dim, dtype) and head_dim % 32 == 0 and group <= 16


def mma_supported(head_dim: int, dtype: torch.dtype) -> bool:
    return dtype == torch.bfloat16 and head_dim in _build.MMA_HEAD_DIMS


def _attention_extras(q: torch.Tensor, null_log2: Optional[torch.Tensor], gate: Optional[torch.Tensor]) -> int:
    """Checks the term without a key and the output gate of an attention launch -> the gate's row stride."""
    _need_cuda(null_log2, gate)
    T, n_q, d = q.shape
    if null_log2 is not None:
        assert null_log2.dtype == torch.float32 and null_log2.numel() == n_q and null_log2.is_contiguous()
    if gate is None:
        return 0
    assert gate.dtype == q.dtype and gate.shape[0] == T
    return _rows_view(gate, n_q * d, "gate")


def attention(q: torch.Tensor, out: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, *,
              q_start: torch.Tensor, kv_len: torch.Tensor, block_table: torch.Tensor,
              nsplit: Optional[torch.Tensor], part_o: Optional[torch.Tensor], part_ml: Optional[torch.Tensor],
              n_kv: int, page_size: int, window: int, max_split: int, scale: float, qlen_min: int, qlen_max: int,
              uniform_decode: bool, variant: int, grid_x: int, order: Optional[torch.Tensor] = None,
              even: Optional[torch.Tensor] = None, even_nb: int = 0, keep_first: int = 0,
              bias_log2: Optional[torch.Tensor] = None, null_log2: Optional[torch.Tensor] = None,
              gate: Optional[torch.Tensor] = None, chunk: int = 0, diff: Optional[Tuple[float, float, float]] = None) -> None:
    """One launch of the paged attention kernel over the requests whose q_len lies in
    [qlen_min, qlen_max]; see csrc/attention.cu for the meaning of every argument.  keep_first: with a window, the first
    keys of a request that stay visible whatever the window; bias_log2: float32 [heads, L], added to the scaled score in
    log2 units by distance min(i - j, L - 1) (both: the bfloat16 mma kernels only, see `window_bias_supported`).  `order` (uniform decode only):
    int32 [B], a permutation of the requests; the launch's i-th block along x takes request order[i].  `even`: the even cut
    of a decode step's keys over `even_nb` blocks per kv head (engine/step.py: plan_even_cut) in place of `grid_x` blocks.
    null_log2: float32 [heads], the score in log2 units of one more term in every softmax's denominator that has no key and no
    value; gate [T, heads * d] (a view into packed rows): the output times sigmoid(gate), element by element.  Both enter where a
    row is normalised, so a launch whose requests are cut hands them to `attention_combine` too.  chunk > 0 (with window 0): a query sees
    the keys of its own chunk of `chunk` positions only, counted from the start of the sequence.  diff = (lambda, eps, scale): query heads 2 h and 2 h + 1 are the two maps of
    output head h, out [T, n_q / 2, d] = v / sqrt(mean(v^2) + eps) * scale with v = a_2h - lambda a_2h+1; the decode variant leaves
    partial results for `attention_combine_diff` whatever the splits."""
    gate_stride = _attention_extras(q, null_log2, gate)
    _need_cuda(q, out, k_cache, v_cache, q_start, kv_len, block_table, nsplit, part_o, part_ml, order, even)
    T, n_q, d = q.shape
    B = kv_len.numel()
    assert q.is_contiguous() and out.is_contiguous() and block_table.dim() == 2 and block_table.stride(1) == 1
    assert q_start.numel() == B + 1 and block_table.shape[0] == B and tuple(out.shape) == (T, n_q if diff is None else n_q // 2, d)
    assert nsplit is None or nsplit.numel() == B
    assert order is None or (uniform_decode and order.numel() == B and order.dtype == torch.int32)
    assert even is None or (uniform_decode and variant == VARIANT_MMA_DECODE and even.dtype == torch.int32 and
                            even.numel() >= even_cut_size(B, even_nb) and even_nb >= 1)
    if max_split > 1 or (diff is not None and variant == VARIANT_MMA_DECODE):
        assert part_o.numel() >= max_split * T * n_q * d and part_ml.numel() >= max_split * T * n_q * 2
    if keep_first or bias_log2 is not None:
        _need_cuda(bias_log2)
        assert even is None, "the even cut of a decode step knows no kept tokens and no bias"
        assert null_log2 is None and gate is None and not chunk and diff is None, "a launch with kept tokens or a bias takes no further term, gate, chunk or pairs of maps"
        if bias_log2 is not None:
            assert bias_log2.dtype == torch.float32 and bias_log2.dim() == 2 and bias_log2.shape[0] == n_q and bias_log2.is_contiguous()
        code = _attn_lib(d).msgl_attention_window(
            _ptr(q), _ptr(out), _ptr(k_cache), _ptr(v_cache), _ptr(q_start), _ptr(kv_len), _ptr(block_table),
            _ptr(nsplit), _ptr(part_o), _ptr(part_ml), B, T, n_q, n_kv, d, page_size, block_table.stride(0), window,
            max_split, float(scale), qlen_min, qlen_max, int(uniform_decode), variant, grid_x, _dt(q), _ptr(order),
            int(keep_first), _ptr(bias_log2), bias_log2.shape[1] if bias_log2 is not None else 0, _stream())
        _check(code, f"attention with kept tokens / bias (head size {d}, variant {variant})")
        return
    code = _attn_lib(d).msgl_attention(
        _ptr(q), _ptr(out), _ptr(k_cache), _ptr(v_cache), _ptr(q_start), _ptr(kv_len), _ptr(block_table),
        _ptr(nsplit), _ptr(part_o), _ptr(part_ml), B, T, n_q, n_kv, d, page_size, block_table.stride(0), window,
        max_split, float(scale), qlen_min, qlen_max, int(uniform_decode), variant, grid_x, _dt(q), _ptr(order), _ptr(even), int(even_nb),
        _ptr(null_log2), _ptr(gate), gate_stride, int(chunk), int(diff is not None), *(diff or (0.0, 0.0, 0.0)), _stream())
    _check(code, f"attention (head size {d}, variant {variant})")


RUNS_MAX_REQUESTS, RUNS_MAX_BLOCKS = 256, 256


def decode_runs_supported(q: torch.Tensor, B: int, n_kv: int, page_size: int, table_width: int, workspace) -> bool:
    """Whether `attention_decode_runs` takes a step of B requests (but for a stream capture that comes before its counters)."""
    return (workspace is not None and q.dtype == torch.bfloat16 and q.shape[2] == 128 and q.shape[1] <= 8 * n_kv and page_size % 16 == 0
            and 0 < B <= RUNS_MAX_REQUESTS and B * n_kv * (table_width * (page_size // 16) + 1) < 1 << 30)


def decode_runs_scratch(q: torch.Tensor, B: int, n_kv: int, workspace) -> Optional[Tuple[torch.Tensor, torch.Tensor]]:
    """(counters, a word a request and kv head and zero between launches; float32 partial results of two segments a block), or None in a capture that comes before the counters exist.
    Tensors of their own: a step's partial results must not reach words that a step of another size counts in.  Counters are made for the largest batch, so that no batch outgrows them."""
    count = workspace.counters("attn_runs", max(RUNS_MAX_REQUESTS, B) * n_kv)
    if count is None:
        return None
    return count, workspace.whole("attn_runs_part", 2 * 8 * (128 + 2) * min(sm_count(q.device), RUNS_MAX_BLOCKS), torch.float32)


def attention_decode_runs(q: torch.Tensor, out: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, *, kv_len: torch.Tensor,
                          block_table: torch.Tensor, n_kv: int, page_size: int, scale: float, workspace, q_start: Optional[torch.Tensor] = None,
                          beside_tiles: bool = False, scratch: Optional[Tuple[torch.Tensor, torch.Tensor]] = None) -> bool:
    """Attention of a decode step (one new token a request, all of a request's keys) in one launch that deals the keys out over the SMs by
    itself and merges its partial results (csrc/attention_runs.cuh).  With q_start, int32 [B + 1], of the requests of any step that bring one token, out's rows of the others
    are left alone; beside_tiles: the launch before this one is the prefill kernel of the same step, beside which it may run; scratch: from `decode_runs_scratch`, asked for ahead of
    that launch, with the sizes looked at.  -> False where it does not apply: bfloat16,
    head size 128, up to eight query heads a kv head, pages of whole units of 16 keys, up to 256 requests; inside a stream capture only once its counters exist."""
    (T, n_q, d), (B, width) = q.shape, block_table.shape
    if scratch is None:
        if (q_start is None and T != B) or not decode_runs_supported(q, B, n_kv, page_size, width, workspace):
            return False
        scratch = decode_runs_scratch(q, B, n_kv, workspace)
        if scratch is None:
            return False
        _need_cuda(q, out, k_cache, v_cache, kv_len, block_table, q_start)
        assert q.is_contiguous() and out.is_contiguous() and block_table.stride(1) == 1
        assert kv_len.numel() == B and out.shape == q.shape and (q_start is None or q_start.numel() == B + 1)
    blocks = min(sm_count(q.device), RUNS_MAX_BLOCKS)
    count, part = scratch[0].data_ptr(), scratch[1].data_ptr()
    code = _attn_lib(d).msgl_attention_decode_runs(
        q.data_ptr(), out.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), kv_len.data_ptr(), block_table.data_ptr(), part, part + blocks * 16 * d * 4,
        count, _ptr(q_start), int(beside_tiles), B, n_q, n_kv, page_size, block_table.stride(0), scale, blocks, _stream())
    _check(code, "attention of a decode step")
    return True


def attention_combine(part_o: torch.Tensor, part_ml: torch.Tensor, token_req: Optional[torch.Tensor],
                      nsplit: torch.Tensor, out: torch.Tensor, max_split: int, null_log2: Optional[torch.Tensor] = None,
                      gate: Optional[torch.Tensor] = None) -> None:
    _need_cuda(part_o, part_ml, token_req, nsplit, out)
    gate_stride = _attention_extras(out, null_log2, gate)
    T, n_q, d = out.shape
    code = _attn_lib(d).msgl_attention_combine(_ptr(part_o), _ptr(part_ml), _ptr(token_req), _ptr(nsplit), _ptr(out),
                                               T, n_q, d, max_split, _dt(out), _ptr(null_log2), _ptr(gate), gate_stride, _stream())
    _check(code, "attention_combine")


def attention_combine_diff(part_o: torch.Tensor, part_ml: torch.Tensor, token_req: Optional[torch.Tensor], nsplit: Optional[torch.Tensor],
                           q_start: torch.Tensor, qlen_max: int, out: torch.Tensor, max_split: int, diff: Tuple[float, float, float]) -> None:
    """The partial results of `attention(diff=...)` launches of the decode variant -> out [T, heads, d], for the tokens of the requests
    that brought at most qlen_max of them or whose keys are cut."""
    _need_cuda(part_o, part_ml, token_req, nsplit, q_start, out)
    T, h, d = out.shape
    assert out.is_contiguous() and part_o.numel() >= max_split * T * 2 * h * d and part_ml.numel() >= max_split * T * 2 * h * 2
    code = _attn_lib(d).msgl_attention_combine_diff(_ptr(part_o), _ptr(part_ml), _ptr(token_req), _ptr(nsplit), _ptr(q_start), int(qlen_max),
                                                    _ptr(out), T, 2 * h, d, max_split, _dt(out), *diff, _stream())
    _check(code, "attention_combine_diff")


# ---------------------------------------------------------------------------------------
# matrix products: the library GEMM (cuBLAS through torch)
# ---------------------------------------------------------------------------------------

def set_true_fp32() -> None:
    """float32 products are real float32: no TF32, no reduced-precision reduction."""
    torch.backends.cuda.matmul.allow_tf32 = False
    torch.backends.cudnn.allow_tf32 = False
    torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
    torch.set_float32_matmul_precision("highest")


SMALL_M_MAX = int(os.environ.get("MSGL_SMALL_M_MAX", "8"))      # tokens up to which the weight-streaming kernel replaces the library GEMM (measured: faster up to 8)
USE_SMALL_M = os.environ.get("MSGL_NO_SMALL_M", "") == ""


# elements of a weight from which on the kernel of one block an SM is ahead; us a product of a chain, blocks of 16 rows / one an SM, one row: [1024, 1024] 1.63 / 1.86, [768, 2048] 2.40 /
# 2.39, gated [1792, 1024] 2.23 / 2.14 and with 8 rows 2.33 / 2.39, [2048, 1024] 2.47 / 2.22, [1024, 3072] 4.02 / 3.08, [4096, 4096] 8.0 / 7.3, [5120, 25600] 54 / 41
STREAM_MIN_WEIGHTS = 2_000_000


def _small_m(weight, x, bias, out, M, N, K, ldo, mode, out_f32, ahead=None) -> int:
    """Weights of some size go through one block an SM (csrc/gemm_stream.cu), smaller ones, for which its barriers and tensor maps cost more than they bring, through
    blocks of 16 rows (csrc/gemm_small_m.cu).  ahead: a weight that gated products of the second kind, with inner sizes below 423, ask into L2 for the product behind them (or None; one that lies
    elsewhere or in pieces is left alone); with the first the product behind has its own weights on their way by itself."""
    if M <= 8 and _stream_rule(M, N, K, mode != 0):
        status = _status_words(x.device) if _status is None else _status
        code = _lib().msgl_gemm_stream(weight.data_ptr(), x.data_ptr(), _ptr(bias), out.data_ptr(), M, N, K, x.stride(0), ldo, mode, out_f32, _ptr(status), _stream())
        if code != 2:             # (2: no tensor map of this layout)
            return code
    if ahead is not None and (not ahead.is_contiguous() or ahead.get_device() != x.get_device()):
        ahead = None
    return _lib().msgl_gemm_small_m(_ptr(weight), _ptr(x), _ptr(bias), _ptr(out), M, N, K, x.stride(0), ldo, mode, out_f32, _ptr(ahead), ahead.numel() * ahead.element_size() if ahead is not None else 0, _stream())


# Where the kernel of one block an SM is ahead; us of a product with weights from memory, other kernel (blocks of 16 rows up to 8 rows, then the library and, gated, the decode-batch kernel) then
# this one.  Lines in columns follow the B200's 148 SMs: 7,104 columns are 48 on each, the most of one pass, 2,072 are 14, 2,960 are 20, (gated) 5,328 are 36.
# Up to 8 rows: behind where a block has more than one pass of few rounds (576 elements of K each), by STREAM_SHORT's pairs of columns and K (the first for plain products alone).  8 rows of [7120, 768]
# 4.2 5.1, [7120, 3072] 10.4 10.9, [7424, 2048] 8.4 8.4, [8192, 1024] 5.3 6.0, [8192, 4096] 16.0 14.2, [9216, 1024] 5.5 6.1, [9728, 1024] 6.0 6.1, [15936, 640] 6.5 7.2; gated [8192, 1024] 5.4 5.7,
# [7424, 2048] 9.0 8.0.  Plain products of five rows and more with two passes or more also where the last of two or three rounds brings 160 elements of K at most: [14784, 1216] 8.8 9.5, [15376, 1280] 9.4 9.7,
# [21344, 704] 8.4 9.0, but [14592, 1024] 7.9 7.8, [21344, 1536] 14.1 13.3.  An inner size that is no multiple of 64 is nine copies a round: [560, 8672] 7.5 11.2, [928, 2976] 3.8 4.4, gated 4.1 6.9, [7712, 1120] 5.5 6.2, gated [4480, 4960] 10.0 10.6, [14224, 288] 4.3 5.0, but [3088, 1056] 3.6 2.9.
# From 9 rows on every SM reads all rows of x, which costs more the more rows there are, and passes cost more: at 9 / 16 / 24 / 32 rows
# [4096, 1024] 4.8 4.8 4.9 4.9, 2.9 3.7 4.1 4.5; [1024, 3072] 8.5 8.5 7.6 7.5, 4.5 4.5 4.9 6.1; [2048, 6144] 10.5 10.5 10.5 10.6, 8.6 9.1 8.1 9.7; [4096, 2048] 6.2 6.3 6.4 6.4, 5.3 5.5 6.2 7.4;
# [6144, 4096] 12.8 12.9 12.1 13.2, 11.8 12.0 13.3 24; [4096, 12288] 22.0 22.1 22.6 22.7, 18.5 19.2 23.4 32; [5120, 25600] 49.6 46.8 46.2 46.3, 43.2 43.4 55 69.  Gated: [6144, 1024] 6.4 6.4 6.7 6.9,
# 4.4 4.7 5.1 7.0; [12288, 2048] 12.0 12.3 12.5 12.9, 11.9 12.3 13.5 16.7; [24576, 4096] 35.8 36.6 36.1 36.8, 37.7 38.9 41.6 54.
# More than one pass at 16 rows: [13776, 6144] 29.8 30.6, [14112, 192] 4.1 4.4, [64064, 448] 12.8 16.1, [116480, 128] 9.5 21.6; gated, two passes: [10240, 1024] 8.1 7.6 and [10240, 1536] 9.6 10.5 at 24 rows, seven:
# [45984, 96] 4.9 11.2.  From K of some 12,900 on the library cuts K up: [1024, 12288] x 16 27.0 15.9, [608, 12992] 13.2 15.7, [1024, 14336] 14.4 17.9, with more columns [2560, 25600] x 9 31.1 25.7.  No multiple of 64: [448, 6880] x 16 8.0 8.8,
# [5872, 608] x 24 4.5 5.0, little in the last round: [3440, 1216] x 32 5.0 5.8, [6224, 704] 4.8 7.2, gated [1408, 5280] x 16 7.8 10.1, [4992, 2528] x 21 8.8 9.7, [8192, 1760] x 16 9.5 10.5.  Gated, long inner sizes, 24 rows: [1024, 8192] 9.5 10.0, [928, 11904] 11.9 13.2, [1184, 6848] 8.8 8.5.
STREAM_ROWS, STREAM_ROWS_FEW_COLUMNS, STREAM_ROWS_SMALL, STREAM_FEW_COLUMNS, STREAM_SMALL_WEIGHTS = 16, 24, 32, 2_072, 4_500_000
STREAM_ROWS_GATED, STREAM_GATED_LEAST, STREAM_GATED_MOST = 24, 4_000_000, 16_000_000      # ([8192, 2048], 16.8 million, is ahead too, [10240, 2048] and [12288, 2048] are not)
STREAM_ONE_PASS, STREAM_ROUND, STREAM_SHORT, STREAM_GATED_INNER, STREAM_GATED_LONG = 7_104, 576, ((7_400, 3_600), (10_000, 1_300), (17_000, 800)), 1_100, 7_000
STREAM_THIN_COLUMNS, STREAM_THIN_INNER, STREAM_THIN_ROUND = 23_000, 1_300, 160
STREAM_LONG_INNER, STREAM_LONG_COLUMNS, STREAM_RAGGED, STREAM_RAGGED_GATED, STREAM_RAGGED_WIDE = 12_500, 2_560, 2_960, 5_328, 17_000


def _stream_rule(rows: int, N: int, K: int, gated: bool) -> bool:
    """Whether a product goes to the kernel of one block an SM."""
    if N * K < STREAM_MIN_WEIGHTS or N % 16 or K % 32 or (K % 64 and N < (STREAM_RAGGED_GATED if gated else STREAM_RAGGED)):
        return False
    thin = 0 < K % STREAM_ROUND <= STREAM_THIN_ROUND          # the last round brings little
    if rows <= 8:
        if N <= STREAM_ONE_PASS or (K <= STREAM_ROUND and (N > STREAM_RAGGED_WIDE or not K % 64)):
            return True
        if K % 64 or any(N <= columns and K <= inner for columns, inner in STREAM_SHORT[gated:]):
            return False
        return gated or rows <= 4 or N > STREAM_THIN_COLUMNS or K > STREAM_THIN_INNER or not thin
    if gated:
        return (rows <= (STREAM_ROWS if K % 64 or K > STREAM_GATED_LONG else STREAM_ROWS_GATED) and STREAM_GATED_LEAST <= N * K <= STREAM_GATED_MOST
                and (N <= STREAM_ONE_PASS or (N <= 2 * STREAM_ONE_PASS and not K % 64 and (rows <= STREAM_ROWS or K <= STREAM_GATED_INNER))))
    if N > STREAM_ONE_PASS or (K > STREAM_LONG_INNER and N < STREAM_LONG_COLUMNS) or (rows > STREAM_ROWS and (K % 64 or (thin and N > STREAM_FEW_COLUMNS))):
        return False
    return rows <= (STREAM_ROWS_SMALL if N * K <= STREAM_SMALL_WEIGHTS else STREAM_ROWS_FEW_COLUMNS if N <= STREAM_FEW_COLUMNS else STREAM_ROWS)


def _by_address(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], N: int) -> bool:
    """Whether operands of a product that was the library's, x [M, K] and weight [N, K], lie as a kernel called by address reads them, on the current device, and nothing looks on that
    it would slip past: gradients, autocast, `_observed`."""
    # (a prompt step of a few tokens waits for the host: one look at everything, each thing asked for once)
    dev, (pitch, step) = x.get_device(), x.stride()
    return (x.dtype is torch.bfloat16 and weight.dtype is torch.bfloat16 and step == 1 and pitch % 8 == 0 and weight.is_contiguous() and weight.get_device() == dev
            and (bias is None or (bias.dtype == torch.bfloat16 and bias.dim() == 1 and bias.shape[0] == N and bias.is_contiguous() and bias.get_device() == dev))
            and not (torch.is_grad_enabled() and (x.requires_grad or weight.requires_grad or (bias is not None and bias.requires_grad)))
            and not _observed(x, weight, bias)                       # (before the addresses are asked for: some of these have none)
            and (x.data_ptr() | weight.data_ptr()) % 16 == 0 and dev == torch._C._cuda_getDevice() and not torch.is_autocast_enabled())


def _gemm_stream(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], mode: int, out_dtype: torch.dtype) -> Optional[torch.Tensor]:
    """x @ weight^T (mode 0) or its gated activation (1: SwiGLU, 2: ReGLU) of 9 rows and more by csrc/gemm_stream.cu; None where another kernel or the library is to be called: by
    `_stream_rule` or `_by_address`."""
    if x.dim() != 2 or weight.dim() != 2:
        return None
    (M, K), (N, k_weight) = x.shape, weight.shape
    if not SMALL_M_MAX < M <= STREAM_ROWS_SMALL or K != k_weight or not _stream_rule(M, N, K, mode != 0) or MID_GEMM or not USE_SMALL_M or not _by_address(x, weight, bias, N):
        return None
    n_out, f32 = N // 2 if mode else N, out_dtype == torch.float32
    out = x.new_empty((M, n_out), dtype=torch.float32) if f32 else x.new_empty((M, n_out))
    status = _status_words(x.device) if _status is None else _status
    code = _lib().msgl_gemm_stream(weight.data_ptr(), x.data_ptr(), _ptr(bias), out.data_ptr(), M, N, K, x.stride(0), n_out, mode, int(f32), _ptr(status), _stream())
    if code == 2:             # no tensor map of this layout
        return None
    _check(code, "gemm_stream")
    return out


def _product_ok(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor]) -> bool:
    """Whether x [M, K] . weight [N, K]^T + bias [N] is a bfloat16 product whose operands lie as the kernels read them: rows of x one behind
    the other on 16-byte pitches, packed weights and bias, one device.  The kernels get addresses and sizes only, so whatever
    does not fit goes to the library, which takes it or refuses it."""
    return (x.dtype is torch.bfloat16 and weight.dtype is torch.bfloat16 and x.dim() == 2 and weight.dim() == 2 and x.shape[1] == (sizes := weight.shape)[1]
            and (strides := x.stride())[1] == 1 and strides[0] % 8 == 0 and weight.is_contiguous() and x.get_device() == weight.get_device()
            and (bias is None or (bias.dtype == torch.bfloat16 and bias.dim() == 1 and bias.shape[0] == sizes[0] and bias.is_contiguous()
                                  and bias.get_device() == weight.get_device())))


def _small_m_ok(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor]) -> bool:
    if not (USE_SMALL_M and 0 < x.shape[0] <= SMALL_M_MAX and _product_ok(x, weight, bias)):
        return False
    N, K = weight.shape
    return K % 32 == 0 and N % 16 == 0


# This engine's tcgen05 GEMM (csrc/gemm_tc.cu) against the library's, measured on B200 at Qwen3-8B's sizes.  With SwiGLU in
# its epilogue the kernel on pairs of SMs (cta_group::2) beats library GEMM + activation kernel from about 256 rows on
# (512 rows: 83 against 86 us, 2,048 rows: 285 against 310 us, 4,096 rows: 0.52 against 0.72 ms; 2,048-token prefill step
# 27.4 -> 26.4 ms).  Its plain products reach 92-95 % of the library's speed at 2,048 rows (the one-block kernel: 88 %), so
# those stay with the library unless MSGL_TC_GEMM=all (prefill step + 1.3 ms).  MSGL_TC_GEMM=0 switches the kernel off,
# MSGL_TC_GEMM_CTAS=1 takes the one-block kernel.
TC_GEMM = os.environ.get("MSGL_TC_GEMM", "swiglu")            # "swiglu" | "all" | "0"
TC_GEMM_MIN_M = int(os.environ.get("MSGL_TC_GEMM_MIN_M", "256"))
TC_GEMM_CTAS = int(os.environ.get("MSGL_TC_GEMM_CTAS", "2"))   # 2: the kernel on pairs of SMs (tcgen05 cta_group::2)
_tc_gemm_usable = True


def _tc_gemm(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], mode: int) -> Optional[torch.Tensor]:
    """x @ weight^T (mode 0) or its gated activation (mode 1: SwiGLU, 2: ReGLU; bias [2I]) by the tcgen05 kernel; None where it
    does not apply."""
    global _tc_gemm_usable
    if not ((TC_GEMM == "all" or (TC_GEMM == "swiglu" and mode != 0)) and _tc_gemm_usable and x.shape[0] >= TC_GEMM_MIN_M
            and _product_ok(x, weight, bias) and weight.shape[1] % 8 == 0):
        return None
    M, (N, K) = x.shape[0], weight.shape
    n_out = N // 2 if mode else N
    if n_out % 8 or (mode and N % 2):
        return None
    out = torch.empty((M, n_out), dtype=torch.bfloat16, device=x.device)
    fn = _lib().msgl_gemm_tc2 if TC_GEMM_CTAS == 2 else _lib().msgl_gemm_tc
    code = fn(_ptr(weight), _ptr(x), _ptr(bias), _ptr(out), M, N, K, x.stride(0), n_out, mode, _ptr(_status_tensor(x.device)), _stream())
    if code == 2:             # no tensor maps on this driver
        _tc_gemm_usable = False
        return None
    _check(code, "gemm_tc")
    return out


# Between the weight-streaming kernel (up to SMALL_M_MAX rows) and the tiled tcgen05 kernel (from TC_GEMM_MIN_M rows) a product has
# too few output tiles to fill the GPU: there the pair kernel cuts K into ranges as well (split-K) and a second kernel adds
# the ranges' float32 partial sums in order.  Off unless MSGL_TC_MID=1: measured on B200 at Qwen3-8B's sizes it is behind the
# library GEMM at 16 to 128 rows (qkv 18-26 against 12.5 us, o 15-21 against 10, gate/up + SwiGLU 44-66 against 42-45, down 26-33
# against 21-22 us), so these sizes stay with the library.
MID_GEMM = os.environ.get("MSGL_TC_MID", "0") == "1"
MID_GEMM_SPLITS = int(os.environ.get("MSGL_TC_MID_SPLITS", "0"))        # 0: chosen per size
_mid_partials = {}
_mid_splits = {}


def _tc_gemm_mid(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], mode: int) -> Optional[torch.Tensor]:
    """x @ weight^T (mode 0) or its gated activation (modes 1, 2) for a middling number of rows by the split-K tcgen05 kernel; None where
    it does not apply."""
    global _tc_gemm_usable
    if not (MID_GEMM and TC_GEMM != "0" and TC_GEMM_CTAS == 2 and _tc_gemm_usable and SMALL_M_MAX < x.shape[0] < TC_GEMM_MIN_M
            and _product_ok(x, weight, bias) and weight.shape[1] % 8 == 0 and weight.shape[0] % 8 == 0 and weight.shape[1] >= 512):
        return None
    M, (N, K) = x.shape[0], weight.shape
    n_out = N // 2 if mode else N
    if n_out % 8 or (mode and N % 16):
        return None
    key = (M, N, K, mode)
    splits = MID_GEMM_SPLITS or _mid_splits.get(key)
    if not splits:
        splits = _mid_splits[key] = int(_lib().msgl_gemm_tc2_splits(M, N, K, mode))
    splits = max(1, min(splits, K // 64))
    part = None
    if splits > 1:
        dev = x.device.index if x.device.index is not None else torch.cuda.current_device()
        part = _mid_partials.get(dev)
        if part is None or part.numel() < splits * M * N:
            part = _mid_partials[dev] = torch.empty(max(splits * M * N, 1 << 22), dtype=torch.float32, device=x.device)
    out = torch.empty((M, n_out), dtype=torch.bfloat16, device=x.device)
    code = _lib().msgl_gemm_tc2_splitk(_ptr(weight), _ptr(x), _ptr(bias), _ptr(out), M, N, K, x.stride(0), n_out, mode, splits,
                                       _ptr(part), _ptr(_status_tensor(x.device)), _stream())
    if code == 2:             # no tensor maps on this driver
        _tc_gemm_usable = False
        return None
    _check(code, "gemm_tc (split-K)")
    if splits > 1:
        global LAUNCHES
        LAUNCHES += 1
    return out


# The product for a decode batch (csrc/gemm_rows.cu: weights on the tensor core's M dimension, tokens on its N dimension) against
# the library's, measured on B200 over the Qwen3 widths.  Gated products, [2 n_out, K] weights, library product + activation kernel
# against this kernel: 16 rows [6144, 1024] 7.2 / 6.0 us, [12288, 2048] 14.1 / 11.4, [24576, 4096] 42.7 / 35.9, [51200, 5120] 99.9 / 82.5;
# 64 rows 7.2 / 7.3, 14.4 / 13.2, 45.0 / 37.4, 103 / 83; 128 rows 7.6 / 9.5, 14.4 / 17.6, 45.3 / 41.8, 107 / 94; 176 rows behind everywhere.  Small
# weights: [512, 256] 48 rows 4.5 / 4.5, 64 rows 4.6 / 5.2, [1536, 512] 5.0 / 4.8 and 5.0 / 5.4, [2048, 1024] 64 rows 6.0 / 5.2.
# Up to 8 rows the weight-streaming kernel is level (35.0 / 34.7 us at one row of [24576, 4096]) or ahead on small weights.
# Float32 products with very many columns (output heads, 151,936 columns): K = 4096, 1 / 8 / 24 / 64 / 128 rows 194 / 200 / 214 / 215 / 233
# (the better of the library and the weight-streaming kernel) against 181 / 184 / 188 / 196 / 227 us, K = 1024, 1 / 64 rows 54 / 64 against
# 51 / 64.  The gain is lost where the last round of blocks (three an SM) is nearly empty, so the rule asks how full the rounds are: 2.67 rounds
# of 3 (151,936 columns) and 2.88 (163,840) are ahead but for up to 3 % at 65 to 80 rows; 2.01 (114,048) and 2.13 (120,832) are 4 to 17 % behind
# at 9 to 16 rows; 2.26 (128,256) and 2.31 (131,072) up to 13 % behind for K <= 2560 and 0 to 14 % ahead from K = 4096 on.  Heads of fewer
# columns stay where they were: with 32,768 columns it is 2 to 18 % behind.  Plain bfloat16 products stay with
# the library (4096 x 4096 at 48 rows: 9.6 against 10.1 us, 128 rows 9.7 against 12.3).
ROWS_GLU_MAX_SMALL, ROWS_GLU_MAX, ROWS_GLU_MAX_LARGE = 48, 64, 128             # rows
ROWS_SMALL_WEIGHT, ROWS_LARGE_WEIGHT = 1_500_000, 40_000_000                    # elements of the weight up to and from which the outer bounds hold
ROWS_F32_MAX, ROWS_F32_MIN_OUT = 128, 114_000                                   # rows; columns
ROWS_F32_FILL, ROWS_F32_FILL_LONG, ROWS_F32_LONG = 0.85, 0.75, 4096             # how full the rounds of blocks have to be, and from which K the second holds


def _rows_glu_max(weights: int) -> int:
    return ROWS_GLU_MAX_LARGE if weights >= ROWS_LARGE_WEIGHT else ROWS_GLU_MAX if weights >= ROWS_SMALL_WEIGHT else ROWS_GLU_MAX_SMALL


def _rows_f32(rows: int, n_out: int, K: int, device) -> bool:
    """Whether a float32 product goes to the decode-batch kernel (figures above)."""
    if n_out < ROWS_F32_MIN_OUT or rows > ROWS_F32_MAX:
        return False
    tiles, slots = -(-n_out // 128), 3 * sm_count(device)
    return tiles >= (ROWS_F32_FILL_LONG if K >= ROWS_F32_LONG else ROWS_F32_FILL) * slots * -(-tiles // slots)


_tensor_maps = None


def tensor_maps() -> bool:
    """Whether the driver makes the tensor maps that the decode-batch product loads by (asked once)."""
    global _tensor_maps
    if _tensor_maps is None:
        _tensor_maps = bool(_lib().msgl_tensor_maps())
    return _tensor_maps


_PLAIN = (torch.Tensor, torch.nn.Parameter)


def _observed(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None) -> bool:
    """Whether something looks on that a kernel called by address would slip past: compiling, tracing, a dispatch mode, vmap and its like, forward-mode
    derivatives, a tensor of another class."""
    return (torch.compiler.is_compiling() or type(x) not in _PLAIN or type(weight) not in _PLAIN or (bias is not None and type(bias) not in _PLAIN) or torch._C._len_torch_dispatch_stack() > 0
            or torch._C._functorch.peek_interpreter_stack() is not None or torch.autograd.forward_ad._current_level >= 0
            or torch._C._get_tracing_state() is not None)


# Plain products of a decode batch with a long inner size (down projections) on the decode-batch kernel, whose ranges of K give them enough blocks; us, library / kernel, at 33 / 48 / 64 rows:
# [1024, 3072] 6.8 / 6.1, 6.8 / 6.2, 6.7 / 6.4; [2048, 8192] 13.4 / 11.2, 13.3 / 11.6, 13.4 / 12.1; [2560, 9728] 15.7 / 13.9, 15.9 / 14.4, 15.6 / 14.6; [4096, 12288] 22.6 / 21.5, 22.5 / 21.9,
# 22.6 / 22.4; [5120, 17408] 39.0 / 33.0, 41.0 / 34.0, 36.1 / 35.1; at 80 rows behind on half of them.  Shorter inner sizes: [5120, 8192] 18.2 / 18.9 at 33 rows, [4096, 4096] 10.3 / 10.7 at 48.
# From K = 20,480 on the library cuts K of few columns up: at 48 rows [512, 18432] 16.5 / 16.0, [512, 20480] 13.9 / 17.4, at 64 [1536, 24576] 20.5 / 22.6, [3584, 32768] 45.2 / 44.2.  Eight ranges of K
# are clusters of eight blocks, a tile of 128 columns each: behind with 33 to 39 tiles, planned two blocks an SM, and from 51 on, planned three, as if 32 and 48 clusters were all that run at once: at 48 rows
# [4096, 16384] 28.9 / 28.2, [4352, 16384] 29.0 / 39.9, [4736, 16128] 30.4 / 40.2, [5120, 16384] 38.9 / 32.1, at 24 [6144, 20480] ahead by 4 to 8 %, [6480, 20352] 49.5 / 58.5.
# (What the rule takes was measured at 533 sizes and rows: one of them, 64 rows of [4096, 14336], is 3 % behind.)
ROWS_PLAIN_MAX, ROWS_PLAIN_INNER, ROWS_PLAIN_WEIGHTS = 64, 3, 3_000_000
ROWS_PLAIN_LONGEST, ROWS_PLAIN_LONG_COLUMNS, ROWS_PLAIN_GAP, ROWS_PLAIN_COLUMNS = 18_432, 3_584, (4_096, 5_120), 6_144


def _rows_plain(rows: int, N: int, K: int) -> bool:
    return (SMALL_M_MAX < rows <= ROWS_PLAIN_MAX and K >= ROWS_PLAIN_INNER * N and N * K >= ROWS_PLAIN_WEIGHTS and (K <= ROWS_PLAIN_LONGEST or N >= ROWS_PLAIN_LONG_COLUMNS)
            and not ROWS_PLAIN_GAP[0] < N < ROWS_PLAIN_GAP[1] and N <= ROWS_PLAIN_COLUMNS and not MID_GEMM)


def _gemm_rows_plain(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], out_dtype: torch.dtype) -> Optional[torch.Tensor]:
    """x @ weight^T by the decode-batch kernel where it is ahead of the library (`_rows_plain`); None where the library is to be called: by that rule or `_by_address`, rows of x that
    overlap, or a stream capture that comes before the status words, which the kernel cannot go without."""
    if x.dim() != 2 or weight.dim() != 2:
        return None
    (M, K), (N, k_weight) = x.shape, weight.shape
    if K != k_weight or not _rows_plain(M, N, K) or K % 8 or N % 2 or not _by_address(x, weight, bias, N):
        return None
    pitch, status, f32 = x.stride(0), _status_words(x.device) if _status is None else _status, out_dtype == torch.float32
    if pitch < K or status is None:
        return None
    out = x.new_empty((M, N), dtype=torch.float32) if f32 else x.new_empty((M, N))
    code = _lib().msgl_gemm_rows_plain(weight.data_ptr(), x.data_ptr(), _ptr(bias), out.data_ptr(), M, N, K, pitch, N, int(f32), status.data_ptr(), _stream())
    if code == 2:             # no tensor map of this layout
        return None
    _check(code, "gemm_rows")
    return out


def _gemm_rows(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], mode: int, out_dtype: torch.dtype) -> Optional[torch.Tensor]:
    """x @ weight^T (mode 0) or its gated activation (1: SwiGLU, 2: ReGLU; bias [2I]) for at most 256 rows by the decode-batch kernel;
    None where it cannot run."""
    if not (0 < x.shape[0] <= 256 and _product_ok(x, weight, bias)
            and not (torch.is_grad_enabled() and (x.requires_grad or weight.requires_grad or (bias is not None and bias.requires_grad)))
            and not _observed(x, weight, bias)):
        return None
    M, (N, K), pitch, x_at, w_at = x.shape[0], weight.shape, x.stride(0), x.data_ptr(), weight.data_ptr()
    if (x_at | w_at) % 16 or K % 8 or (pitch < K and M != 1):
        return None
    n_out = N // 2 if mode else N
    if n_out % 2 or (mode and N % 2) or (mode and out_dtype != torch.bfloat16) or not tensor_maps():
        return None
    out = x.new_empty((M, n_out), dtype=out_dtype)
    code = _lib().msgl_gemm_rows(w_at, x_at, _ptr(bias), out.data_ptr(), M, n_out, K, pitch, n_out, mode, int(out_dtype == torch.float32),
                                 0.0, 0, None, 0, 0, 0, _ptr(_status_tensor(x.device)), _stream())
    if code == 2:             # no tensor map of this layout
        return None
    _check(code, "gemm_rows")
    return out


# Float32 products on the tensor cores against the library's, us, library / kernel.  [4096, 1024] at 4 rows 9.0 / 9.8, 9: 19.2 / 9.8, 64: 21.8 / 12.3, 256: 45.0 / 23.4,
# 600: 121 / 63; [1024, 2048] at 9: 19.9 / 9.2, 256: 39.5 / 17.2; [5120, 5120] at 9: 88 / 48, 1,000: 1,031 / 409; [512, 1024] at 9: 9.1 / 8.4, 64: 16.6 / 10.7; [2048, 512] at 9: 11.1 / 8.7,
# 64: 11.5 / 11.5, 128: 12.5 / 11.6; [1024, 512] at 16: 7.6 / 9.1, 128: 11.5 / 11.7.  With 4 rows the library is ahead on half of 17 sizes, with 6 on none that the rule has;
# from 9, above the bfloat16 kernels for a few rows, the kernel is never behind.  Errors against 64 bits, relative: 0.9e-7 to 1.3e-7, the library's 1.9e-7 to 1e-6.
F32_MIN_ROWS, F32_MIN_INNER, F32_LONG_INNER, F32_MIN_WEIGHT, F32_MIN_WEIGHT_LONG = 9, 512, 1024, 1_000_000, 500_000


def _f32_rule(rows: int, n_out: int, K: int) -> bool:
    return rows >= F32_MIN_ROWS and K >= F32_MIN_INNER and n_out * K >= (F32_MIN_WEIGHT_LONG if K >= F32_LONG_INNER else F32_MIN_WEIGHT)


def _tf32() -> bool:
    """Whether the library's float32 products may use TF32.  The older question is five times as quick, but raises where the newer switches were used."""
    try:
        return torch._C._get_cublas_allow_tf32()
    except RuntimeError:
        return torch._C._get_fp32_precision_getter("cuda", "matmul") == "tf32"


def _gemm_f32(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    """x @ weight^T + bias in float32 on the tensor cores (csrc/gemm_f32.cu); None where the library's float32 product is to be called: few rows or
    small weights, operands that do not lie as the kernel reads them or on another device than the current one, products that the caller wants in another precision (autocast, TF32),
    and whatever a kernel called by address would slip past."""
    if not (x.dtype == torch.float32 and weight.dtype == torch.float32 and x.dim() == 2 and weight.dim() == 2):
        return None
    (M, K), (N, k_weight) = x.shape, weight.shape
    if K != k_weight or K % 8 or not _f32_rule(M, N, K):
        return None
    pitch, dev = x.stride(0), x.get_device()
    if not (x.stride(1) == 1 and pitch % 4 == 0 and pitch >= K and weight.is_contiguous() and weight.get_device() == dev
            and (bias is None or (bias.dtype == torch.float32 and bias.dim() == 1 and bias.shape[0] == N and bias.is_contiguous() and bias.get_device() == dev))
            and not (torch.is_grad_enabled() and (x.requires_grad or weight.requires_grad or (bias is not None and bias.requires_grad)))
            and not _observed(x, weight, bias)):                     # (before the addresses are asked for: some of these have none)
        return None
    x_at, w_at = x.data_ptr(), weight.data_ptr()
    if (x_at | w_at) % 16 or dev != torch._C._cuda_getDevice():      # (the launch goes to the current device's stream; the library changes the device)
        return None
    if torch.is_autocast_enabled() or _tf32():
        return None
    status = _status_words(x.device)
    if status is None:
        return None
    out = torch.empty((M, N), dtype=torch.float32, device=x.device)
    _check(_lib().msgl_gemm_f32(w_at, x_at, _ptr(bias), out.data_ptr(), M, N, K, pitch, N, status.data_ptr(), _stream()), "gemm_f32")
    return out


_PRODUCT_RESULTS = (None, torch.bfloat16, torch.float32)


# Prompt steps of a few tokens wait for the host, so what stands ahead of a product's launch counts (us of host time a call on 9 to 64 bfloat16 rows: F.linear 10.2, this function ahead of it 0.8, on
# the streaming kernel 10.5 in all, on the decode-batch kernel 10.5): a tensor's dtype and device are asked for at 50 ns, its shape at 130, a single size or stride at 220
def linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None,
           out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    """y = x @ weight^T (+ bias); weight is [out, in] as stored in the checkpoint.

    Up to SMALL_M_MAX bfloat16 rows, and up to 16 or 32 by the weight's size (`_stream_rule`), go through this engine's weight-streaming kernels (csrc/gemm_stream.cu,
    csrc/gemm_small_m.cu), float32 results of
    very many columns for a decode batch and plain products with long inner sizes through its decode-batch kernel (csrc/gemm_rows.cu, `_rows_f32`, `_rows_plain`), float32 operands through the float32
    kernel of the tensor cores (csrc/gemm_f32.cu, `_f32_rule`); everything else is the
    library GEMM unless MSGL_TC_GEMM or MSGL_TC_MID ask for the tiled kernels."""
    if not (x.is_cuda and weight.is_cuda and (bias is None or bias.is_cuda)):
        _need_cuda(x, weight, bias)
    if out_dtype == torch.float32 and x.dim() == 2 and _rows_f32(x.shape[0], weight.shape[0], x.shape[1], x.device):
        y = _gemm_rows(x, weight, bias, 0, torch.float32)
        if y is not None:
            return y
    rows = x.shape[0]
    if rows <= SMALL_M_MAX and _small_m_ok(x, weight, bias) and out_dtype in _PRODUCT_RESULTS:
        M, (N, K) = rows, weight.shape
        od = out_dtype or torch.bfloat16
        out = torch.empty((M, N), dtype=od, device=x.device)
        code = _small_m(weight, x, bias, out, M, N, K, N, 0, int(od == torch.float32))
        _check(code, "gemm_small_m")
        return out
    if SMALL_M_MAX < rows <= ROWS_PLAIN_MAX and x.dtype is torch.bfloat16 and out_dtype in _PRODUCT_RESULTS:
        y = _gemm_stream(x, weight, bias, 0, out_dtype or torch.bfloat16) if rows <= STREAM_ROWS_SMALL else None
        if y is None and (sizes := weight.shape)[-1] >= ROWS_PLAIN_INNER * sizes[0]:
            y = _gemm_rows_plain(x, weight, bias, out_dtype or torch.bfloat16)
        if y is not None:
            return y
    if (rows >= TC_GEMM_MIN_M or MID_GEMM) and out_dtype in (None, torch.bfloat16):
        y = _tc_gemm(x, weight, bias, 0) if rows >= TC_GEMM_MIN_M else _tc_gemm_mid(x, weight, bias, 0)
        if y is not None:
            return y
    if x.dtype == torch.float32 and out_dtype in (None, torch.float32):
        y = _gemm_f32(x, weight, bias)
        if y is not None:
            return y
    if out_dtype is not None and out_dtype != x.dtype:
        y = torch.mm(x, weight.t(), out_dtype=out_dtype)
        if bias is not None:
            y += bias.to(out_dtype)
        return y
    return torch.nn.functional.linear(x, weight, bias)


GLU_MODES = {0: 1, 4: 2}          # the ACT_ numbers whose gated products have fused kernels (silu, relu) -> the kernels' mode


def linear_glu(x: torch.Tensor, gate_up: torch.Tensor, bias: Optional[torch.Tensor] = None, act: int = 0,
               ahead: Optional[torch.Tensor] = None) -> torch.Tensor:
    """act(x @ gate^T + bg) * (x @ up^T + bu) with gate_up = [gate; up] packed row-wise ([2I, H]) and bias = [bg; bu] or None;
    act: one of the ACT_ numbers.  Where a kernel with the activation in its epilogue applies (silu and relu; a few rows, or
    many rows in bfloat16) the [T, 2I] intermediate never exists.  ahead: the weight of the product that takes the result, which the kernel for a few rows
    and a small weight asks into L2 as it ends."""
    if not (x.is_cuda and gate_up.is_cuda and (bias is None or bias.is_cuda)):
        _need_cuda(x, gate_up, bias)
    mode = GLU_MODES.get(act)
    if mode is not None:
        rows = x.shape[0]
        if rows <= SMALL_M_MAX and _small_m_ok(x, gate_up, bias) and (gate_up.shape[0] // 2) % 8 == 0:
            M, (N, K) = rows, gate_up.shape
            out = torch.empty((M, N // 2), dtype=torch.bfloat16, device=x.device)
            code = _small_m(gate_up, x, bias, out, M, N, K, N // 2, mode, 0, ahead)
            _check(code, "gemm_small_m (gated)")
            return out
        if SMALL_M_MAX < rows <= STREAM_ROWS_SMALL:
            y = _gemm_stream(x, gate_up, bias, mode, torch.bfloat16)
            if y is not None:
                return y
        if rows <= ROWS_GLU_MAX_LARGE and x.dim() == 2 and not MID_GEMM and rows <= _rows_glu_max(gate_up.numel()):
            y = _gemm_rows(x, gate_up, bias, mode, torch.bfloat16)
            if y is not None:
                return y
        y = _tc_gemm(x, gate_up, bias, mode) if rows >= TC_GEMM_MIN_M else _tc_gemm_mid(x, gate_up, bias, mode)
        if y is not None:
            return y
    gu = torch.nn.functional.linear(x, gate_up, bias)
    if act == 0:
        return swiglu(gu)
    I = gate_up.shape[0] // 2
    out = torch.empty((x.shape[0], I), dtype=x.dtype, device=x.device)
    gated_act(gu[:, :I], gu[:, I:], out, act)
    return out


def linear_swiglu(x: torch.Tensor, gate_up: torch.Tensor, ahead: Optional[torch.Tensor] = None) -> torch.Tensor:
    """silu(x @ gate^T) * (x @ up^T): `linear_glu` without biases."""
    return linear_glu(x, gate_up, ahead=ahead)


# ---------------------------------------------------------------------------------------
# norms, convolutions, windowed and linear attention, gated activations (csrc/mixers.cu)
# ---------------------------------------------------------------------------------------
_mixers = None
ACT_SILU, ACT_GELU_TANH, ACT_SIGMOID, ACT_RELU2, ACT_RELU = 0, 1, 2, 3, 4
WINDOW_ATTENTION_ROWS = 8         # (token, head) rows of a block of the windowed attention kernel
CONV_MAX_TAPS = 16
WINDOW_ATTENTION_MAX_HEAD_DIM = 512
DECAY_ATTENTION_MAX_KEY_DIM = 512


def _mix_lib():
    global _mixers
    if _mixers is None:
        lib = _build.mixers_library()
        lib.msgl_dyntanh.argtypes = [c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_float, c_void_p, c_int, c_int,
                                     c_int, c_void_p]
        lib.msgl_conv_norm_kvwrite.argtypes = [c_void_p, c_ll, c_int, c_int, c_int, c_int, c_int, c_int, c_int] + [c_void_p] * 4 + \
            [c_float] + [c_void_p] * 8 + [c_int, c_int, c_int, c_int, c_int, c_void_p]
        lib.msgl_window_attention.argtypes = [c_void_p] * 6 + [c_int, c_int, c_int, c_void_p, c_int, c_void_p, c_ll, c_int,
                                              c_void_p, c_ll, c_int] + [c_int] * 9 + [c_float, c_float, c_int, c_void_p]
        lib.msgl_decay_attention.argtypes = [c_void_p, c_ll, c_int, c_int, c_int, c_int, c_int, c_int] + [c_void_p] * 5 + \
            [c_int, c_int, c_void_p]
        lib.msgl_rms_gate.argtypes = [c_void_p, c_int, c_void_p, c_float, c_void_p, c_ll, c_int, c_void_p, c_ll, c_int, c_float, c_int,
                                      c_int, c_void_p]
        lib.msgl_gated_act.argtypes = [c_void_p, c_ll, c_int, c_int, c_void_p, c_ll, c_int, c_int, c_int, c_int, c_int, c_void_p]
        lib.msgl_head_gate.argtypes = [c_void_p, c_void_p, c_ll, c_int, c_void_p, c_ll, c_int, c_int, c_int, c_float, c_int, c_int, c_void_p]
        lib.msgl_decay_attention_chunked.argtypes = [c_void_p, c_ll, c_int, c_int, c_int, c_int, c_int, c_int] + [c_void_p] * 6 + \
            [c_int, c_int, c_int, c_void_p]
        lib.msgl_scaled_embedding.argtypes = [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_float, c_int, c_void_p]
        lib.msgl_postnorm_residual.argtypes = [c_void_p, c_int, c_void_p, c_float, c_float, c_void_p, c_void_p, c_float, c_void_p, c_int,
                                               c_int, c_int, c_void_p]
        lib.msgl_latent_prep.argtypes = [c_void_p, c_ll, c_int, c_int, c_int, c_int, c_int, c_int, c_void_p, c_void_p, c_float, c_void_p,
                                         c_float, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p]
        lib.msgl_rope_heads.argtypes = [c_void_p, c_ll, c_int, c_int, c_void_p, c_int, c_int, c_int, c_int, c_int, c_void_p, c_float,
                                        c_void_p, c_int, c_int, c_void_p]
        lib.msgl_gate_mul.argtypes = [c_void_p, c_ll, c_void_p, c_ll, c_void_p, c_ll, c_int, c_int, c_int, c_int, c_void_p]
        lib.msgl_gated_decay_attention.argtypes = [c_void_p, c_ll, c_int, c_int, c_int, c_int, c_int, c_int, c_void_p, c_void_p, c_float,
                                                   c_float, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_void_p]
        lib.msgl_gated_decay_attention_chunked.argtypes = [c_void_p, c_ll, c_int, c_int, c_int, c_int, c_int, c_int, c_void_p, c_void_p,
                                                           c_float, c_float] + [c_void_p] * 7 + [c_int, c_int, c_int, c_void_p]
        lib.msgl_group_rms_gate.argtypes = [c_void_p, c_int, c_int, c_void_p, c_float, c_void_p, c_ll, c_void_p, c_ll, c_float, c_int,
                                            c_int, c_int, c_void_p]
        _mixers = lib
    return _mixers


def _rows_view(t: torch.Tensor, width: int, what: str) -> int:
    """A [T, width] view into packed rows: unit stride along the row; -> the row stride in elements."""
    assert t.dim() == 2 and t.shape[1] == width and (t.stride(1) == 1 or width == 1), f"{what}: [T, {width}] with unit stride wanted"
    return t.stride(0)


def dyntanh(weight: torch.Tensor, bias: torch.Tensor, alpha: float, *, x: Optional[torch.Tensor] = None,
            residual: Optional[torch.Tensor] = None, residual_out: Optional[torch.Tensor] = None,
            rows: Optional[torch.Tensor] = None, out_dtype: torch.dtype = torch.bfloat16) -> torch.Tensor:
    """y = tanh(alpha * v) * weight + bias with v = residual + x in float32 (either may be None); v goes to `residual_out`
    when it is given; `rows` (int32) picks the rows.  x: float32 or `out_dtype`; weight, bias: float32 [H]."""
    _need_cuda(weight, bias, x, residual, residual_out, rows)
    src = x if x is not None else residual
    assert src is not None and src.dim() == 2 and src.is_contiguous()
    H = src.shape[1]
    assert weight.dtype == torch.float32 and bias.dtype == torch.float32 and weight.numel() == H and bias.numel() == H
    if x is not None:
        assert x.dtype in (torch.float32, out_dtype) and x.is_contiguous()
    if residual is not None:
        assert residual.dtype == torch.float32 and residual.shape[1] == H and residual.is_contiguous()
    n_out = rows.numel() if rows is not None else src.shape[0]
    out = torch.empty((n_out, H), dtype=out_dtype, device=src.device)
    code = _mix_lib().msgl_dyntanh(_ptr(x), int(x is not None and x.dtype == torch.float32), _ptr(residual), _ptr(residual_out),
                                   _ptr(rows), _ptr(weight), _ptr(bias), float(alpha), _ptr(out), n_out, H, _DT[out_dtype], _stream())
    _check(code, "dyntanh")
    return out


def conv_norm_kvwrite(q_in: torch.Tensor, k_in: torch.Tensor, *, n_kv: int, head_dim: int, q_taps: torch.Tensor, k_taps: torch.Tensor,
                      q_norm: torch.Tensor, k_norm: torch.Tensor, eps: float, state: torch.Tensor, token_req: torch.Tensor,
                      q_start: torch.Tensor, slots: torch.Tensor, out_loc: Optional[torch.Tensor], k_cache: Optional[torch.Tensor],
                      v_cache: Optional[torch.Tensor], page_size: int, one_token: bool = False) -> torch.Tensor:
    """Short causal convolution over time on every channel of q_in [T, Cq] and k_in [T, Ck] (views into one packed
    projection) with taps q_taps [taps, Cq] and k_taps [taps, Ck] (float32, the oldest input's tap first), continued from `state` [slots, taps - 1, Cq + Ck] (the request's last inputs, which the call brings up to
    date), then an RMS norm over the whole of q and of k.  The normed k goes to `k_cache`, the un-normed k to `v_cache`
    (layout [page][kv head][slot][head_dim]) at token slots `out_loc`; the normed q comes back as [T, Cq].  one_token: every
    request brings exactly one token (the state is then brought up to date by the same launch)."""
    _need_cuda(q_in, k_in, q_taps, k_taps, q_norm, k_norm, state, token_req, q_start, slots, out_loc, k_cache, v_cache)
    T, Cq, Ck = q_in.shape[0], q_in.shape[1], k_in.shape[1]
    stride = _rows_view(q_in, Cq, "q")
    assert _rows_view(k_in, Ck, "k") == stride and q_in.dtype == k_in.dtype
    item = q_in.element_size()
    q_off = 0
    k_off = (k_in.data_ptr() - q_in.data_ptr()) // item
    taps = q_taps.shape[0]
    assert q_taps.shape == (taps, Cq) and k_taps.shape == (taps, Ck) and q_taps.dtype == torch.float32 and k_taps.dtype == torch.float32
    assert q_taps.is_contiguous() and k_taps.is_contiguous()
    assert q_norm.dtype == torch.float32 and k_norm.dtype == torch.float32 and q_norm.numel() == Cq and k_norm.numel() == Ck
    assert state.dtype == q_in.dtype and state.is_contiguous() and tuple(state.shape[1:]) == (max(taps - 1, 0), Cq + Ck)
    if k_cache is not None:
        assert k_cache.dtype == q_in.dtype and v_cache.dtype == q_in.dtype and out_loc is not None and out_loc.numel() == T
    q_out = torch.empty((T, Cq), dtype=q_in.dtype, device=q_in.device)
    B = q_start.numel() - 1
    code = _mix_lib().msgl_conv_norm_kvwrite(_ptr(q_in), stride, q_off, k_off, Cq, Ck, head_dim, n_kv, taps, _ptr(q_taps), _ptr(k_taps),
                                             _ptr(q_norm), _ptr(k_norm), float(eps), _ptr(state), _ptr(token_req), _ptr(q_start),
                                             _ptr(slots), _ptr(out_loc), _ptr(q_out), _ptr(k_cache), _ptr(v_cache), page_size, T, B,
                                             int(bool(one_token)), _dt(q_in), _stream())
    _check(code, f"conv_norm_kvwrite ({taps} taps)")
    global LAUNCHES
    LAUNCHES += int(taps > 1 and not (one_token and T == B))
    return q_out


def window_attention_geometry(n_q: int, n_kv: int) -> Tuple[int, int]:
    """(tokens per query tile, query heads of one kv head per block) of the windowed attention kernel."""
    G = n_q // n_kv
    gh = min(G, WINDOW_ATTENTION_ROWS)
    return WINDOW_ATTENTION_ROWS // gh, gh


def window_attention(q: torch.Tensor, out: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, *, q_start: torch.Tensor,
                     kv_len: torch.Tensor, block_table: torch.Tensor, n_kv: int, page_size: int, window: int, keep_first: int,
                     scale: float, q_lens: Optional[Sequence[int]], bias: Optional[torch.Tensor] = None,
                     gate: Optional[torch.Tensor] = None, out_scale: float = 1.0) -> None:
    """Causal softmax attention over the paged cache in which the query at position i sees key j if i - j < window or
    j < keep_first (window <= 0: every earlier key).  bias: float32 [heads, L], added to the scaled score by distance
    min(i - j, L - 1).  gate: [T, heads] (a view into packed rows): the head's output is multiplied by its sigmoid; out_scale
    multiplies everything.  q [T, heads, d]; out [T, heads * d] (may be a view into packed rows).  q_lens: the requests'
    numbers of tokens as the host knows them (they size the launch), or None when every request brings one token."""
    _need_cuda(q, out, k_cache, v_cache, q_start, kv_len, block_table, bias, gate)
    T, n_q, d = q.shape
    assert q.is_contiguous() and k_cache.dtype == q.dtype and v_cache.dtype == q.dtype and out.dtype == q.dtype
    out_stride = _rows_view(out, n_q * d, "out")
    B = kv_len.numel()
    QT, GH = window_attention_geometry(n_q, n_kv)
    if bias is not None:
        assert bias.dtype == torch.float32 and bias.dim() == 2 and bias.shape[0] == n_q and bias.is_contiguous()
    gate_stride = 0
    if gate is not None:
        assert gate.dtype == q.dtype
        gate_stride = _rows_view(gate, n_q, "gate")
    n_tiles = sum(-(-n // QT) for n in q_lens) if q_lens is not None else B
    code = _mix_lib().msgl_window_attention(
        _ptr(q), _ptr(k_cache), _ptr(v_cache), _ptr(q_start), _ptr(kv_len), _ptr(block_table), block_table.stride(0),
        int(q_lens is None), n_tiles,
        _ptr(bias), bias.shape[1] if bias is not None else 0, _ptr(gate), gate_stride, 0, _ptr(out), out_stride, 0,
        B, n_q, n_kv, d, page_size, int(window), int(keep_first), QT, GH, float(scale), float(out_scale), _dt(q), _stream())
    _check(code, f"window_attention (head size {d})")


DECAY_CHUNK = 64                 # tokens per chunk of the chunked form of the decaying linear attention
DECAY_CHUNKED_FROM = 16          # a step whose longest request brings this many tokens takes the chunked form


def head_gate(x: torch.Tensor, gate: Optional[torch.Tensor], out: torch.Tensor, scale: float = 1.0) -> None:
    """out[t, h, :] = x[t, h, :] * sigmoid(gate[t, h]) * scale; x [T, heads, d] contiguous, gate [T, heads] and out
    [T, heads * d] views into packed rows."""
    _need_cuda(x, gate, out)
    T, H, d = x.shape
    assert x.is_contiguous() and out.dtype == x.dtype
    gs = 0
    if gate is not None:
        assert gate.dtype == x.dtype
        gs = _rows_view(gate, H, "gate")
    code = _mix_lib().msgl_head_gate(_ptr(x), _ptr(gate), gs, 0, _ptr(out), _rows_view(out, H * d, "out"), 0, H, d, float(scale), T,
                                     _dt(x), _stream())
    _check(code, "head_gate")


def decay_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, *, heads: int, decay: torch.Tensor, state: torch.Tensor,
                    q_start: torch.Tensor, slots: torch.Tensor, q_lens: Optional[Sequence[int]] = None,
                    workspace=None) -> torch.Tensor:
    """Linear attention with a fixed decay per head over the step's tokens, continued from and written back to `state`
    [slots, heads, dk, dv] float32: S <- decay_h S + k v^T, o = S^T q with q, k, v = silu of the given projections
    ([T, heads * dk], [T, heads * dk], [T, heads * dv]: views into one packed projection).  -> float32 [T, heads * dv].
    q_lens: the requests' numbers of tokens as the host knows them; when the longest has DECAY_CHUNKED_FROM or more, the
    step is computed in chunks of DECAY_CHUNK tokens that run in parallel (the same sums in another order), else, and
    without q_lens, every request's tokens are walked in order.  workspace: a parts.Workspace for the chunks' states."""
    _need_cuda(q, k, v, decay, state, q_start, slots)
    T = q.shape[0]
    dk, dv = q.shape[1] // heads, v.shape[1] // heads
    stride = _rows_view(q, heads * dk, "q")
    assert _rows_view(k, heads * dk, "k") == stride and _rows_view(v, heads * dv, "v") == stride and q.dtype == k.dtype == v.dtype
    item = q.element_size()
    k_off, v_off = (k.data_ptr() - q.data_ptr()) // item, (v.data_ptr() - q.data_ptr()) // item
    assert decay.dtype == torch.float32 and decay.numel() == heads
    assert state.dtype == torch.float32 and state.is_contiguous() and tuple(state.shape[1:]) == (heads, dk, dv)
    out = torch.empty((T, heads * dv), dtype=torch.float32, device=q.device)
    B = q_start.numel() - 1
    if q_lens is not None and max(q_lens, default=0) >= DECAY_CHUNKED_FROM:
        n_chunks = sum(-(-n // DECAY_CHUNK) for n in q_lens)
        numel = n_chunks * heads * dk * dv
        U = workspace.get("decay_chunk_states", numel, torch.float32) if workspace is not None else \
            torch.empty(numel, dtype=torch.float32, device=q.device)
        code = _mix_lib().msgl_decay_attention_chunked(_ptr(q), stride, 0, k_off, v_off, heads, dk, dv, _ptr(decay), _ptr(state),
                                                       _ptr(q_start), _ptr(slots), _ptr(out), _ptr(U), n_chunks, B, _dt(q), _stream())
        _check(code, f"decay_attention in chunks (key size {dk})")
        global LAUNCHES
        LAUNCHES += 2
        return out
    code = _mix_lib().msgl_decay_attention(_ptr(q), stride, 0, k_off, v_off, heads, dk, dv, _ptr(decay), _ptr(state), _ptr(q_start),
                                           _ptr(slots), _ptr(out), B, _dt(q), _stream())
    _check(code, f"decay_attention (key size {dk})")
    return out


def rms_gate(x: torch.Tensor, weight: torch.Tensor, eps: float, gate: Optional[torch.Tensor], out: torch.Tensor, scale: float = 1.0) -> None:
    """out = x / sqrt(mean(x^2) + eps) * weight * sigmoid(gate) * scale; x float32 [T, N] contiguous, weight float32 [N],
    gate and out [T, N] views into packed rows of the activation type."""
    _need_cuda(x, weight, gate, out)
    T, N = x.shape
    assert x.dtype == torch.float32 and x.is_contiguous() and weight.dtype == torch.float32 and weight.numel() == N
    gs = _rows_view(gate, N, "gate") if gate is not None else 0
    if gate is not None:
        assert gate.dtype == out.dtype
    code = _mix_lib().msgl_rms_gate(_ptr(x), N, _ptr(weight), float(eps), _ptr(gate), gs, 0, _ptr(out), _rows_view(out, N, "out"), 0,
                                    float(scale), T, _dt(out), _stream())
    _check(code, "rms_gate")


def gated_act(gate: torch.Tensor, up: torch.Tensor, out: torch.Tensor, act: int) -> None:
    """out = act(gate) * up, act = ACT_SILU, ACT_GELU_TANH (0.5 z (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3)))), ACT_SIGMOID,
    ACT_RELU2 or ACT_RELU; all three [T, I] views into packed rows, gate and up in the same rows."""
    _need_cuda(gate, up, out)
    T, I = gate.shape
    stride = _rows_view(gate, I, "gate")
    assert _rows_view(up, I, "up") == stride and gate.dtype == up.dtype == out.dtype
    up_off = (up.data_ptr() - gate.data_ptr()) // gate.element_size()
    code = _mix_lib().msgl_gated_act(_ptr(gate), stride, 0, up_off, _ptr(out), _rows_view(out, I, "out"), 0, I, int(act), T, _dt(gate),
                                     _stream())
    _check(code, "gated_act")


def scaled_embedding(ids: torch.Tensor, table: torch.Tensor, scale: float) -> torch.Tensor:
    """ids int32 [T], table [V, H] -> float32 [T, H] = float(table[ids]) * scale."""
    _need_cuda(ids, table)
    T, (V, H) = ids.numel(), table.shape
    assert ids.dtype == torch.int32 and table.is_contiguous()
    out = torch.empty((T, H), dtype=torch.float32, device=table.device)
    _check(_mix_lib().msgl_scaled_embedding(_ptr(ids), _ptr(table), _ptr(out), T, H, V, float(scale), _dt(table), _stream()),
           "scaled_embedding")
    return out


def postnorm_residual(a: torch.Tensor, weight: torch.Tensor, eps: float, scale: float, residual: torch.Tensor, *,
                      next_weight: Optional[torch.Tensor] = None, next_eps: float = 0.0,
                      out_dtype: torch.dtype = torch.bfloat16) -> Optional[torch.Tensor]:
    """residual += scale * rmsnorm(a) * weight in float32, in place (a sublayer's output that is normed before it joins the
    stream); with `next_weight` also -> rmsnorm(residual) * next_weight in `out_dtype`, the next sublayer's input, from the same
    pass over the row.  a: [T, H] float32 or `out_dtype`; weights float32 [H]."""
    _need_cuda(a, weight, residual, next_weight)
    T, H = a.shape
    assert a.is_contiguous() and a.dtype in (torch.float32, out_dtype)
    assert residual.dtype == torch.float32 and residual.is_contiguous() and residual.shape == a.shape
    assert weight.dtype == torch.float32 and weight.numel() == H
    y = None
    if next_weight is not None:
        assert next_weight.dtype == torch.float32 and next_weight.numel() == H
        y = torch.empty((T, H), dtype=out_dtype, device=a.device)
    code = _mix_lib().msgl_postnorm_residual(_ptr(a), int(a.dtype == torch.float32), _ptr(weight), float(eps), float(scale),
                                             _ptr(residual), _ptr(next_weight), float(next_eps), _ptr(y), T, H, _DT[out_dtype], _stream())
    _check(code, "postnorm_residual")
    return y


def latent_prep(proj: torch.Tensor, *, dq_off: int, q_rank: int, dkv_off: int, kv_rank: int, rot_dim: int, rot_dims: int,
                dq_norm: Optional[torch.Tensor], dkv_norm: torch.Tensor, eps: float, freq: Optional[torch.Tensor], mag: float,
                positions: torch.Tensor, out_loc: Optional[torch.Tensor], cache: Optional[torch.Tensor],
                page_size: int) -> Optional[torch.Tensor]:
    """What a token of a latent attention leaves in the cache, and its query latent.  proj [T, .] holds the query's
    down-projection (q_rank columns at dq_off; q_rank = 0: none) and the key/value down-projection (kv_rank + rot_dim columns
    at dkv_off).  The cache row of a token (`cache` [pages, 1, page, kv_rank + rot_dim] at token slot out_loc) gets the RMS-normed
    latent followed by the last rot_dim columns, whose first rot_dims are rotated by position * freq (pairs i, i + rot_dims / 2;
    cos and sin times `mag`).  -> the RMS-normed query latent [T, q_rank], or None."""
    _need_cuda(proj, dq_norm, dkv_norm, freq, positions, out_loc, cache)
    T = proj.shape[0]
    assert proj.dim() == 2 and proj.stride(1) == 1 and dkv_off + kv_rank + rot_dim <= proj.shape[1]
    assert dkv_norm.dtype == torch.float32 and dkv_norm.numel() == kv_rank
    assert positions.dtype == torch.int32 and positions.numel() == T
    cq = None
    if q_rank:
        assert dq_norm is not None and dq_norm.dtype == torch.float32 and dq_norm.numel() == q_rank and dq_off + q_rank <= proj.shape[1]
        cq = torch.empty((T, q_rank), dtype=proj.dtype, device=proj.device)
    if rot_dims:
        assert freq is not None and freq.dtype == torch.float32 and freq.numel() == rot_dims // 2
    if cache is not None:
        assert cache.dtype == proj.dtype and cache.is_contiguous() and cache.shape[1] == 1 and cache.shape[3] == kv_rank + rot_dim
        assert out_loc is not None and out_loc.dtype == torch.int32 and out_loc.numel() == T
    code = _mix_lib().msgl_latent_prep(_ptr(proj), proj.stride(0), dq_off, dkv_off, q_rank, kv_rank, rot_dim, rot_dims, _ptr(dq_norm),
                                       _ptr(dkv_norm), float(eps), _ptr(freq), float(mag), _ptr(positions), _ptr(out_loc), _ptr(cq),
                                       _ptr(cache), page_size, T, _dt(proj), _stream())
    _check(code, "latent_prep")
    return cq


def rope_heads(src: torch.Tensor, src_off: int, dst: torch.Tensor, dst_off: int, *, rot_dim: int, rot_dims: int,
               freq: torch.Tensor, mag: float, positions: torch.Tensor) -> None:
    """dst[t, h, dst_off : dst_off + rot_dim] = the part src[t, h, src_off : src_off + rot_dim] of every head with its first
    rot_dims elements rotated by position * freq (pairs i, i + rot_dims / 2; cos and sin times `mag`).  src [T, heads, a] may be
    a view with a row stride of its own, dst [T, heads, b] is contiguous."""
    _need_cuda(src, dst, freq, positions)
    T, heads, sh = src.shape
    assert dst.is_contiguous() and dst.shape[:2] == src.shape[:2] and dst.dtype == src.dtype
    assert src.stride(2) == 1 and src.stride(1) == sh
    assert freq.dtype == torch.float32 and freq.numel() == rot_dims // 2 and positions.dtype == torch.int32
    code = _mix_lib().msgl_rope_heads(_ptr(src), src.stride(0), sh, src_off, _ptr(dst), dst.shape[2], dst_off, heads, rot_dim, rot_dims,
                                      _ptr(freq), float(mag), _ptr(positions), T, _dt(src), _stream())
    _check(code, "rope_heads")


def gate_mul(gate: torch.Tensor, x: torch.Tensor, out: torch.Tensor, act: int) -> None:
    """out = act(gate) * x with act = ACT_SIGMOID or ACT_SILU; [T, N] views into rows of their own strides."""
    _need_cuda(gate, x, out)
    T, N = x.shape
    assert gate.dtype == x.dtype == out.dtype
    code = _mix_lib().msgl_gate_mul(_ptr(gate), _rows_view(gate, N, "gate"), _ptr(x), _rows_view(x, N, "x"), _ptr(out),
                                    _rows_view(out, N, "out"), N, int(act), T, _dt(x), _stream())
    _check(code, "gate_mul")


GATED_DECAY_CHUNKED_FROM = 32    # a step whose longest request brings this many tokens takes the chunked form


def gated_decay_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, z: torch.Tensor, z_bias: torch.Tensor, *, heads: int,
                          tau: float, q_scale: float, state: torch.Tensor, q_start: torch.Tensor, slots: torch.Tensor,
                          q_lens: Optional[Sequence[int]] = None, workspace=None) -> torch.Tensor:
    """Linear attention whose decay comes from the input, per token and key channel, continued from and written back to `state`
    [slots, heads, dk, dv] float32: alpha = sigmoid(z + z_bias)^(1 / tau), S <- diag(alpha) S + k v^T, o = S^T (q * q_scale).
    q, k [T, heads * dk] and v [T, heads * dv] are views into one packed projection; z float32 [T, heads * dk] contiguous,
    z_bias float32 [heads * dk].  -> float32 [T, heads * dv].  q_lens: the requests' numbers of tokens as the host knows them
    (None: every request is walked token by token); when the longest has GATED_DECAY_CHUNKED_FROM or more, the step is computed
    in chunks of DECAY_CHUNK tokens that run in parallel (the same sums in another order).  workspace: a parts.Workspace for the
    chunks' scratch."""
    _need_cuda(q, k, v, z, z_bias, state, q_start, slots)
    T = q.shape[0]
    dk, dv = q.shape[1] // heads, v.shape[1] // heads
    stride = _rows_view(q, heads * dk, "q")
    assert _rows_view(k, heads * dk, "k") == stride and _rows_view(v, heads * dv, "v") == stride and q.dtype == k.dtype == v.dtype
    item = q.element_size()
    k_off, v_off = (k.data_ptr() - q.data_ptr()) // item, (v.data_ptr() - q.data_ptr()) // item
    assert z.dtype == torch.float32 and z.is_contiguous() and tuple(z.shape) == (T, heads * dk)
    assert z_bias.dtype == torch.float32 and z_bias.numel() == heads * dk
    assert state.dtype == torch.float32 and state.is_contiguous() and tuple(state.shape[1:]) == (heads, dk, dv)
    out = torch.empty((T, heads * dv), dtype=torch.float32, device=q.device)
    B = q_start.numel() - 1
    if q_lens is not None and max(q_lens, default=0) >= GATED_DECAY_CHUNKED_FROM:
        n_chunks = sum(-(-n // DECAY_CHUNK) for n in q_lens)
        sizes = (("gated_chunk_states", n_chunks * heads * dk * dv), ("gated_chunk_decays", T * heads * dk),
                 ("gated_chunk_weights", n_chunks * heads * DECAY_CHUNK * DECAY_CHUNK))
        U, bcum, P = (workspace.get(name, n, torch.float32) if workspace is not None else
                      torch.empty(n, dtype=torch.float32, device=q.device) for name, n in sizes)
        code = _mix_lib().msgl_gated_decay_attention_chunked(
            _ptr(q), stride, 0, k_off, v_off, heads, dk, dv, _ptr(z), _ptr(z_bias), float(tau), float(q_scale), _ptr(state),
            _ptr(q_start), _ptr(slots), _ptr(out), _ptr(U), _ptr(bcum), _ptr(P), n_chunks, B, _dt(q), _stream())
        _check(code, f"gated_decay_attention in chunks (key size {dk})")
        global LAUNCHES
        LAUNCHES += 4
        return out
    code = _mix_lib().msgl_gated_decay_attention(_ptr(q), stride, 0, k_off, v_off, heads, dk, dv, _ptr(z), _ptr(z_bias), float(tau),
                                                 float(q_scale), _ptr(state), _ptr(q_start), _ptr(slots), _ptr(out), B, _dt(q), _stream())
    _check(code, f"gated_decay_attention (key size {dk})")
    return out


def group_rms_gate(x: torch.Tensor, heads: int, weight: torch.Tensor, eps: float, gate: Optional[torch.Tensor], out: torch.Tensor,
                   act: int = ACT_SILU, scale: float = 1.0) -> None:
    """out[t, h, :] = x[t, h, :] / sqrt(mean(x[t, h, :]^2) + eps) * weight * act(gate[t, h, :]) * scale: an RMS norm over every
    head of a row with one weight [d] for all heads.  x float32 [T, heads * d] contiguous; gate and out [T, heads * d] views
    into packed rows of the activation type; act = ACT_SILU or ACT_SIGMOID."""
    _need_cuda(x, weight, gate, out)
    T, N = x.shape
    d = N // heads
    assert x.dtype == torch.float32 and x.is_contiguous() and N == heads * d and weight.dtype == torch.float32 and weight.numel() == d
    gs = 0
    if gate is not None:
        assert gate.dtype == out.dtype
        gs = _rows_view(gate, N, "gate")
    code = _mix_lib().msgl_group_rms_gate(_ptr(x), heads, d, _ptr(weight), float(eps), _ptr(gate), gs, _ptr(out),
                                          _rows_view(out, N, "out"), float(scale), int(act), T, _dt(out), _stream())
    _check(code, "group_rms_gate")


# ---------------------------------------------------------------------------------------
# sigmoid attention, gated recurrences, state-space scan, routed experts (csrc/mixers_gated.cu)
# ---------------------------------------------------------------------------------------
_gated = None
SIGMOID_ATTENTION_ROWS = 8          # (token, head) rows of a block of the sigmoid attention kernel
SIGMOID_ATTENTION_MAX_HEAD_DIM = 512
MINGRU_CHUNK = 32                   # tokens of a chunk when a long portion's recurrence runs in chunks side by side
SIGMOID_ATTENTION_MMA_ROWS = 64     # rows of a block of the tensor-core kernel
SIGMOID_ATTENTION_MMA_MAX_HEAD_DIM = 128
SIGMOID_ATTENTION_SPLIT_KEYS = 256  # keys of a piece when a one-token step cuts a request's keys over several blocks
SSM_MAX_STATE = 512
SSM_CHUNK = 64                      # tokens of a chunk when a long portion's state-space recurrence runs in chunks side by side
SSM_CHUNKED_FROM = 128              # the longest request's tokens from which a step runs in chunks
SSM_CHUNK_MAX_STATE = 256           # state sizes whose chunk tiles fit shared memory
ROUTE_MAX_EXPERTS, ROUTE_MAX_GROUPS = 1024, 64
EXPERTS_FEW_PAIRS = 64              # up to this many (token, choice) pairs the experts' products stream the weights


def _gated_lib():
    global _gated
    if _gated is None:
        lib = _build.gated_mixers_library()
        lib.msgl_embed_positions.argtypes = [c_void_p] * 5 + [c_int, c_int, c_int, c_int, c_float, c_int, c_void_p]
        lib.msgl_headnorm_kvwrite.argtypes = [c_void_p, c_ll] + [c_int] * 7 + [c_void_p, c_void_p, c_float, c_float, c_int] + \
            [c_void_p] * 5 + [c_int, c_int, c_int, c_void_p]
        lib.msgl_sigmoid_attention.argtypes = [c_void_p] * 6 + [c_int, c_int, c_int, c_void_p, c_int, c_void_p, c_ll, c_void_p] + \
            [c_int] * 11 + [c_float, c_int, c_void_p]
        lib.msgl_sigmoid_attention_mma.argtypes = [c_void_p] * 6 + [c_int, c_int, c_int, c_void_p, c_int, c_void_p, c_ll, c_void_p] + \
            [c_int] * 9 + [c_float, c_void_p]
        lib.msgl_mingru.argtypes = [c_void_p, c_ll, c_int, c_int, c_int, c_int] + [c_void_p] * 6 + [c_ll, c_float, c_int, c_int, c_void_p]
        lib.msgl_mingru_chunked.argtypes = [c_void_p, c_ll, c_int, c_int, c_int, c_int] + [c_void_p] * 6 + [c_ll, c_float, c_int, c_int, c_int,
                                            c_void_p, c_void_p, c_int, c_void_p]
        lib.msgl_pair_norm.argtypes = [c_void_p, c_void_p, c_int, c_void_p, c_void_p, c_float, c_float, c_void_p, c_int, c_int, c_void_p]
        lib.msgl_causal_conv_act.argtypes = [c_void_p, c_ll, c_int, c_int, c_int] + [c_void_p] * 7 + [c_int, c_int, c_int, c_int, c_void_p]
        lib.msgl_ssm_scan.argtypes = [c_void_p, c_int, c_int, c_int, c_int, c_void_p, c_ll, c_int] + [c_void_p] * 7 + [c_int, c_int, c_void_p]
        lib.msgl_ssm_scan_chunked.argtypes = [c_void_p, c_int, c_int, c_int, c_int, c_void_p, c_ll, c_int] + [c_void_p] * 7 + \
            [c_int, c_int, c_void_p, c_void_p, c_int, c_void_p]
        lib.msgl_gate_group_norm.argtypes = [c_void_p, c_int, c_int, c_void_p, c_float, c_void_p, c_ll, c_void_p, c_ll, c_float, c_int,
                                             c_int, c_void_p]
        lib.msgl_unary_act.argtypes = [c_void_p, c_ll, c_void_p, c_ll, c_int, c_int, c_float, c_int, c_int, c_void_p]
        lib.msgl_route.argtypes = [c_void_p, c_ll, c_void_p, c_void_p] + [c_int] * 5 + [c_void_p, c_void_p] + [c_int] * 5 + [c_void_p] * 3
        lib.msgl_plain_experts_few.argtypes = [c_void_p, c_ll] + [c_void_p] * 4 + [c_int] * 5 + [c_void_p] * 3 + [c_int, c_int, c_void_p]
        lib.msgl_expert_combine_self.argtypes = [c_void_p, c_int, c_void_p, c_void_p, c_int, c_int, c_void_p, c_ll, c_void_p, c_void_p, c_int,
                                                 c_int, c_void_p]
        lib.msgl_experts_few.argtypes = [c_void_p, c_ll] + [c_void_p] * 4 + [c_int, c_int, c_int, c_void_p, c_float, c_void_p, c_int, c_int,
                                                                            c_float, c_void_p, c_void_p, c_void_p]
        lib.msgl_clamped_glu.argtypes = [c_void_p, c_ll, c_int, c_float, c_void_p, c_int, c_int, c_void_p]
        lib.msgl_expert_rows.argtypes = [c_void_p, c_ll, c_void_p, c_int, c_int, c_int, c_int, c_int, c_void_p, c_void_p, c_void_p, c_int, c_void_p]
        lib.msgl_expert_order.argtypes = [c_void_p, c_int, c_int, c_void_p, c_void_p, c_void_p, c_void_p]
        lib.msgl_expert_gather.argtypes = [c_void_p, c_ll, c_void_p, c_int, c_int, c_void_p, c_int, c_int, c_void_p]
        lib.msgl_expert_combine.argtypes = [c_void_p, c_int, c_void_p, c_void_p, c_int, c_int, c_float, c_void_p, c_int, c_void_p, c_void_p,
                                            c_void_p]
        _gated = lib
    return _gated


def _col_off(view: torch.Tensor, base: torch.Tensor) -> int:
    """Column at which `view` starts inside the packed rows that `base` starts."""
    return (view.data_ptr() - base.data_ptr()) // base.element_size()


def embed_positions(ids: torch.Tensor, positions: torch.Tensor, table: torch.Tensor, places: torch.Tensor, scale: float) -> torch.Tensor:
    """ids, positions int32 [T]; table [V, H], places [P, H] -> float32 [T, H] = float(table[ids]) * scale + float(places[positions])."""
    _need_cuda(ids, positions, table, places)
    T, (V, H) = ids.numel(), table.shape
    assert ids.dtype == torch.int32 and positions.dtype == torch.int32 and table.is_contiguous() and places.is_contiguous()
    assert places.shape[1] == H and places.dtype == table.dtype
    out = torch.empty((T, H), dtype=torch.float32, device=table.device)
    _check(_gated_lib().msgl_embed_positions(_ptr(ids), _ptr(positions), _ptr(table), _ptr(places), _ptr(out), T, H, V, places.shape[0],
                                             float(scale), _dt(table), _stream()), "embed_positions")
    return out


def headnorm_kvwrite(q_in: torch.Tensor, k_in: torch.Tensor, v_in: torch.Tensor, *, n_q: int, n_kv: int, q_weight: torch.Tensor,
                     k_weight: torch.Tensor, eps: float, temp_coef: float, temp_every: int, positions: torch.Tensor,
                     out_loc: Optional[torch.Tensor], k_cache: Optional[torch.Tensor], v_cache: Optional[torch.Tensor],
                     page_size: int) -> torch.Tensor:
    """q_in [T, n_q * d], k_in [T, n_kv * d], v_in [T, n_kv * dv]: views into one packed projection.  Every head of q and of k is
    RMS-normed by itself with one weight [d] for all heads (float32); q is then multiplied by 1 + temp_coef * ln(floor((position +
    1) / temp_every) + 1) (temp_coef 0: not).  The normed k goes to `k_cache` [pages, n_kv, page, d], v as it is to `v_cache`
    [pages, n_kv, page, dv] at token slots `out_loc`; the q rows come back as [T, n_q, d]."""
    _need_cuda(q_in, k_in, v_in, q_weight, k_weight, positions, out_loc, k_cache, v_cache)
    T = q_in.shape[0]
    d, dv = q_in.shape[1] // n_q, v_in.shape[1] // n_kv
    stride = _rows_view(q_in, n_q * d, "q")
    assert _rows_view(k_in, n_kv * d, "k") == stride and _rows_view(v_in, n_kv * dv, "v") == stride and q_in.dtype == k_in.dtype == v_in.dtype
    assert q_weight.dtype == torch.float32 and k_weight.dtype == torch.float32 and q_weight.numel() == d and k_weight.numel() == d
    assert positions.dtype == torch.int32 and positions.numel() >= T
    if k_cache is not None:
        assert k_cache.dtype == q_in.dtype and v_cache.dtype == q_in.dtype and k_cache.is_contiguous() and v_cache.is_contiguous()
        assert tuple(k_cache.shape[1:]) == (n_kv, page_size, d) and tuple(v_cache.shape[1:]) == (n_kv, page_size, dv)
        assert out_loc is not None and out_loc.dtype == torch.int32 and out_loc.numel() >= T
    else:
        out_loc = None
    q_out = torch.empty((T, n_q, d), dtype=q_in.dtype, device=q_in.device)
    code = _gated_lib().msgl_headnorm_kvwrite(_ptr(q_in), stride, 0, _col_off(k_in, q_in), _col_off(v_in, q_in), n_q, n_kv, d, dv,
                                              _ptr(q_weight), _ptr(k_weight), float(eps), float(temp_coef), int(temp_every),
                                              _ptr(positions), _ptr(out_loc), _ptr(q_out), _ptr(k_cache), _ptr(v_cache), page_size, T,
                                              _dt(q_in), _stream())
    _check(code, "headnorm_kvwrite")
    return q_out


def sigmoid_attention_geometry(n_q: int, n_kv: int, tensor_cores: bool = False) -> Tuple[int, int]:
    """(tokens per query tile, query heads of one kv head per block) of the sigmoid attention kernels."""
    G = n_q // n_kv
    rows = SIGMOID_ATTENTION_MMA_ROWS if tensor_cores else SIGMOID_ATTENTION_ROWS
    gh = min(G, rows)
    return rows // gh, gh


def sigmoid_attention_on_tensor_cores(dtype: torch.dtype, d: int, dv: int) -> bool:
    """Whether the tensor-core kernel takes these rows: bfloat16, head sizes in steps of 8 up to 128."""
    return dtype == torch.bfloat16 and d % 8 == 0 and dv % 8 == 0 and max(d, dv) <= SIGMOID_ATTENTION_MMA_MAX_HEAD_DIM


def sigmoid_attention(q: torch.Tensor, out: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, *, q_start: torch.Tensor,
                      kv_len: torch.Tensor, block_table: torch.Tensor, n_kv: int, page_size: int, scale: float, bias: torch.Tensor,
                      q_lens: Optional[Sequence[int]], workspace=None, tensor_cores: Optional[bool] = None) -> None:
    """Causal attention over the paged cache whose weight of key j for the query at position i is sigmoid(q . k * scale +
    bias[head][min(i - j, L - 1)]), each key by itself (nothing is normed over the keys).  q [T, heads, d]; K cache [pages, n_kv,
    page, d], V cache [pages, n_kv, page, dv]; bias float32 [heads, L]; out [T, heads * dv] (may be a view into packed rows).
    q_lens: the requests' numbers of tokens as the host knows them (they size the launch), or None when every request brings one
    token: the keys are then cut into pieces of SIGMOID_ATTENTION_SPLIT_KEYS for as many blocks as the block table's width asks
    for, whose sums are added in order (workspace: a parts.Workspace for the pieces).  tensor_cores: None = the bfloat16 kernel
    with mma products where it takes the sizes (`sigmoid_attention_on_tensor_cores`), the float32 one elsewhere; False = the float32
    arithmetic kernel in any case."""
    _need_cuda(q, out, k_cache, v_cache, q_start, kv_len, block_table, bias)
    T, n_q, d = q.shape
    dv = v_cache.shape[3]
    assert q.is_contiguous() and k_cache.dtype == q.dtype and v_cache.dtype == q.dtype and out.dtype == q.dtype
    out_stride = _rows_view(out, n_q * dv, "out")
    B = kv_len.numel()
    if tensor_cores is None:
        tensor_cores = sigmoid_attention_on_tensor_cores(q.dtype, d, dv) and out_stride % 2 == 0 and out.data_ptr() % 4 == 0
    QT, GH = sigmoid_attention_geometry(n_q, n_kv, tensor_cores)
    assert bias.dtype == torch.float32 and bias.dim() == 2 and bias.shape[0] == n_q and bias.is_contiguous()
    uniform = q_lens is None
    n_tiles = B if uniform else sum(-(-n // QT) for n in q_lens)
    splits, part = 1, None
    if uniform:
        splits = max(1, -(-(block_table.shape[1] * page_size) // SIGMOID_ATTENTION_SPLIT_KEYS))
        if splits > 1:
            numel = splits * T * n_q * dv
            part = workspace.get("sigmoid_attention_pieces", numel, torch.float32) if workspace is not None else \
                torch.empty(numel, dtype=torch.float32, device=q.device)
    if tensor_cores:
        code = _gated_lib().msgl_sigmoid_attention_mma(
            _ptr(q), _ptr(k_cache), _ptr(v_cache), _ptr(q_start), _ptr(kv_len), _ptr(block_table), block_table.stride(0), int(uniform),
            n_tiles, _ptr(bias), bias.shape[1], _ptr(out), out_stride, _ptr(part), splits, SIGMOID_ATTENTION_SPLIT_KEYS, T, B, n_q,
            n_kv, d, dv, page_size, float(scale), _stream())
    else:
        code = _gated_lib().msgl_sigmoid_attention(
            _ptr(q), _ptr(k_cache), _ptr(v_cache), _ptr(q_start), _ptr(kv_len), _ptr(block_table), block_table.stride(0), int(uniform),
            n_tiles, _ptr(bias), bias.shape[1], _ptr(out), out_stride, _ptr(part), splits, SIGMOID_ATTENTION_SPLIT_KEYS, T, B, n_q, n_kv,
            d, dv, page_size, QT, GH, float(scale), _dt(q), _stream())
    _check(code, f"sigmoid_attention (head sizes {d}, {dv})")
    if splits > 1:
        global LAUNCHES
        LAUNCHES += 1


def mingru(z: torch.Tensor, x: torch.Tensor, g: torch.Tensor, z_bias: torch.Tensor, x_bias: torch.Tensor, *, state: torch.Tensor,
           q_start: torch.Tensor, slots: torch.Tensor, out: torch.Tensor, scale: float = 1.0, q_lens: Optional[Sequence[int]] = None,
           workspace=None) -> None:
    """A gated recurrence per channel over the step's tokens, continued from and written back to `state` [slots, W] float32:
    zz = sigmoid(z + z_bias), a = x + x_bias, c = a + 1/2 where a >= 0 and sigmoid(a) below, S <- (1 - zz) S + zz c;
    out = S * silu(g) * scale.  z, x, g [T, W]: views into one packed projection; out [T, W] (may be a view).  q_lens: the
    requests' numbers of tokens as the host knows them; with a request of 2 * MINGRU_CHUNK tokens or more the tokens run in chunks
    side by side (same sums in float32, another order), else one by one."""
    _need_cuda(z, x, g, z_bias, x_bias, state, q_start, slots, out)
    T, W = z.shape
    stride = _rows_view(z, W, "z")
    assert _rows_view(x, W, "x") == stride and _rows_view(g, W, "g") == stride and z.dtype == x.dtype == g.dtype == out.dtype
    assert z_bias.dtype == torch.float32 and x_bias.dtype == torch.float32 and z_bias.numel() == W and x_bias.numel() == W
    assert state.dtype == torch.float32 and state.is_contiguous() and tuple(state.shape[1:]) == (W,)
    B = q_start.numel() - 1
    if q_lens is not None and max(q_lens, default=0) >= 2 * MINGRU_CHUNK:
        L = MINGRU_CHUNK
        n_chunks = sum(-(-n // L) for n in q_lens)
        numel = (2 * n_chunks + B) * W
        buf = workspace.get("mingru_chunks", numel, torch.float32) if workspace is not None else \
            torch.empty(numel, dtype=torch.float32, device=z.device)
        code = _gated_lib().msgl_mingru_chunked(_ptr(z), stride, 0, _col_off(x, z), _col_off(g, z), W, _ptr(z_bias), _ptr(x_bias), _ptr(state),
                                                _ptr(q_start), _ptr(slots), _ptr(out), _rows_view(out, W, "out"), float(scale), B, L,
                                                n_chunks, _ptr(buf), _ptr(buf[2 * n_chunks * W:]), _dt(z), _stream())
        _check(code, "mingru (chunks)")
        global LAUNCHES
        LAUNCHES += 1
        return
    code = _gated_lib().msgl_mingru(_ptr(z), stride, 0, _col_off(x, z), _col_off(g, z), W, _ptr(z_bias), _ptr(x_bias), _ptr(state),
                                    _ptr(q_start), _ptr(slots), _ptr(out), _rows_view(out, W, "out"), float(scale), B, _dt(z), _stream())
    _check(code, "mingru")


def pair_norm(a: torch.Tensor, b: torch.Tensor, a_weight: torch.Tensor, b_weight: torch.Tensor, eps: float, scale: float) -> torch.Tensor:
    """-> float32 [T, H] = scale * (a / rms(a) * a_weight + b / rms(b) * b_weight), each row normed by itself; a, b [T, H] float32 or
    bfloat16 (both alike), weights float32 [H]."""
    _need_cuda(a, b, a_weight, b_weight)
    T, H = a.shape
    assert a.is_contiguous() and b.is_contiguous() and a.shape == b.shape and a.dtype == b.dtype
    assert a_weight.dtype == torch.float32 and b_weight.dtype == torch.float32 and a_weight.numel() == H and b_weight.numel() == H
    _dt(a)
    out = torch.empty((T, H), dtype=torch.float32, device=a.device)
    _check(_gated_lib().msgl_pair_norm(_ptr(a), _ptr(b), int(a.dtype == torch.float32), _ptr(a_weight), _ptr(b_weight), float(eps),
                                       float(scale), _ptr(out), T, H, _stream()), "pair_norm")
    return out


def causal_conv_act(x: torch.Tensor, taps: torch.Tensor, bias: Optional[torch.Tensor], *, state: Optional[torch.Tensor],
                    token_req: torch.Tensor, q_start: torch.Tensor, slots: torch.Tensor, act: int = ACT_SILU) -> torch.Tensor:
    """Short causal convolution over time on every channel of x [T, C] (a view into packed rows) with taps [K, C] (float32, the
    oldest input's tap first) and bias [C], then silu (act = ACT_SILU) or nothing (act < 0); continued from `state` [slots, K - 1,
    C] (the request's last inputs, oldest first), which the call brings up to date.  -> [T, C] contiguous."""
    _need_cuda(x, taps, bias, state, token_req, q_start, slots)
    T, C = x.shape
    K = taps.shape[0]
    assert taps.shape == (K, C) and taps.dtype == torch.float32 and taps.is_contiguous()
    if bias is not None:
        assert bias.dtype == torch.float32 and bias.numel() == C
    if K > 1:
        assert state is not None and state.dtype == x.dtype and state.is_contiguous() and tuple(state.shape[1:]) == (K - 1, C)
    out = torch.empty((T, C), dtype=x.dtype, device=x.device)
    B = q_start.numel() - 1
    code = _gated_lib().msgl_causal_conv_act(_ptr(x), _rows_view(x, C, "x"), 0, C, K, _ptr(taps), _ptr(bias), _ptr(state), _ptr(token_req),
                                             _ptr(q_start), _ptr(slots), _ptr(out), 0 if act == ACT_SILU else -1, T, B, _dt(x), _stream())
    _check(code, f"causal_conv_act ({K} taps)")
    if K > 1:
        global LAUNCHES
        LAUNCHES += 1
    return out


def ssm_scan(xbc: torch.Tensor, dt: torch.Tensor, *, heads: int, groups: int, state_size: int, dt_bias: torch.Tensor, a_log: torch.Tensor,
             skip: torch.Tensor, state: torch.Tensor, q_start: torch.Tensor, slots: torch.Tensor,
             q_lens: Optional[Sequence[int]] = None, workspace=None) -> torch.Tensor:
    """State-space recurrence per head over the step's tokens, continued from and written back to `state` [slots, heads, N, P]
    float32: step = softplus(dt + dt_bias), S <- exp(-exp(a_log) step) S + step B x^T, y = S^T C + skip x, with head h on group
    h // (heads / groups).  xbc [T, heads * P + 2 groups * N] contiguous = x | B | C; dt [T, heads] a view into packed rows.
    -> float32 [T, heads * P].  q_lens: the requests' numbers of tokens as the host knows them; when the longest has
    SSM_CHUNKED_FROM or more (and the state size is at most SSM_CHUNK_MAX_STATE) the step is computed in chunks of SSM_CHUNK tokens
    that run side by side (the same sums in float32, another order), else, and without q_lens, every request's tokens are walked in
    order.  workspace: a parts.Workspace for the chunks' states."""
    _need_cuda(xbc, dt, dt_bias, a_log, skip, state, q_start, slots)
    T = xbc.shape[0]
    N = state_size
    P = (xbc.shape[1] - 2 * groups * N) // heads
    assert xbc.is_contiguous() and xbc.shape[1] == heads * P + 2 * groups * N and dt.dtype == xbc.dtype
    for w in (dt_bias, a_log, skip):
        assert w.dtype == torch.float32 and w.numel() == heads
    assert state.dtype == torch.float32 and state.is_contiguous() and tuple(state.shape[1:]) == (heads, N, P)
    y = torch.empty((T, heads * P), dtype=torch.float32, device=xbc.device)
    B = q_start.numel() - 1
    if q_lens is not None and max(q_lens, default=0) >= SSM_CHUNKED_FROM and N <= SSM_CHUNK_MAX_STATE:
        n_chunks = sum(-(-n // SSM_CHUNK) for n in q_lens)
        numel = n_chunks * heads * (N * P + 1)
        buf = workspace.get("ssm_chunk_states", numel, torch.float32) if workspace is not None else \
            torch.empty(numel, dtype=torch.float32, device=xbc.device)
        code = _gated_lib().msgl_ssm_scan_chunked(_ptr(xbc), heads, groups, N, P, _ptr(dt), _rows_view(dt, heads, "dt"), 0, _ptr(dt_bias),
                                                  _ptr(a_log), _ptr(skip), _ptr(state), _ptr(q_start), _ptr(slots), _ptr(y), B, n_chunks,
                                                  _ptr(buf), _ptr(buf[n_chunks * heads * N * P:]), _dt(xbc), _stream())
        _check(code, f"ssm_scan in chunks (state size {N})")
        global LAUNCHES
        LAUNCHES += 2
        return y
    code = _gated_lib().msgl_ssm_scan(_ptr(xbc), heads, groups, N, P, _ptr(dt), _rows_view(dt, heads, "dt"), 0, _ptr(dt_bias), _ptr(a_log),
                                      _ptr(skip), _ptr(state), _ptr(q_start), _ptr(slots), _ptr(y), B, _dt(xbc), _stream())
    _check(code, f"ssm_scan (state size {N})")
    return y


def gate_group_norm(y: torch.Tensor, gate: torch.Tensor, weight: torch.Tensor, parts: int, eps: float, out: torch.Tensor,
                    scale: float = 1.0) -> None:
    """out = v / rms(v) * weight * scale with v = y * silu(gate) and the root mean square taken over each of `parts` equal parts of
    the row by itself (the gate comes before the norm).  y float32 [T, N] contiguous; gate and out [T, N] views into packed rows of
    the activation type; weight float32 [N]."""
    _need_cuda(y, gate, weight, out)
    T, N = y.shape
    assert y.dtype == torch.float32 and y.is_contiguous() and weight.dtype == torch.float32 and weight.numel() == N and gate.dtype == out.dtype
    code = _gated_lib().msgl_gate_group_norm(_ptr(y), N, int(parts), _ptr(weight), float(eps), _ptr(gate), _rows_view(gate, N, "gate"),
                                             _ptr(out), _rows_view(out, N, "out"), float(scale), T, _dt(out), _stream())
    _check(code, "gate_group_norm")


def unary_act(x: torch.Tensor, act: int, scale: float = 1.0, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """act(x) * scale, element by element; act = ACT_SILU, ACT_GELU_TANH, ACT_SIGMOID, ACT_RELU2 (relu(x)^2) or ACT_RELU."""
    _need_cuda(x, out)
    T, N = x.shape
    if out is None:
        out = torch.empty((T, N), dtype=x.dtype, device=x.device)
    assert out.dtype == x.dtype
    code = _gated_lib().msgl_unary_act(_ptr(x), _rows_view(x, N, "x"), _ptr(out), _rows_view(out, N, "out"), N, int(act), float(scale), T,
                                       _dt(x), _stream())
    _check(code, "unary_act")
    return out


ROUTE_SCORES = {"sigmoid": 0, "logits": 1, "softmax": 2}


def route(h: torch.Tensor, router: torch.Tensor, correction: Optional[torch.Tensor], *, n_groups: int, keep: int,
          top: int, score: str = "sigmoid", group_score: str = "top2", renormalize: bool = True,
          gate_row: Optional[torch.Tensor] = None):
    """The experts a token uses and their weights.  Scores s = sigmoid(router h), or with score = "softmax" the softmax of the
    logits over all E outputs, in float32; the choice goes by s + correction among the experts of the `keep` best of `n_groups`
    equal groups of neighbouring experts (a group counts by the sum of its two largest choice scores, or with group_score = "max"
    by the largest), the `top` largest win; the weights are the winners' s, over their sum unless renormalize = False.
    h [T, H], router [E, H] -> (int32 [T, top], float32 [T, top]).
    score = "logits": the logits router h themselves are what the choice goes by (the largest win, the lower index at a tie), and
    the weights are the softmax over the chosen logits only.  gate_row [H]: one more row that is no expert.  With either of
    the two the call returns a third item, float32 [T] = sigmoid(gate_row . h) or None."""
    _need_cuda(h, router, correction, gate_row)
    T, H = h.shape
    E = router.shape[0]
    assert router.shape == (E, H) and router.is_contiguous() and router.dtype == h.dtype
    assert group_score in ("top2", "max")
    if correction is not None:
        assert correction.dtype == torch.float32 and correction.numel() == E
    idx = torch.empty((T, top), dtype=torch.int32, device=h.device)
    wts = torch.empty((T, top), dtype=torch.float32, device=h.device)
    gate_out = None
    if gate_row is not None:
        assert gate_row.dtype == h.dtype and gate_row.numel() == H and gate_row.is_contiguous()
        gate_out = torch.empty(T, dtype=torch.float32, device=h.device)
    code = _gated_lib().msgl_route(_ptr(h), _rows_view(h, H, "h"), _ptr(router), _ptr(correction), H, E, int(n_groups), int(keep),
                                   int(top), _ptr(idx), _ptr(wts), T, _dt(h), ROUTE_SCORES[score], int(group_score == "max"),
                                   int(bool(renormalize)), _ptr(gate_row), _ptr(gate_out), _stream())
    _check(code, f"route ({E} experts)")
    if score == "logits" or gate_row is not None:
        return idx, wts, gate_out
    return idx, wts


def plain_experts_few(h: torch.Tensor, up: torch.Tensor, down: torch.Tensor, idx: torch.Tensor, wts: torch.Tensor, act: int,
                      extra: Optional[torch.Tensor] = None) -> torch.Tensor:
    """-> float32 [T, H] = sum_k wts[t, k] * y_k + extra[t] for experts without a gate: y_k = down[e] act(up[e] h_t), e = idx[t, k],
    the chosen experts' rows read straight from the stacked weights up [E, F, H] and down [E, H, F]; e >= E stands for the input
    itself, y_k = h_t.  For a few tokens.  act: one of the ACT_ numbers; extra: float32 [T, H] (a shared expert's output)."""
    _need_cuda(h, up, down, idx, wts, extra)
    T, H = h.shape
    E, F, _ = up.shape
    top = idx.shape[1]
    assert up.shape == (E, F, H) and down.shape == (E, H, F) and up.is_contiguous() and down.is_contiguous()
    assert up.dtype == down.dtype == h.dtype
    assert idx.dtype == torch.int32 and wts.dtype == torch.float32 and idx.is_contiguous() and wts.is_contiguous()
    if extra is not None:
        assert extra.dtype == torch.float32 and extra.is_contiguous() and tuple(extra.shape) == (T, H)
    a = torch.empty((T * top, F), dtype=h.dtype, device=h.device)
    out = torch.empty((T, H), dtype=torch.float32, device=h.device)
    code = _gated_lib().msgl_plain_experts_few(_ptr(h), _rows_view(h, H, "h"), _ptr(up), _ptr(down), _ptr(idx), _ptr(wts), top, E, H, F,
                                               int(act), _ptr(a), _ptr(extra), _ptr(out), T, _dt(h), _stream())
    _check(code, "plain_experts_few")
    global LAUNCHES
    LAUNCHES += 1
    return out


def expert_combine_self(y: torch.Tensor, place: torch.Tensor, wts: torch.Tensor, h: torch.Tensor,
                        extra: Optional[torch.Tensor] = None) -> torch.Tensor:
    """-> float32 [T, H] = extra[t] + sum_k wts[t, k] * (y[place[t * top + k]], or h[t] where that place is -1)."""
    _need_cuda(y, place, wts, h, extra)
    T, top = wts.shape
    H = y.shape[1]
    assert y.is_contiguous() and y.dtype in (torch.float32, h.dtype) and wts.dtype == torch.float32 and wts.is_contiguous()
    assert h.shape == (T, H) and place.numel() == T * top
    if extra is not None:
        assert extra.dtype == torch.float32 and extra.is_contiguous() and tuple(extra.shape) == (T, H)
    out = torch.empty((T, H), dtype=torch.float32, device=y.device)
    _check(_gated_lib().msgl_expert_combine_self(_ptr(y), int(y.dtype == torch.float32), _ptr(place), _ptr(wts), top, H, _ptr(h),
                                                 _rows_view(h, H, "h"), _ptr(extra), _ptr(out), T, _dt(h), _stream()), "expert_combine_self")
    return out


def _expert_operands(h: torch.Tensor, gate_up: torch.Tensor, down: torch.Tensor, idx: torch.Tensor, wts: torch.Tensor,
                     extra: Optional[torch.Tensor], extra_gate: Optional[torch.Tensor]) -> Tuple[torch.Tensor, torch.Tensor]:
    """What every kernel of the routed experts is told by addresses and sizes alone has to lie as they read it: raises, or returns idx and wts of h's tokens,
    both [T, top]."""
    _need_cuda(h, gate_up, down, idx, wts, extra, extra_gate)
    if extra is not None:
        assert extra.dtype == torch.float32 and extra.is_contiguous() and tuple(extra.shape) == tuple(h.shape)
        assert extra_gate is None or (extra_gate.dtype == torch.float32 and extra_gate.numel() == h.shape[0])
    T, H = h.shape
    E, _, F, _ = gate_up.shape
    assert gate_up.shape == (E, 2, F, H) and down.shape == (E, H, F)
    assert gate_up.is_contiguous() and down.is_contiguous() and gate_up.dtype == down.dtype == h.dtype
    assert idx.dtype == torch.int32 and wts.dtype == torch.float32 and idx.is_contiguous() and wts.is_contiguous()
    if idx.shape[0] != T or wts.shape != idx.shape:           # more rows than tokens, weights in one row: the first numbers count
        top = idx.shape[1]
        assert idx.shape[0] >= T and wts.numel() >= T * top
        idx, wts = idx[:T], wts.view(-1)[:T * top].view(T, top)
    return idx, wts


def experts_few(h: torch.Tensor, gate_up: torch.Tensor, down: torch.Tensor, idx: torch.Tensor, wts: torch.Tensor,
                scale: float = 1.0, limit: float = 0.0, extra: Optional[torch.Tensor] = None,
                extra_gate: Optional[torch.Tensor] = None) -> torch.Tensor:
    """-> float32 [T, H] = scale * sum_k wts[t, k] * down[e] (silu(gate[e] h_t) * (up[e] h_t)), e = idx[t, k], with the chosen
    experts' rows read straight from the stacked weights gate_up [E, 2, F, H] (an expert's gate, then its up) and down [E, H, F]:
    for decode steps and a few tokens, in bfloat16 by the grouped decode-batch product but for very small experts
    (`_experts_grouped`).  limit > 0: the activation is g * sigmoid(1.702 g) * (u + 1) with g = min(gate, limit) and
    u = clamp(up, -limit, limit).  extra float32 [T, H] (a shared expert's output) is added inside the sum, times
    extra_gate float32 [T] where given."""
    idx, wts = _expert_operands(h, gate_up, down, idx, wts, extra, extra_gate)
    T, H = h.shape
    F, top = gate_up.shape[2], idx.shape[1]
    out = _experts_by_rows(h, gate_up, down, idx, wts, scale, limit, extra, extra_gate, torch.float32) if _experts_grouped(T * top, F * H) else None
    if out is not None:
        return out
    act = torch.empty((T * top, F), dtype=h.dtype, device=h.device)
    out = torch.empty((T, H), dtype=torch.float32, device=h.device)
    code = _gated_lib().msgl_experts_few(_ptr(h), _rows_view(h, H, "h"), _ptr(gate_up), _ptr(down), _ptr(idx), _ptr(wts), top, H, F,
                                         _ptr(act), float(scale), _ptr(out), T, _dt(h), float(limit), _ptr(extra),
                                         _ptr(extra_gate) if extra is not None else None, _stream())
    _check(code, "experts_few")
    global LAUNCHES
    LAUNCHES += 1
    return out


def experts_few_shared(h: torch.Tensor, gate_up: torch.Tensor, down: torch.Tensor, idx: torch.Tensor, wts: torch.Tensor, shared_gate_up: torch.Tensor,
                       shared_down: torch.Tensor, shared_gate: torch.Tensor, limit: float) -> Optional[torch.Tensor]:
    """`experts_few` with limit > 0 beside a shared expert of the experts' own sizes, shared_gate_up [2 F, H] and shared_down [H, F], whose output counts shared_gate [T] times: in the
    same grouped launches, as one more expert that every token uses.  None where these do not apply or the tokens are more than a run of rows."""
    T, H = h.shape
    F, top = gate_up.shape[2], idx.shape[1]
    if (T > SHARED_ROWS_MAX or limit <= 0 or not _experts_grouped(T * top, F * H) or tuple(shared_gate_up.shape) != (2 * F, H) or tuple(shared_down.shape) != (H, F)
            or shared_gate_up.dtype != h.dtype or shared_down.dtype != h.dtype or not shared_gate_up.is_contiguous() or not shared_down.is_contiguous()
            or (shared_gate_up.data_ptr() | shared_down.data_ptr()) % 16 or shared_gate.dtype != torch.float32 or shared_gate.numel() != T):
        return None
    _need_cuda(shared_gate_up, shared_down, shared_gate)
    idx, wts = _expert_operands(h, gate_up, down, idx, wts, None, None)
    return _experts_by_rows(h, gate_up, down, idx, wts, 1.0, limit, None, shared_gate, torch.float32, (shared_gate_up, shared_down))


# us of the whole mixture (32 experts of [2 x 1536, 2048] + [2048, 1536], four a token), shared expert as launches of its own / in the grouped ones: 1 token 45.3 / 38.7, 8: 92.7 / 85.7, 16: 117.4 / 107.5,
# 64: 132.0 / 124.0, 128: 135.3 / 127.6.  Over nine mixtures (8 to 256 experts of 256 to 1,536, two to eight a token) at 1 to 128 tokens 1.13 times as fast in the mean, the worst 0.99.  The line is the largest batch
# that is replayed as a graph, not where the gain ends: decode steps of 160 to 256 tokens were measured 1.00 to 1.31 times as fast but for one of 27 (8 experts, 256 tokens: 66.5 / 72.0).
SHARED_ROWS_MAX = 128


# The chosen experts' products on the decode-batch kernel (csrc/gemm_rows.cu, grouped: an expert's weights are read once, whatever the
# number of tokens that chose it) against the others, measured on B200: a feed-forward of 32 experts of [2 x 1536, 2048] + [2048, 1536], four
# a token, beside a shared one.  Against a warp per row and (token, choice) pair: 1 token 82 -> 66 us, 8 tokens 224 -> 106, 24 tokens
# 528 -> 132, 128 tokens 2,516 -> 140.  Against the library's grouped product with the activation between: 300 tokens 230 -> 156,
# 700 tokens 247 -> 184, 1,024 tokens (128 rows an expert) 267 -> 214; with 150 rows an expert its products take 178 us, the library's
# 145: such tiles leave one block an SM.  Those are random choices; without the shared expert and the router, library / this kernel: 700
# tokens, Zipf-distributed choices (exponent 1.2) 181 / 157, all tokens at the same four experts 92 / 107; 1,024 tokens 209 / 177 and 111 / 139.
EXPERT_ROWS_MEAN_MAX = 128
EXPERT_ROWS_MAX_PAIRS = 8192
# Very small experts in decode steps: the two launches per pair are ahead of the grouped product's four until the pairs' weights add up.  Experts
# of 512 x 128, two of eight a token, cold: 1 token 6.4 / 12.3 us, 32 tokens 12.3 / 13.4, 64 tokens 19.8 / 14.0; 1,024 x 256, six of 64: 1 token 18.1 /
# 16.4, 8 tokens 38 / 26; 2,048 x 512, two of eight: 1 token 29 / 20 (all weights in L2 already: 14.5 / 16 and 15.5 / 17.5 us at one token).
EXPERT_ROWS_MIN_WEIGHTS, EXPERT_ROWS_MIN_WORK = 200_000, 5_000_000      # elements of one matrix of an expert; the same times pairs


def _experts_grouped(pairs: int, weights: int) -> bool:
    return weights >= EXPERT_ROWS_MIN_WEIGHTS or pairs * weights >= EXPERT_ROWS_MIN_WORK


def expert_rows(h: torch.Tensor, idx: torch.Tensor, n_experts: int) -> Optional[Tuple[torch.Tensor, torch.Tensor, torch.Tensor]]:
    """idx int32 [T, top], numbers below n_experts -> (rows [T * top, H]: every token's row once per expert it uses, in the order of the experts,
    pairs of one expert in their own order; place int32 [T * top]: row of every pair; ends int32 [n_experts]: running sum of the experts'
    rows) in one launch; None where the sizes are not the kernel's (see `expert_order`, `expert_gather`)."""
    _need_cuda(h, idx)
    T, H = h.shape
    top = idx.shape[1]
    V = 16 // h.element_size()
    if T * top > EXPERT_ROWS_MAX_PAIRS or H % V or h.stride(0) % V or h.stride(1) != 1 or h.data_ptr() % 16 or n_experts > ROUTE_MAX_EXPERTS:
        return None
    assert idx.dtype == torch.int32 and idx.is_contiguous() and idx.shape[0] == T
    rows = torch.empty((T * top, H), dtype=h.dtype, device=h.device)
    place = torch.empty(T * top, dtype=torch.int32, device=h.device)
    ends = torch.empty(n_experts, dtype=torch.int32, device=h.device)
    _check(_gated_lib().msgl_expert_rows(_ptr(h), h.stride(0), _ptr(idx), T * top, top, n_experts, H, 0, _ptr(rows), _ptr(place), _ptr(ends), _dt(h),
                                         _stream()), "expert_rows")
    return rows, place, ends


def _experts_by_rows(h: torch.Tensor, gate_up: torch.Tensor, down: torch.Tensor, idx: torch.Tensor, wts: torch.Tensor, scale: float, limit: float,
                     extra: Optional[torch.Tensor], extra_gate: Optional[torch.Tensor], y_dtype: torch.dtype,
                     shared: Optional[Tuple[torch.Tensor, torch.Tensor]] = None) -> Optional[torch.Tensor]:
    """The chosen experts, gate_up [E, 2, F, H] and down [E, H, F], on the decode-batch kernel: `expert_rows`, both products with the activation
    between them, `expert_combine`; None where that does not apply.  shared = ([2 F, H], [H, F]) in place of extra, y_dtype float32: one more expert that every token uses.  The operands have been through `_expert_operands`.  The ranges of K, and
    with them the order of the sums, follow from the sizes: float32 outputs of the experts (decode steps) take those of a single token's
    step, so that a request's tokens are the same in every batch, rounded ones those of a step that uses all experts.  (One
    function and three scratch tensors for the four launches: small eager steps wait for the host.)"""
    T, H = h.shape
    E, _, F, _ = gate_up.shape
    top = idx.shape[1]
    P = T * top
    if h.dtype != torch.bfloat16 or H % 8 or F % 8 or P > EXPERT_ROWS_MEAN_MAX * E or P > EXPERT_ROWS_MAX_PAIRS or E > ROUTE_MAX_EXPERTS or \
            h.stride(1) != 1 or h.stride(0) % 8 or (h.data_ptr() | gate_up.data_ptr() | down.data_ptr()) % 16 or not tensor_maps():
        return None
    dev, R = h.device, P if shared is None else P + T          # R: rows of x and y
    numbers, buf = torch.empty(P + E + 1, dtype=torch.int32, device=dev), torch.empty(R * (H + F), dtype=torch.bfloat16, device=dev)
    y, out = torch.empty(R * H, dtype=y_dtype, device=dev), torch.empty((T, H), dtype=torch.float32, device=dev)
    place, rows, yp = numbers.data_ptr(), buf.data_ptr(), y.data_ptr()
    ends, act = place + 4 * P, rows + 2 * R * H
    gu_apart, down_apart = (None, None) if shared is None else (shared[0].data_ptr(), shared[1].data_ptr())
    f32, status, stream, lib, gated = int(y_dtype == torch.float32), _status_tensor(dev).data_ptr(), _stream(), _lib(), _gated_lib()
    ranges = -1 if f32 else 0
    _check(gated.msgl_expert_rows(h.data_ptr(), h.stride(0), idx.data_ptr(), P, top, E, H, R - P, rows, place, ends, _DT[torch.bfloat16], stream), "expert_rows")
    code = lib.msgl_gemm_rows_apart(gate_up.data_ptr(), gu_apart, rows, None, act, P, F, H, H, F, 3 if limit > 0 else 1, 0, float(limit), E, ends, T, ranges, 0, status, stream)
    if code == 2:             # no tensor map of this layout
        return None
    _check(code, "gemm_rows (experts)")
    _check(lib.msgl_gemm_rows_apart(down.data_ptr(), down_apart, act, None, yp, P, H, F, F, H, 0, f32, 0.0, E, ends, T, ranges, 0, status, stream), "gemm_rows (experts)")
    more = _ptr(extra) if shared is None else yp + 4 * P * H
    _check(gated.msgl_expert_combine(yp, f32, place, wts.data_ptr(), top, H, float(scale), out.data_ptr(), T, more,
                                     _ptr(extra_gate) if more is not None else None, stream), "expert_combine")
    return out


def experts_many(h: torch.Tensor, gate_up: torch.Tensor, down: torch.Tensor, idx: torch.Tensor, wts: torch.Tensor, scale: float = 1.0,
                 limit: float = 0.0, extra: Optional[torch.Tensor] = None, extra_gate: Optional[torch.Tensor] = None) -> Optional[torch.Tensor]:
    """`experts_few` for the tokens of a prompt portion (the experts' outputs are rounded to the activation type before they are
    summed): None where the decode-batch kernel does not apply or the library's grouped product is ahead."""
    idx, wts = _expert_operands(h, gate_up, down, idx, wts, extra, extra_gate)
    return _experts_by_rows(h, gate_up, down, idx, wts, scale, limit, extra, extra_gate, h.dtype)


def expert_order(idx: torch.Tensor, n_experts: int) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """idx int32 [T, top] -> (counts int32 [E]: pairs per expert; ends int32 [E]: their running sum; place int32 [T * top]: row of every (token, choice) pair when the
    pairs are put in the order of their experts, pairs of one expert in their own order; -1 for a pair whose number is n_experts
    or more, which has no row)."""
    _need_cuda(idx)
    assert idx.dtype == torch.int32 and idx.is_contiguous()
    counts = torch.empty(n_experts, dtype=torch.int32, device=idx.device)
    ends = torch.empty(n_experts, dtype=torch.int32, device=idx.device)
    place = torch.empty(idx.numel(), dtype=torch.int32, device=idx.device)
    _check(_gated_lib().msgl_expert_order(_ptr(idx), idx.numel(), n_experts, _ptr(counts), _ptr(place), _ptr(ends), _stream()), "expert_order")
    global LAUNCHES
    LAUNCHES += 1
    return counts, ends, place


def expert_gather(h: torch.Tensor, place: torch.Tensor, top: int) -> torch.Tensor:
    """rows[place[t * top + k]] = h[t]: every token's row once per expert it uses, in expert order (places below 0: no row)."""
    _need_cuda(h, place)
    T, H = h.shape
    rows = torch.empty((T * top, H), dtype=h.dtype, device=h.device)
    _check(_gated_lib().msgl_expert_gather(_ptr(h), _rows_view(h, H, "h"), _ptr(place), top, H, _ptr(rows), T * top, _dt(h), _stream()),
           "expert_gather")
    return rows


def clamped_glu(gate_up: torch.Tensor, limit: float) -> torch.Tensor:
    """[T, 2F] (gate first) -> [T, F] = g * sigmoid(1.702 g) * (u + 1) with g = min(gate, limit), u = clamp(up, -limit, limit)."""
    _need_cuda(gate_up)
    T, F = gate_up.shape[0], gate_up.shape[1] // 2
    assert gate_up.dim() == 2 and gate_up.shape[1] == 2 * F
    out = torch.empty((T, F), dtype=gate_up.dtype, device=gate_up.device)
    _check(_gated_lib().msgl_clamped_glu(_ptr(gate_up), _rows_view(gate_up, 2 * F, "gate_up"), F, float(limit), _ptr(out), T, _dt(gate_up),
                                         _stream()), "clamped_glu")
    return out


def expert_combine(y: torch.Tensor, place: torch.Tensor, wts: torch.Tensor, scale: float = 1.0, extra: Optional[torch.Tensor] = None,
                   extra_gate: Optional[torch.Tensor] = None) -> torch.Tensor:
    """-> float32 [T, H] = scale * (sum_k wts[t, k] * y[place[t * top + k]] + extra_gate[t] * extra[t]); y [T * top, H] float32 or
    bfloat16; extra float32 [T, H] and extra_gate float32 [T] are optional (no gate: the extra term counts fully)."""
    _need_cuda(y, place, wts, extra, extra_gate)
    if extra is not None:
        assert extra.dtype == torch.float32 and extra.is_contiguous() and extra.shape[1] == y.shape[1]
        assert extra_gate is None or (extra_gate.dtype == torch.float32 and extra_gate.numel() == wts.shape[0])
    T, top = wts.shape
    H = y.shape[1]
    assert y.is_contiguous() and y.shape[0] == T * top and wts.dtype == torch.float32 and wts.is_contiguous()
    _dt(y)
    out = torch.empty((T, H), dtype=torch.float32, device=y.device)
    _check(_gated_lib().msgl_expert_combine(_ptr(y), int(y.dtype == torch.float32), _ptr(place), _ptr(wts), top, H, float(scale), _ptr(out),
                                            T, _ptr(extra), _ptr(extra_gate) if extra is not None else None, _stream()), "expert_combine")
    return out


# ---------------------------------------------------------------------------------------
# attention with a sink, the gated delta rule, scaled sums and the per-layer token input (csrc/mixers_delta.cu)
# ---------------------------------------------------------------------------------------
_delta = None
SINK_ATTENTION_ROWS = 8             # (token, head) rows of a block of the attention kernel with a sink
SINK_ATTENTION_MAX_HEAD_DIM = 512
SINK_ATTENTION_SPLIT_KEYS = 256     # keys of a piece when a one-token step cuts a request's keys over several blocks
DELTA_RULE_MAX_KEY_DIM = 512
DELTA_CHUNK, DELTA_CHUNK_KEY_DIMS = 32, (128,)      # tokens of a chunk; key sizes whose runs of tokens are taken in chunks
# Tokens of a request in one step from which they are taken in chunks: a whole chunk, and two of float32, whose rows are three parts.  Token by token / in chunks, us, all kernels,
# heads of 128 x 128.  Bfloat16, 16 heads: one request of 24 14.6 / 11.5, 64: 29 / 13, 100: 42 / 16; 16 of 24: 61 / 43, of 100: 208 / 102; 64 of 24: 229 / 161.  One beside 63 single
# tokens, which then take kernels of their own: 24 60 / 67, 32: 63 / 66, 48: 70 / 69, 64: 77 / 69; 32 heads 24: 128 / 134, 32: 130 / 135, 64: 137 / 138, 100: 159 / 143; beside one, 2 heads,
# 24: 14.5 / 16.6.  Float32: one of 24 14.4 / 13.9; 16 of 33: 78 / 104, of 48: 106 / 104, of 64: 136 / 106, of 65: 139 / 138; 64 of 48: 402 / 410, of 64: 518 / 419, of 65: 529 / 532, of
# 100: 780 / 652; 64 beside 63 single ones, 16 heads 77 / 72, 32: 138 / 147.
DELTA_CHUNK_MIN_TOKENS = 32


def _delta_lib():
    global _delta
    if _delta is None:
        lib = _build.delta_mixers_library()
        lib.msgl_scaled_add_norm.argtypes = [c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_float, c_void_p, c_int, c_int, c_int, c_void_p]
        lib.msgl_rotary_angles.argtypes = [c_void_p, c_void_p, ctypes.c_double, c_void_p, c_int, c_int, c_void_p]
        lib.msgl_sink_qkv_prep.argtypes = [c_void_p, c_ll, c_void_p, c_int, c_void_p, c_ll, c_float] + [c_void_p] * 4 + [c_int] * 7 + \
            [c_void_p, c_void_p, c_int, c_float, c_int, c_int, c_int, c_void_p]
        lib.msgl_sink_attention.argtypes = [c_void_p] * 6 + [c_int, c_int, c_int, c_void_p, c_void_p, c_ll, c_void_p, c_void_p] + \
            [c_int] * 12 + [c_float, c_float, c_int, c_void_p, c_ll, c_int, c_void_p]
        lib.msgl_sink_attention_mma.argtypes = [c_void_p] * 6 + [c_int, c_int, c_int, c_void_p, c_void_p, c_ll, c_void_p, c_void_p] + \
            [c_int] * 10 + [c_float, c_float, c_void_p, c_ll, c_int, c_void_p]
        lib.msgl_delta_rule.argtypes = [c_void_p, c_void_p, c_ll, c_int, c_int] + [c_void_p] * 7 + [c_int] * 11 + [c_void_p] * 2
        lib.msgl_delta_rule_scratch.argtypes = [c_int] * 8
        lib.msgl_delta_rule_scratch.restype = c_ll
        lib.msgl_side_gate_mul.argtypes = [c_void_p, c_ll, c_void_p, c_int, c_int, c_void_p, c_int, c_void_p, c_int, c_int, c_int, c_void_p]
        _delta = lib
    return _delta


def scaled_add_norm(x: torch.Tensor, scale: torch.Tensor, residual: torch.Tensor, *, weight: Optional[torch.Tensor] = None,
                    eps: float = 0.0, out_dtype: Optional[torch.dtype] = None) -> Optional[torch.Tensor]:
    """residual += x * scale in float32, in place (scale: float32 [H], one factor per column).  With `weight` (float32 [H])
    -> rmsnorm(residual) * weight in `out_dtype`, from the same pass; without it -> residual itself in `out_dtype`, or nothing
    when `out_dtype` is None.  x [T, H] float32 or bfloat16."""
    _need_cuda(x, scale, residual, weight)
    T, H = x.shape
    assert x.is_contiguous() and x.dtype in (torch.float32, torch.bfloat16)
    assert residual.dtype == torch.float32 and residual.is_contiguous() and residual.shape == x.shape
    assert scale.dtype == torch.float32 and scale.numel() == H and (weight is None or (weight.dtype == torch.float32 and weight.numel() == H))
    y = torch.empty((T, H), dtype=out_dtype, device=x.device) if out_dtype is not None else None
    assert weight is None or y is not None
    code = _delta_lib().msgl_scaled_add_norm(_ptr(x), int(x.dtype == torch.float32), _ptr(scale), _ptr(residual), _ptr(weight), float(eps),
                                             _ptr(y), _DT[out_dtype] if out_dtype is not None else 0, T, H, _stream())
    _check(code, "scaled_add_norm")
    return y


def rotary_angles(positions: torch.Tensor, freq: torch.Tensor, magnitude: float, T: int) -> torch.Tensor:
    """positions int32 [>= T], freq float64 [n] -> float32 [T, 2n] = magnitude * (cos | sin)(position * freq), the product and the
    circular functions in double precision."""
    _need_cuda(positions, freq)
    assert positions.dtype == torch.int32 and positions.numel() >= T and freq.dtype == torch.float64 and freq.is_contiguous()
    n = freq.numel()
    out = torch.empty((T, 2 * n), dtype=torch.float32, device=freq.device)
    _check(_delta_lib().msgl_rotary_angles(_ptr(positions), _ptr(freq), float(magnitude), _ptr(out), T, n, _stream()), "rotary_angles")
    return out


def sink_qkv_prep(proj: torch.Tensor, *, n_q: int, n_kv: int, d: int, dv: int, angles: Optional[torch.Tensor],
                  v_first: Optional[torch.Tensor], lam: float, out_loc: Optional[torch.Tensor], k_cache: Optional[torch.Tensor],
                  v_cache: Optional[torch.Tensor], page_size: int, q_norm: Optional[torch.Tensor] = None,
                  k_norm: Optional[torch.Tensor] = None, v_unit: bool = False, eps: float = 0.0, interleaved: bool = False,
                  qk_unit: bool = False, maps: int = 1) -> torch.Tensor:
    """proj [T, >= n_q * d + n_kv * d + n_kv * dv] packed rows [q | k | v | ...].  Where weights are given (q_norm, k_norm float32
    [d], one for all heads) every q and k head is RMS-normed by itself first; the first angles.shape[1] elements of every q and
    k head turn in halves (element i against i + rot / 2), or with `interleaved` in neighbouring pairs, by `angles` float32 [T, rot]
    = cos | sin of the tokens' positions; with qk_unit every q and k head is then divided by its root mean square; v
    becomes (1 - lam) v + lam v_first where `v_first` [T, n_kv * dv] (a view into packed rows) is given, and with
    v_unit every v head is then divided by its root mean square (eps inside the root); k goes to `k_cache` [pages, n_kv, page, d] and v to `v_cache` [pages, n_kv, page, dv] at token slots `out_loc`; the q rows come back as [T, n_q, d].
    maps = M > 1: every q and kv head has M vectors of d elements (proj [n_q * M * d | n_kv * M * d | n_kv * dv | ...]), each treated
    as a head of its own; `k_cache` rows are M * d long, and q comes back as [T, n_q * M, M * d], vector (h, m) in place m of its
    row and zeros in the others.  Without a cache the packed rows need hold q only."""
    _need_cuda(proj, angles, v_first, out_loc, k_cache, v_cache)
    T = proj.shape[0]
    width = n_q * maps * d + (n_kv * (maps * d + dv) if k_cache is not None else 0)
    stride = _rows_view(proj, proj.shape[1], "proj")
    assert proj.shape[1] >= width
    rot = 0
    if angles is not None:
        rot = angles.shape[1]
        assert angles.dtype == torch.float32 and angles.is_contiguous() and angles.shape[0] >= T
    vf_stride = 0
    if v_first is not None:
        assert v_first.dtype == proj.dtype and v_first.shape == (T, n_kv * dv)
        vf_stride = _rows_view(v_first, n_kv * dv, "v_first")
    if k_cache is not None:
        assert k_cache.dtype == proj.dtype and v_cache.dtype == proj.dtype and k_cache.is_contiguous() and v_cache.is_contiguous()
        assert tuple(k_cache.shape[1:]) == (n_kv, page_size, maps * d) and tuple(v_cache.shape[1:]) == (n_kv, page_size, dv)
        assert out_loc is not None and out_loc.dtype == torch.int32 and out_loc.numel() >= T
    assert (q_norm is None) == (k_norm is None)
    if q_norm is not None:
        assert q_norm.dtype == k_norm.dtype == torch.float32 and q_norm.numel() == k_norm.numel() == d
        assert q_norm.is_contiguous() and k_norm.is_contiguous()
        _need_cuda(q_norm, k_norm)
    q_out = torch.empty((T, n_q * maps, maps * d), dtype=proj.dtype, device=proj.device)
    code = _delta_lib().msgl_sink_qkv_prep(_ptr(proj), stride, _ptr(angles), rot, _ptr(v_first), vf_stride, float(lam), _ptr(out_loc),
                                           _ptr(q_out), _ptr(k_cache), _ptr(v_cache), page_size, n_q, n_kv, d, dv, T, _dt(proj), _ptr(q_norm), _ptr(k_norm),
                                           int(bool(v_unit)), float(eps), int(bool(interleaved)), int(bool(qk_unit)), int(maps), _stream())
    _check(code, "sink_qkv_prep")
    return q_out


SINK_ATTENTION_MMA_ROWS = 64        # rows of a block of the tensor-core kernel
SINK_ATTENTION_MMA_MAX_HEAD_DIM = 128


def sink_attention_geometry(n_q: int, n_kv: int, tensor_cores: bool = False) -> Tuple[int, int]:
    """(tokens per query tile, query heads of one kv head per block) of the attention kernels with a sink."""
    rows = SINK_ATTENTION_MMA_ROWS if tensor_cores else SINK_ATTENTION_ROWS
    gh = min(n_q // n_kv, rows)
    return rows // gh, gh


def sink_attention_on_tensor_cores(dtype: torch.dtype, d: int, dv: int) -> bool:
    """Whether the tensor-core kernel takes these rows: bfloat16, head sizes in steps of 8 up to 128."""
    return dtype == torch.bfloat16 and d % 8 == 0 and dv % 8 == 0 and max(d, dv) <= SINK_ATTENTION_MMA_MAX_HEAD_DIM


def sink_attention_splits(table_width: int, page_size: int, window: int, chunk: int = 0) -> int:
    """Pieces a one-token step cuts a request's keys into: as many as the block table's width asks for, or as a window or a chunk
    touches."""
    splits = max(1, -(-(table_width * page_size) // SINK_ATTENTION_SPLIT_KEYS))
    if window > 0 or chunk > 0:
        splits = min(splits, ((window or chunk) - 1) // SINK_ATTENTION_SPLIT_KEYS + 2)
    return splits


def sink_attention(q: torch.Tensor, out: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, *, q_start: torch.Tensor,
                   kv_len: torch.Tensor, block_table: torch.Tensor, n_kv: int, page_size: int, scale: float, softcap: float,
                   window: int, sink: Optional[torch.Tensor], q_lens: Optional[Sequence[int]], workspace=None,
                   tensor_cores: Optional[bool] = None, gate: Optional[torch.Tensor] = None, chunk: int = 0) -> None:
    """Causal softmax attention over the paged cache: the query at position i sees the keys j <= i with i - j < window (window 0:
    all; or, with chunk > 0 and window 0, the keys j <= i of its own chunk, j // chunk == i // chunk), score = q . k * scale, capped as softcap * tanh(score / softcap) where softcap > 0, and every softmax's denominator
    holds exp(sink[head]) besides the seen keys' terms (sink None: it does not).  q [T, heads, d]; K cache [pages, n_kv, page, d], V cache [pages, n_kv,
    page, dv]; sink float32 [heads]; out [T, heads * dv].  q_lens: the requests' numbers of tokens as the host knows them (they
    size the launch), or None when every request brings one token: the keys are then cut into pieces of
    SINK_ATTENTION_SPLIT_KEYS for blocks of their own, joined in order by a second kernel (workspace: a parts.Workspace for
    the pieces).  tensor_cores: None = the bfloat16 kernel with mma products where it takes the sizes
    (`sink_attention_on_tensor_cores`), the float32-arithmetic one elsewhere; False = the float32-arithmetic kernel in any case.
    gate [T, heads * dv] (a view into packed rows): the output is multiplied by sigmoid(gate), element by element."""
    _need_cuda(q, out, k_cache, v_cache, q_start, kv_len, block_table, sink, gate)
    T, n_q, d = q.shape
    dv = v_cache.shape[3]
    assert q.is_contiguous() and k_cache.dtype == q.dtype and v_cache.dtype == q.dtype and out.dtype == q.dtype
    assert sink is None or (sink.dtype == torch.float32 and sink.numel() == n_q)
    out_stride = _rows_view(out, n_q * dv, "out")
    gate_stride = 0
    if gate is not None:
        assert gate.dtype == q.dtype and gate.shape[0] == T
        gate_stride = _rows_view(gate, n_q * dv, "gate")
    B = kv_len.numel()
    if tensor_cores is None:
        tensor_cores = sink_attention_on_tensor_cores(q.dtype, d, dv) and out_stride % 2 == 0 and out.data_ptr() % 4 == 0 and \
            gate_stride % 2 == 0 and (gate is None or gate.data_ptr() % 4 == 0)
    QT, GH = sink_attention_geometry(n_q, n_kv, tensor_cores)
    uniform = q_lens is None
    n_tiles = B if uniform else sum(-(-n // QT) for n in q_lens)
    splits, part_o, part_ml = 1, None, None
    if uniform:
        splits = sink_attention_splits(block_table.shape[1], page_size, int(window), int(chunk))
        if splits > 1:
            rows = splits * T * n_q
            if workspace is not None:
                part_o, part_ml = workspace.get("sink_attention_o", rows * dv, torch.float32), workspace.get("sink_attention_ml", rows * 2, torch.float32)
            else:
                part_o = torch.empty(rows * dv, dtype=torch.float32, device=q.device)
                part_ml = torch.empty(rows * 2, dtype=torch.float32, device=q.device)
    if tensor_cores:
        code = _delta_lib().msgl_sink_attention_mma(
            _ptr(q), _ptr(k_cache), _ptr(v_cache), _ptr(q_start), _ptr(kv_len), _ptr(block_table), block_table.stride(0), int(uniform),
            n_tiles, _ptr(sink), _ptr(out), out_stride, _ptr(part_o), _ptr(part_ml), splits, SINK_ATTENTION_SPLIT_KEYS, T, B, n_q, n_kv, d,
            dv, page_size, int(window), float(scale), float(softcap), _ptr(gate), gate_stride, int(chunk), _stream())
    else:
        code = _delta_lib().msgl_sink_attention(
            _ptr(q), _ptr(k_cache), _ptr(v_cache), _ptr(q_start), _ptr(kv_len), _ptr(block_table), block_table.stride(0), int(uniform),
            n_tiles, _ptr(sink), _ptr(out), out_stride, _ptr(part_o), _ptr(part_ml), splits, SINK_ATTENTION_SPLIT_KEYS, T, B, n_q, n_kv, d,
            dv, page_size, QT, GH, int(window), float(scale), float(softcap), _dt(q), _ptr(gate), gate_stride, int(chunk), _stream())
    _check(code, f"sink_attention (head sizes {d}, {dv})")
    if splits > 1:
        global LAUNCHES
        LAUNCHES += 1


def delta_rule(qkv: torch.Tensor, a: torch.Tensor, b: torch.Tensor, *, heads: int, kv_heads: int, key_dim: int, value_dim: int,
               a_log: torch.Tensor, dt_bias: torch.Tensor, state: torch.Tensor, q_start: torch.Tensor, slots: torch.Tensor,
               q_lens: Optional[Sequence[int]] = None, workspace=None) -> torch.Tensor:
    """The gated delta rule over the step's tokens, continued from and written back to `state` [slots, heads, key_dim, value_dim]
    float32.  qkv [T, 2 * kv_heads * key_dim + heads * value_dim] contiguous (q | k | v as the convolution left them); a, b
    [T, heads]: views into one packed projection (decay and write-strength pre-activations).  Per head: unit-length q (times
    key_dim^-1/2) and k, beta = sigmoid(b), g = exp(-exp(a_log) softplus(a + dt_bias)), S <- g S, u = beta (v - S^T k),
    S <- S + k u^T, o = S^T q.  -> float32 [T, heads * value_dim]."""
    _need_cuda(qkv, a, b, a_log, dt_bias, state, q_start, slots)
    T = qkv.shape[0]
    assert qkv.is_contiguous() and qkv.shape[1] == 2 * kv_heads * key_dim + heads * value_dim
    assert a.dtype == qkv.dtype and b.dtype == qkv.dtype and a.shape == (T, heads) and b.shape == (T, heads)
    stride = _rows_view(a, heads, "a")
    assert _rows_view(b, heads, "b") == stride
    assert state.dtype == torch.float32 and state.is_contiguous() and tuple(state.shape[1:]) == (heads, key_dim, value_dim)
    assert a_log.dtype == torch.float32 and dt_bias.dtype == torch.float32 and a_log.numel() == heads and dt_bias.numel() == heads
    out = torch.empty((T, heads * value_dim), dtype=torch.float32, device=qkv.device)
    B = q_start.numel() - 1
    # runs of tokens go in chunks, single tokens and short runs token by token: a matter of the request's own tokens in this step
    # and of the sizes, so a request's results do not depend on the requests beside it
    least = min(DELTA_CHUNK_MIN_TOKENS if qkv.dtype == torch.bfloat16 else 2 * DELTA_CHUNK_MIN_TOKENS, 0x7fffffff)
    long_runs = [n for n in q_lens or () if n >= least] if key_dim in DELTA_CHUNK_KEY_DIMS and value_dim % 16 == 0 else []
    status = _status_words(qkv.device) if long_runs else None
    if status is None:
        long_runs = []
    n_chunks = sum(-(-n // DELTA_CHUNK) for n in long_runs)
    short = not long_runs or any(0 < n < least for n in q_lens)
    if n_chunks and qkv.data_ptr() % 16:
        qkv = qkv.clone()            # the chunks' rows are read by 16 bytes
    # what does not depend on the state (unit q and k, beta, g, and for chunks all that lies within one) is made for all tokens at once
    lib, dt = _delta_lib(), _dt(qkv)
    numel = lib.msgl_delta_rule_scratch(T, heads, kv_heads, key_dim, value_dim, n_chunks, short, dt)
    scratch = workspace.get("delta_rule_prep", numel, torch.float32) if workspace is not None else \
        torch.empty(numel, dtype=torch.float32, device=qkv.device)
    code = lib.msgl_delta_rule(qkv.data_ptr(), a.data_ptr(), stride, 0, _col_off(b, a), a_log.data_ptr(), dt_bias.data_ptr(), state.data_ptr(), q_start.data_ptr(),
                               slots.data_ptr(), out.data_ptr(), scratch.data_ptr(), heads, kv_heads, key_dim, value_dim, T, B, dt, n_chunks,
                               len(long_runs), least, short, _ptr(status), _stream())
    _check(code, f"delta_rule (key size {key_dim})")
    global LAUNCHES
    LAUNCHES += 1 + 2 * int(short and n_chunks > 0)
    return out


def side_gate_mul(gate: torch.Tensor, table: torch.Tensor, ids: torch.Tensor, offset: int) -> torch.Tensor:
    """gate [T, dim], table [V, columns], ids int32 [T] -> [T, dim] = gelu_tanh(gate) * table[ids][offset : offset + dim]."""
    _need_cuda(gate, table, ids)
    T, dim = gate.shape
    assert table.dtype == gate.dtype and table.is_contiguous() and ids.dtype == torch.int32 and ids.numel() >= T
    out = torch.empty((T, dim), dtype=gate.dtype, device=gate.device)
    code = _delta_lib().msgl_side_gate_mul(_ptr(gate), _rows_view(gate, dim, "gate"), _ptr(table), table.shape[1], int(offset), _ptr(ids),
                                           table.shape[0], _ptr(out), dim, T, _dt(gate), _stream())
    _check(code, "side_gate_mul")
    return out


# ---------------------------------------------------------------------------------------
# several copies of the residual stream, heads that are the difference of two maps (csrc/mixers_streams.cu)
# ---------------------------------------------------------------------------------------
_streams = None
MAX_STREAMS = 32


def _streams_lib():
    global _streams
    if _streams is None:
        lib = _build.stream_mixers_library()
        lib.msgl_stream_mix_norm.argtypes = [c_void_p, c_ll, c_ll, c_void_p, c_void_p, c_int] + [c_void_p] * 5 + [c_float, c_int, c_void_p, c_void_p] + \
            [c_int] * 4 + [c_void_p]
        lib.msgl_map_difference.argtypes = [c_void_p, c_int, c_void_p, c_ll, c_float, c_float, c_float, c_int, c_int, c_int, c_int, c_void_p]
        _streams = lib
    return _streams


def stream_mix_norm(x: torch.Tensor, *, streams: int, weight: torch.Tensor, bias: Optional[torch.Tensor], eps: float, center: bool,
                    w_in: Optional[torch.Tensor], y: Optional[torch.Tensor] = None, mix: Optional[torch.Tensor] = None,
                    w_out: Optional[torch.Tensor] = None, x_out: Optional[torch.Tensor] = None, rows: Optional[torch.Tensor] = None,
                    out_dtype: torch.dtype = torch.float32) -> torch.Tensor:
    """S copies of the stream: x float32 [T, S, H], or [T, H] where all copies are still the same row.  With `y` [T, H] (what a
    sublayer hands over) every copy becomes sum_s mix[s][t] x_s + w_out[t] y (mix [S, S] from s to t, w_out [S]; float32), all from
    the old ones, and goes to `x_out` [T, S, H] where it is given (may be x).  -> norm(sum_t w_in[t] x_t) * weight (+ bias) in
    `out_dtype`, w_in float32 [S] (None: ones); center: a layer norm, else an RMS norm.  rows (int32): the rows that are normed
    (nothing is written to the copies then)."""
    _need_cuda(x, weight, bias, w_in, y, mix, w_out, x_out, rows)
    S, H = streams, x.shape[-1]
    T = x.shape[0]
    assert x.dtype == torch.float32 and x.is_contiguous() and (x.dim() == 2 or x.shape[1] == S)
    assert weight.dtype == torch.float32 and weight.numel() == H and (bias is None or (bias.dtype == torch.float32 and bias.numel() == H))
    for t, n in ((w_in, S), (mix, S * S), (w_out, S)):
        assert t is None or (t.dtype == torch.float32 and t.numel() == n and t.is_contiguous())
    if y is not None:
        assert y.shape == (T, H) and y.is_contiguous() and y.dtype in (out_dtype, torch.float32)
    assert x_out is None or (x_out.shape == (T, S, H) and x_out.is_contiguous() and x_out.dtype == torch.float32)
    n = T if rows is None else rows.numel()
    out = torch.empty((n, H), dtype=out_dtype, device=x.device)
    code = _streams_lib().msgl_stream_mix_norm(_ptr(x), H * (S if x.dim() == 3 else 1), H if x.dim() == 3 else 0, _ptr(x_out), _ptr(y),
                                               int(y is not None and y.dtype == torch.float32), _ptr(mix), _ptr(w_out), _ptr(w_in), _ptr(weight),
                                               _ptr(bias), float(eps), int(bool(center)), _ptr(rows), _ptr(out), n, S, H, _DT[out_dtype], _stream())
    _check(code, f"stream_mix_norm ({S} streams, width {H})")
    return out


def map_difference(a: torch.Tensor, out: torch.Tensor, *, heads: int, lam: float, eps: float, scale: float) -> None:
    """a [T, heads * 2, dv] (a head's two maps side by side), out [T, heads * dv]: with v = a_1 - lam a_2 per head,
    out = v / sqrt(mean(v^2) + eps) * scale, in float32."""
    _need_cuda(a, out)
    T, dv = a.shape[0], a.shape[2]
    assert a.is_contiguous() and a.shape[1] == 2 * heads and a.dtype in (out.dtype, torch.float32)
    o_stride = _rows_view(out, heads * dv, "out")
    code = _streams_lib().msgl_map_difference(_ptr(a), int(a.dtype == torch.float32), _ptr(out), o_stride, float(lam), float(eps), float(scale),
                                              T, heads, dv, _dt(out), _stream())
    _check(code, f"map_difference (value size {dv})")


# ---------------------------------------------------------------------------------------
# the whole decode step in one persistent kernel (csrc/decode_step.cu)
# ---------------------------------------------------------------------------------------
# Off unless MSGL_FUSED_DECODE=1: measured on B200 at Qwen3-8B's sizes the one-kernel step takes 4.2 / 5.4 ms at batch 1 / 8
# (context 4,096) against 3.4 / 4.2 ms kernel by kernel (see profiles/decode_step_kernel_b1_b8.md for where the time goes).
USE_FUSED_DECODE = os.environ.get("MSGL_FUSED_DECODE", "0") == "1"
FUSED_DECODE_MAX_TOKENS = 8
STATUS_WORD_DECODE_STEP = 3


class DsLayer(ctypes.Structure):
    """One run of a layer for the decode-step kernel; mirrors `struct DsLayer`."""
    _fields_ = [("w_qkv", c_void_p), ("b_qkv", c_void_p), ("w_o", c_void_p), ("w_gu", c_void_p), ("w_down", c_void_p),
                ("norm_in", c_void_p), ("norm_post", c_void_p), ("q_norm", c_void_p), ("k_norm", c_void_p),
                ("k_cache", c_void_p), ("v_cache", c_void_p),
                ("eps_in", c_float), ("eps_post", c_float), ("eps_qk", c_float),
                ("norm_f32", c_int), ("qk_norm_f32", c_int), ("pad_", c_int)]


class DsStep(ctypes.Structure):
    """Arguments of one decode step; mirrors `struct DsStep`."""
    _fields_ = [("layers", c_void_p), ("n_layers", c_int), ("M", c_int),
                ("H", c_int), ("n_q", c_int), ("n_kv", c_int), ("I", c_int), ("V", c_int),
                ("page_size", c_int), ("page_shift", c_int), ("bt_stride", c_int), ("max_split", c_int),
                ("scale", c_float),
                ("rope", c_void_p), ("rot", c_int), ("max_pos", c_int),
                ("ids", c_void_p), ("positions", c_void_p), ("kv_len", c_void_p), ("block_table", c_void_p),
                ("out_loc", c_void_p), ("nsplit", c_void_p),
                ("embed", c_void_p), ("final_norm", c_void_p), ("final_f32", c_int), ("eps_final", c_float),
                ("lm_head", c_void_p),
                ("res", c_void_p), ("xn", c_void_p), ("ssq", c_void_p), ("qkv", c_void_p), ("attn", c_void_p), ("act", c_void_p),
                ("part_o", c_void_p), ("part_ml", c_void_p), ("tickets", c_void_p), ("logits", c_void_p),
                ("bar", c_void_p), ("status", c_void_p)]


_decode_libs = {}


def _decode_lib(head_dim: int):
    lib = _decode_libs.get(head_dim)
    if lib is None:
        lib = _build.decode_step_library(head_dim)
        lib.msgl_decode_step_blocks.argtypes = [c_int] * 6
        lib.msgl_decode_step_blocks.restype = c_int
        lib.msgl_decode_step.argtypes = [ctypes.POINTER(DsStep), c_void_p]
        if lib.msgl_decode_step_layer_bytes() != ctypes.sizeof(DsLayer) or lib.msgl_decode_step_struct_bytes() != ctypes.sizeof(DsStep):
            raise KernelError("decode_step: the argument structures of the library and of ops.py differ")
        _decode_libs[head_dim] = lib
    return lib


def decode_step_blocks(tokens: int, hidden: int, n_q: int, n_kv: int, head_dim: int, intermediate: int, vocab: int) -> int:
    """Blocks the decode-step kernel runs with for these sizes on the current device; 0: it does not take them
    (the caller then runs the step kernel by kernel).  Not inside a stream capture the first time."""
    if not USE_FUSED_DECODE or head_dim % 32 or head_dim < 32 or head_dim > 128:      # beyond 128 the accumulators spill
        return 0
    return int(_decode_lib(head_dim).msgl_decode_step_blocks(tokens, hidden, n_q, n_kv, intermediate, vocab))


def decode_step(step: DsStep, head_dim: int) -> None:
    """Launch the decode-step kernel on the current stream."""
    code = _decode_lib(head_dim).msgl_decode_step(ctypes.byref(step), _stream())
    _check(code, f"decode_step (head size {head_dim})")
