"""Python host side of the attention path: torch tensors in, C-ABI calls out.

torch is used for device memory and streams only; all arithmetic happens in
``libarc_sdpa.so``.  The functions in the second half keep the names, argument
order and error behaviour of the reference's C++ call sites so its call stacks
map one to one (reference files are cited per function).
"""
from __future__ import annotations

import ctypes as C
from typing import Optional, Union

import torch

from . import _lib
from ._lib import MASK_CAUSAL, MASK_EXPLICIT, MASK_NONE, NO_WINDOW, ArcError, check

__all__ = [
    "MASK_NONE", "MASK_EXPLICIT", "MASK_CAUSAL", "NO_WINDOW", "ArcError",
    "sdpa_prefill", "sdpa_decode", "sdpa_merge", "mul_sigmoid_inplace", "fill_causal_mask",
    "gqa_attention_sdpa", "gqa_attention", "batched_attention", "qwen35_xmx_attention",
    "qwen35_online_attention", "qwen35_xmx_attention_decode_gqa",
    "device_status", "clear_device_status", "launch_count", "Workspace", "exchange_bytes",
]


def _stream_ptr(t: torch.Tensor) -> int:
    return torch.cuda.current_stream(t.device).cuda_stream


def _require(t: torch.Tensor, dtype, name: str) -> None:
    if not isinstance(t, torch.Tensor) or t.device.type != "cuda":
        raise ValueError(f"{name} must be a CUDA tensor (there is no CPU path)")
    if t.dtype != dtype:
        raise ValueError(f"{name} must be {dtype}, got {t.dtype}")


class Workspace:
    """Grow-only device scratch for split-KV partials and scanned masks, to pass as ``workspace=``.

    Reallocates only when a call needs more than any earlier call (the reference measured what
    per-call attention scratch costs: notes/diffusion_gemma/NVFP4_DPAS_KERNEL.md:243-250).  One of them
    serves the calls of one stream; it is the caller's to keep from being used on two at once.  Calls
    without one take their scratch from torch's caching allocator on their stream and share it with no
    other call.
    """

    _per_device: dict[int, "Workspace"] = {}

    def __init__(self, device: torch.device):
        self.device = device
        self.buf: Optional[torch.Tensor] = None

    @classmethod
    def for_device(cls, device: torch.device) -> "Workspace":
        idx = device.index if device.index is not None else torch.cuda.current_device()
        ws = cls._per_device.get(idx)
        if ws is None:
            ws = cls._per_device[idx] = cls(torch.device("cuda", idx))
        return ws

    def reserve(self, nbytes: int) -> torch.Tensor:
        if self.buf is None or self.buf.numel() < nbytes:
            self.buf = torch.empty(max(nbytes, 1 << 20), dtype=torch.uint8, device=self.device)
        return self.buf


def _native():
    """The compiled binding: it reads the tensors, checks them, fills the parameter struct and calls the
    library.  Replaced by the module's own getter once loaded, so a call costs one global lookup."""
    global _native
    module = _lib.native()
    _native = lambda: module  # noqa: E731
    return module


def sdpa_prefill(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, *, scale: float,
                 mask_type: int = MASK_NONE, window: int = NO_WINDOW, mask: Optional[torch.Tensor] = None,
                 gate: Optional[torch.Tensor] = None, out: Optional[torch.Tensor] = None,
                 num_splits: int = 0, return_lse: bool = False,
                 workspace: Optional[Workspace] = None,
                 block_ids: Optional[torch.Tensor] = None, block_ids_offset: int = 0,
                 out_copies: Optional[torch.Tensor] = None):
    """Prefill / canvas attention.  q: (B, S, nq, hd) or (S, nq, hd); k, v: (B, L, nkv, hd) or (L, nkv, hd).

    ``out`` may be ``q`` itself.  Returns ``out`` (and the natural-log LSE (B, S, nq) when asked).
    ``block_ids`` (device int32, one per absolute position, -1 = text; causal masks only): Gemma4's
    vision blocks — a query inside a block also sees the block's later keys
    (src/common/kernels/attention_mask.hpp:44-73); ``block_ids[block_ids_offset + j]`` is key j's id.
    ``out_copies`` (device int64, at most 15 addresses): further buffers laid out like ``out`` that the
    kernel's epilogue stores the result to as well — other GPUs' mapped buffers when a head-sharded output
    is to be gathered (see ``sharded.GatheredPrefill``).
    """
    return _native().sdpa_prefill(q, k, v, scale, mask_type, window, mask, gate, out, num_splits, return_lse, workspace,
                                  block_ids, block_ids_offset, out_copies)


def sdpa_decode(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, *, scale: float,
                kv_len: Union[int, torch.Tensor, None] = None, kv_row_offset: Optional[torch.Tensor] = None,
                gate: Optional[torch.Tensor] = None, out: Optional[torch.Tensor] = None,
                return_partial: bool = False, want_out: bool = True, num_ctas: int = 0,
                partial_out: Optional[torch.Tensor] = None, partial_lse: Optional[torch.Tensor] = None,
                exchange: Optional[tuple] = None, workspace: Optional[Workspace] = None,
                exchange_wait_cycles: int = 0):
    """Split-KV decode of one query token per sequence.

    q: (B, nq, hd).  k, v: either (B, max_len, nkv, hd) (one cache block per sequence) or
    (rows, nkv, hd) packed with ``kv_row_offset`` (int64 device tensor, first row of each sequence).
    ``kv_len``: int (same for all) or int32 device tensor (B,).
    Returns ``out`` (B, nq, hd) bf16; with ``return_partial`` also (out_f32, lse) — the
    ungated fp32 result and natural-log LSE a sequence-sharded caller exchanges.
    ``exchange`` = (peer_ptrs int64 device tensor (world,), world, rank, step) turns on the
    in-kernel exchange of those records over NVLink peer memory: ``out`` is then the result
    merged over all ranks' key slices (see :class:`arcaine_b200.sharded.SeqShardedDecode`);
    ``exchange_wait_cycles`` bounds the wait for the other ranks' records (0: about a second).
    """
    return _native().sdpa_decode(q, k, v, scale, kv_len, kv_row_offset, gate, out, return_partial, want_out, num_ctas,
                                 partial_out, partial_lse, exchange, workspace, exchange_wait_cycles)


def sdpa_merge(part_out: torch.Tensor, part_lse: torch.Tensor, *, gate: Optional[torch.Tensor] = None,
               out: Optional[torch.Tensor] = None, want_f32: bool = False, want_lse: bool = False):
    """LSE merge of partial results: part_out (P, rows..., hd) f32, part_lse (P, rows...) f32.

    The leading (part) dimension may be strided — e.g. views into one packed
    ``[out | lse]`` record per rank — as long as each part is dense.
    """
    _require(part_out, torch.float32, "part_out")
    _require(part_lse, torch.float32, "part_lse")
    P, hd = part_out.shape[0], part_out.shape[-1]
    row_shape = tuple(part_out.shape[1:-1])
    rows = 1
    for s in row_shape:
        rows *= s
    if tuple(part_lse.shape) != (P, *row_shape):
        raise ValueError("part_lse shape mismatch")
    if not part_out[0].is_contiguous() or not part_lse[0].is_contiguous():
        raise ValueError("each part must be dense")
    so = part_out.stride(0) if P > 1 else rows * hd
    sl = part_lse.stride(0) if P > 1 else rows
    if out is None:
        out = torch.empty((*row_shape, hd), dtype=torch.bfloat16, device=part_out.device)
    _require(out, torch.bfloat16, "out")
    if not out.is_contiguous():
        raise ValueError("out must be contiguous")
    if gate is not None:
        _require(gate, torch.bfloat16, "gate")
        if not gate.is_contiguous() or gate.numel() != out.numel():
            raise ValueError("gate must be contiguous and shaped like out")
    o32 = torch.empty((*row_shape, hd), dtype=torch.float32, device=part_out.device) if want_f32 else None
    lse = torch.empty(row_shape, dtype=torch.float32, device=part_out.device) if want_lse else None
    with torch.cuda.device(part_out.device):
        check(_lib.load().arc_sdpa_merge(part_out.data_ptr(), part_lse.data_ptr(), P, rows, hd, so, sl,
                                         gate.data_ptr() if gate is not None else None, out.data_ptr(),
                                         o32.data_ptr() if o32 is not None else None,
                                         lse.data_ptr() if lse is not None else None, _stream_ptr(part_out)),
              "arc_sdpa_merge")
    res = (out,)
    if want_f32:
        res += (o32,)
    if want_lse:
        res += (lse,)
    return res[0] if len(res) == 1 else res


def mul_sigmoid_inplace(a: torch.Tensor, gate: torch.Tensor) -> torch.Tensor:
    """a *= sigmoid(gate) in bf16 storage / fp32 math (src/modeling/qwen3_5_moe/kernels.hpp:80-88)."""
    return _native().mul_sigmoid_inplace(a, gate)


def fill_causal_mask(q_len: int, kv_len: int, past_offset: int, sliding_window: int = NO_WINDOW, *,
                     device="cuda", out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Additive (q_len, kv_len) f32 mask (src/common/kernels/attention_mask.hpp:12-38)."""
    if out is None:
        out = torch.empty((q_len, kv_len), dtype=torch.float32, device=device)
    return _native().fill_causal_mask(out, q_len, kv_len, past_offset, sliding_window)


def fill_causal_mask_with_block_ids(block_ids: Optional[torch.Tensor], q_len: int, kv_len: int, past_offset: int,
                                    sliding_window: int = NO_WINDOW, *, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Causal / sliding-window mask with Gemma4's bidirectional vision blocks
    (src/common/kernels/attention_mask.hpp:44-73).  block_ids: device int32, one per absolute position."""
    device = block_ids.device if block_ids is not None else (out.device if out is not None else "cuda")
    if out is None:
        out = torch.empty((q_len, kv_len), dtype=torch.float32, device=device)
    _require(out, torch.float32, "out")
    if not out.is_contiguous() or out.numel() < q_len * kv_len:
        raise ValueError("out must be contiguous and hold q_len * kv_len values")
    if block_ids is not None:
        _require(block_ids, torch.int32, "block_ids")
        if block_ids.numel() < past_offset + q_len:
            raise ValueError("block_ids must cover every position up to past_offset + q_len")
    with torch.cuda.device(out.device):
        check(_lib.load().arc_fill_causal_mask_with_block_ids(
            out.data_ptr(), block_ids.data_ptr() if block_ids is not None else None, q_len, kv_len, past_offset,
            sliding_window, _stream_ptr(out)), "arc_fill_causal_mask_with_block_ids")
    return out


# ---------------------------------------------------------------------------
# Reference-named entry points (one sequence, token-major tensors)
# ---------------------------------------------------------------------------
def gqa_attention_sdpa(Q, seq, nq, hd, Kc, Vc, kv_len, nkv, mask=None, mask_type=MASK_NONE, out=None):
    """src/modeling/diffusion_gemma/attention.cpp:930-995 — no scale; mask_type 0 / 1 / 3."""
    return _native().attention(Q, seq, nq, hd, Kc, Vc, kv_len, nkv, 1.0, mask_type, NO_WINDOW, mask, out, None, 0, True)


def gqa_attention(Q, seq, nq, hd, Kc, Vc, kv_len, nkv, past_offset, sliding_window, causal, out=None):
    """src/modeling/diffusion_gemma/attention.cpp:706-821 — the matmul/softmax/matmul path's result."""
    del past_offset  # queries and keys share it; the visibility rule does not depend on it
    return _native().attention(Q, seq, nq, hd, Kc, Vc, kv_len, nkv, 1.0, MASK_CAUSAL if causal else MASK_NONE,
                               sliding_window if causal else NO_WINDOW, None, out, None, 0, False)


def batched_attention(Q, seq_len, nq_heads, q_head_dim, K, V, kv_len, nkv_heads, kv_head_dim, past_offset,
                      sliding_window, scale=1.0, skip_mask=False, block_ids=None, out=None):
    """src/common/layers/attention_batched.hpp:71-136.  ``block_ids`` (device int32 per absolute position)
    turns on the vision-block rule of fill_causal_mask_with_block_ids, evaluated inside the kernel: key j
    of ``K`` sits at absolute position past_offset - (kv_len - seq_len) + j."""
    if q_head_dim != kv_head_dim:
        raise RuntimeError("batched_attention: q and kv head_dim differ")
    if block_ids is not None and skip_mask:
        block_ids = None  # the reference builds no mask at all in that case
    return _native().attention(Q, seq_len, nq_heads, q_head_dim, K, V, kv_len, nkv_heads, scale,
                               MASK_NONE if skip_mask else MASK_CAUSAL, NO_WINDOW if skip_mask else sliding_window, None, out,
                               block_ids, past_offset - (kv_len - seq_len) if block_ids is not None else 0, False)


def gemma4_sliding_decode_attention(Q, K_cache, V_cache, kv_len, kv_start, nq_heads, nkv_heads, head_dim, out=None):
    """Single-token decode of a Gemma4 sliding layer over cache rows [kv_start, kv_start + kv_len)
    (sliding_decode_attention, src/modeling/gemma4_unified/attention.cpp:93-137; no scale: Q and K are
    RMS-normed).  The reference keeps two extra copies of the cache for this call, K head-major
    (nkv, max_seq, hd) and V transposed (nkv, hd, max_seq), because its strided GEMMs want them; here the
    token-major cache (max_seq, nkv, hd) of src/modeling/gemma4_unified/kv_cache.hpp:8-9 is read in place —
    the GQA group is folded into the MMA, so those copies and their upkeep disappear."""
    res = _native().decode_one(Q, K_cache, V_cache, out, kv_start, kv_start + kv_len, nq_heads, nkv_heads, head_dim, 1.0, None,
                               True)
    return res if out is None else res.view(nq_heads, head_dim)


def gemma4_full_decode_attention(Q, K_cache, V_cache, kv_len, nq_heads, head_dim, out=None):
    """The nkv == 1 decode path of Gemma4's full-attention layers
    (src/modeling/gemma4_unified/attention.cpp:274-288): every query head shares the one KV head, the cache
    (kv_len, 1, hd) is read once for all of them.  Head dims 128 and 256 (the 512-wide global heads are
    outside what the attention kernels cover)."""
    q = Q.view(1, nq_heads, head_dim)
    o = out.view(1, nq_heads, head_dim) if out is not None else None
    nsplit = 1
    if nq_heads > 16:
        # more than 16 query heads on one KV head: the same cache rows serve several groups of <= 16 heads
        for d in range(1, nq_heads + 1):
            if nq_heads % d == 0 and nq_heads // d <= 16:
                nsplit = d
                break
    k = K_cache.view(-1, 1, head_dim)[:kv_len]
    v = V_cache.view(-1, 1, head_dim)[:kv_len]
    if nsplit == 1:
        return sdpa_decode(q, k, v, scale=1.0, kv_len=kv_len, out=o).view(nq_heads, head_dim)
    # "batch" of nsplit query groups over the same rows (row offset 0 for all)
    qb = q.view(nsplit, nq_heads // nsplit, head_dim)
    ob = o.view(nsplit, nq_heads // nsplit, head_dim) if o is not None else None
    offs = torch.zeros(nsplit, dtype=torch.int64, device=Q.device)
    lens = torch.full((nsplit,), kv_len, dtype=torch.int32, device=Q.device)
    res = sdpa_decode(qb, k, v, scale=1.0, kv_len=lens, kv_row_offset=offs, out=ob)
    return res.view(nq_heads, head_dim)


def qwen35_xmx_attention(query, key, value, output, seq, past, query_heads, key_heads, head_dim, scale):
    """src/modeling/qwen3_5/kernels.hpp:761-905 — causal over past + seq keys; output may alias query."""
    if key_heads <= 0 or query_heads % key_heads != 0:
        raise RuntimeError("Qwen3.5 attention requires integral GQA ratio")
    return _native().qwen_attention(query, key, value, output, seq, past, query_heads, head_dim, scale)


qwen35_online_attention = qwen35_xmx_attention  # src/modeling/qwen3_5/kernels.hpp:621-679, same contract


def qwen35_xmx_attention_decode_gqa(query, key, value, output, past, query_heads, key_heads, head_dim, scale,
                                    gate=None):
    """src/modeling/qwen3_5/kernels.hpp:910-1054, optionally with the sigmoid gate of operators.hpp:160 fused."""
    if key_heads <= 0 or query_heads % key_heads != 0:
        raise RuntimeError("Qwen3.5 attention requires integral GQA ratio")
    return _native().decode_one(query, key, value, output, 0, past + 1, query_heads, key_heads, head_dim, scale, gate, False)


def qkv_prepare(q: Optional[torch.Tensor], k: Optional[torch.Tensor], v: Optional[torch.Tensor], *,
                k_cache: Optional[torch.Tensor] = None, v_cache: Optional[torch.Tensor] = None, past_len: int = 0,
                q_weight: Optional[torch.Tensor] = None, k_weight: Optional[torch.Tensor] = None,
                eps: float = 1e-6, theta: float = 10000.0, partial_rotary_factor: float = 1.0,
                rope_cos: Optional[torch.Tensor] = None, rope_sin: Optional[torch.Tensor] = None,
                pos_offset=None, v_from_k: bool = False, rotary_dim: Optional[int] = None,
                mrope_positions: Optional[torch.Tensor] = None, mrope_section=None, v_copy: bool = False) -> None:
    """RMSNorm (+ RoPE) of the projected Q / K rows, unit-RMS norm of V and the KV-cache append, one launch.

    q: (B, S, nq, hd) or (S, nq, hd), rewritten in place.  k, v: (B, S, nkv, hd) projections.  K and V go to
    ``k_cache`` / ``v_cache`` (B, capacity, nkv, hd) at rows ``past_len .. past_len + S`` (no separate copy);
    without caches K is rewritten in place and V too.  ``v_from_k``: V = unit-RMS norm of the raw K projection
    (full-attention layers, src/modeling/diffusion_gemma/attention.cpp:587-595).  ``pos_offset``: the position
    of the first token, an int or a device int32 tensor (B,); defaults to ``past_len``.  With ``rope_cos`` /
    ``rope_sin`` (S, n_active_pairs) or (B, S, n_active_pairs) f32 the angles are read, otherwise computed.

    Qwen3.5 form (qwen35_apply_mrope, src/modeling/qwen3_5/kernels.hpp:576-617): ``rotary_dim`` rotates pairs
    (f, f + rotary_dim/2) with frequency exponent 2f / rotary_dim; ``mrope_positions`` (B, 3, S) or (3, S) int32
    with ``mrope_section`` (three ints) gives each frequency the position of its axis; ``v_copy`` appends V
    without a norm.
    """
    _native().qkv_prepare(q, k, v, k_cache, v_cache, past_len, q_weight, k_weight, eps, theta, partial_rotary_factor,
                          rope_cos, rope_sin, pos_offset, v_from_k, rotary_dim, mrope_positions, mrope_section, v_copy)


def rms_norm(x: torch.Tensor, weight: Optional[torch.Tensor], eps: float) -> torch.Tensor:
    """In-place RMSNorm over the last dimension of (rows, H) / (S, heads, H): rms_norm / rms_norm_no_scale,
    src/common/kernels/rms_norm.hpp:9-56 (weight None = unit scale)."""
    x3 = x if x.dim() == 3 else x.view(x.shape[0], 1, x.shape[-1])
    qkv_prepare(x3, None, None, q_weight=weight, eps=eps, partial_rotary_factor=0.0)
    return x


def fused_norm_rope_inplace(x: torch.Tensor, weight: torch.Tensor, offset: int, theta: float, partial: float,
                            eps: float, rope_cos: Optional[torch.Tensor] = None,
                            rope_sin: Optional[torch.Tensor] = None) -> torch.Tensor:
    """fused_norm_rope_inplace(x (seq, nheads, hd), weight, offset, theta, partial, eps, cos, sin):
    src/modeling/diffusion_gemma/attention_kernels.hpp:99-153."""
    qkv_prepare(x, None, None, q_weight=weight, eps=eps, theta=theta, partial_rotary_factor=partial,
                rope_cos=rope_cos, rope_sin=rope_sin, pos_offset=offset)
    return x


def exchange_bytes(world: int, batch: int, nq: int, hd: int) -> int:
    """Size of one rank's peer-exchange buffer for sequence-sharded decode."""
    return int(_lib.load().arc_sdpa_exchange_bytes(world, batch, nq, hd))


FAULT_WAIT_PEER = 9      # device fault codes (csrc/ptx.cuh)
FAULT_BAD_KV_RANGE = 10


def device_status(device=None) -> tuple[int, int]:
    """(fault code, detail) of the device-side status word; synchronises the device."""
    code, detail = C.c_uint32(0), C.c_uint32(0)
    with torch.cuda.device(device if device is not None else torch.cuda.current_device()):
        rc = _lib.load().arc_sdpa_device_status(C.byref(code), C.byref(detail))
    if rc not in (_lib.ARC_OK, _lib.ARC_ERR_DEVICE_WAIT_TIMEOUT, _lib.ARC_ERR_DEVICE_BAD_RANGE):
        raise ArcError(rc, "arc_sdpa_device_status")
    return int(code.value), int(detail.value)


def clear_device_status(device=None) -> None:
    with torch.cuda.device(device if device is not None else torch.cuda.current_device()):
        check(_lib.load().arc_sdpa_clear_device_status(), "arc_sdpa_clear_device_status")


def launch_count() -> int:
    return int(_lib.load().arc_sdpa_launch_count())
