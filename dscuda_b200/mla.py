"""Host side of the MLA path: torch tensors in, C-ABI calls out.

The functions mirror what the reference's `benchmarks/mla.py:79-117` does by
hand (raw `data_ptr()`s, the current stream, caller-owned outputs and
workspace).  They allocate outputs with torch, launch on the current stream and
return without synchronising; the work behind each signature is in the Python
extension (`csrc/bindings/torch_bridge.cpp`).  Inputs must be contiguous CUDA
tensors; bf16 unless stated.  No CPU fallback exists.
"""

from __future__ import annotations

import torch

from .library import checked, extension, library  # noqa: F401 (re-exported for callers)


def prefill_backward_launches(batch, max_seq, total, heads, packed=False) -> int:
    """Kernels one `dscuda_mla_prefill_backward` call launches: the delta pre-pass, the dk_pe sum, and
    the two main kernels (dense batches: once per group of heads that fits the scratch limit)."""
    return library("mla").dscuda_mla_prefill_backward_launches(batch, max_seq, total, heads, int(packed))


def prefill_backward_scratch_limit(limit_bytes=-1) -> int:
    """Sets the workspace the dense backward may spend on dS^T (`dscuda_mla_prefill_backward_scratch_limit`);
    returns the previous limit.  0 selects the recomputing dQ kernel, a negative value only reads."""
    return library("mla").dscuda_mla_prefill_backward_scratch_limit(limit_bytes)


def mla_forward(query, query_rope, latent, key_rope, scale):
    """Absorbed causal forward (`dscuda_mla_forward`).
    query [B,T,H,512], query_rope [B,T,H,64], latent [B,T,512], key_rope [B,T,64]
    -> (output [B,T,H,512] bf16, lse [B,H,T] fp32)."""
    return extension().mla_forward(query, query_rope, latent, key_rope, scale)


def mla_backward(dout, output, lse, query, query_rope, latent, key_rope, scale):
    """Absorbed backward (`dscuda_mla_backward`) -> (dquery, dquery_rope, dlatent, dkey_rope)."""
    return extension().mla_backward(dout, output, lse, query, query_rope, latent, key_rope, scale)


def decode_workspace(batch, heads, splits, rank=512, device="cuda"):
    lib = library("mla")
    return torch.empty(lib.dscuda_mla_workspace_elements(batch, heads, splits, rank), device=device, dtype=torch.float32)


def decode_splits(lengths, heads=128, minimum=8, clusters=74, maximum=64) -> int:
    """Partial slots per (sequence, head) that let the decode kernel cut the batch's 128-key tiles into equal ranges,
    one per pair of SMs.  The kernel never makes a range shorter than longest sequence / (splits - 1) tiles (a sequence
    may not spread over more ranges than it has slots), so a small batch of long sequences needs more slots than the
    reference harness's 8 to keep every SM pair busy.  `lengths`: cached tokens per sequence (a list or a CPU tensor)."""
    tiles = [(int(n) + 127) // 128 for n in lengths]
    head_tiles = (heads + 127) // 128
    per_range = max(1, -(-sum(tiles) * head_tiles // clusters))
    return max(minimum, min(maximum, 1 + -(-max(tiles, default=1) // per_range)))


def mla_decode(query, paged_cache, block_table, lengths, scale, splits=8, workspace=None, output=None, lse=None, checked_pages=False):
    """Paged decode (`dscuda_mla_decode`; `dscuda_mla_decode_checked` with `checked_pages`, which also
    passes the number of cache pages so that a page number outside the cache is replaced and reported).
    query [B,1,H,576], paged_cache [blocks,page,1,576], block_table [B,pages] int32,
    lengths [B] int32 -> (output [B,1,H,512] bf16, lse [B,H,1] fp32)."""
    return extension().mla_decode(query, paged_cache, block_table, lengths, scale, splits, workspace, output, lse, checked_pages)


def cache_append(paged_cache, kv_latent, key_rope, block_table, start_positions=None, token_counts=None):
    """Writes new tokens into the paged cache in place (`dscuda_mla_cache_append`).
    paged_cache [blocks,page,1,576], kv_latent [B,T,512], key_rope [B,T,64] bf16, block_table [B,pages] int32;
    start_positions / token_counts [B] int32 or None (0 / all T rows).  Token t of sequence b lands at
    position start_positions[b] + t."""
    return extension().cache_append(paged_cache, kv_latent, key_rope, block_table, start_positions, token_counts)


FP8_CACHE_ROW_BYTES = 656       # 512 e4m3 + four fp32 group scales + 64 bf16 rotary values


def cache_append_fp8(paged_fp8_cache, kv_latent, key_rope, block_table, start_positions=None, token_counts=None):
    """`cache_append` into the FP8 cache (`dscuda_mla_cache_append_fp8`): paged_fp8_cache [blocks, page, 656] uint8."""
    return extension().cache_append_fp8(paged_fp8_cache, kv_latent, key_rope, block_table, start_positions, token_counts)


def cache_dequantize_fp8(paged_fp8_cache, paged_cache=None, first_row=0, rows=None):
    """FP8 cache rows -> the bf16 cache layout the decode reads (`dscuda_mla_cache_dequantize_fp8`).
    Rows are physical (page * page_size + slot); by default the whole cache."""
    return extension().cache_dequantize_fp8(paged_fp8_cache, paged_cache, first_row, rows)


def rope_apply(q_pe=None, k_pe=None, positions=None, theta=10000.0):
    """Rotary embedding in place (`dscuda_mla_rope_apply`) of q_pe [..., H, 64] and/or k_pe [..., 1, 64] (bf16).
    `positions` int32 [rows] on the device, or None for dense [B, S, ...] tensors (position = index along S)."""
    return extension().rope_apply(q_pe, k_pe, positions, theta)


def up_project(kv_latent, w_uk, w_uv, heads):
    """Per-head keys and values from the latent (`dscuda_mla_up_project`): kv_latent [..., 512],
    w_uk / w_uv [H*128, 512] -> (k_nope [..., H, 128], v [..., H, 128])."""
    return extension().up_project(kv_latent, w_uk, w_uv, heads)


def absorb_query(q_nope, w_uk):
    """W_UK folded into the query (`dscuda_mla_absorb_query`): q_nope [..., H, 128], w_uk [H*128, 512] -> q_latent [..., H, 512]."""
    return extension().absorb_query(q_nope, w_uk)


def unabsorb_output(output_latent, w_uv):
    """W_UV applied to the latent output (`dscuda_mla_unabsorb_output`): o_latent [..., H, 512], w_uv [H*128, 512] -> out [..., H, 128]."""
    return extension().unabsorb_output(output_latent, w_uv)


def prefill_forward(q_nope, q_pe, k_nope, k_pe, v, scale, cu_seqlens=None, max_seqlen=None, output=None, lse=None):
    """Non-absorbed causal forward (`dscuda_mla_prefill_forward`).
    Dense [B,S,H,*] or packed [total,H,*] with int32 cu_seqlens on the device.
    -> (output like v, lse [B,H,S] or [H,total])."""
    return extension().prefill_forward(q_nope, q_pe, k_nope, k_pe, v, scale, cu_seqlens, max_seqlen, output, lse)


def prefill_backward_workspace(batch, max_seq, total, heads, device="cuda"):
    lib = library("mla")
    return torch.empty(lib.dscuda_mla_prefill_backward_workspace_bytes(batch, max_seq, total, heads),
                       device=device, dtype=torch.uint8)


def prefill_backward(dout, output, lse, q_nope, q_pe, k_nope, k_pe, v, scale, cu_seqlens=None, max_seqlen=None,
                     workspace=None, grads=None):
    """Non-absorbed backward (`dscuda_mla_prefill_backward`)
    -> (dq [...,H,192], dk_nope [...,H,128], dk_pe [...,1,64], dv [...,H,128])."""
    return extension().prefill_backward(dout, output, lse, q_nope, q_pe, k_nope, k_pe, v, scale, cu_seqlens, max_seqlen, workspace, grads)


def flash_forward(query, key, value, scale):
    """Causal D=128 GQA forward (`dscuda_flash_forward`).
    query [B,T,Hq,128], key/value [B,T,Hkv,128] -> (output, lse [B,Hq,T])."""
    return extension().flash_forward(query, key, value, scale)


def device_status(reset=False) -> int:
    """0 when no kernel of this library has hit a bounded-wait timeout."""
    mla = library("mla").dscuda_mla_device_status(int(reset))
    flash = library("flash_attention").dscuda_flash_device_status(int(reset))
    return mla or flash
