"""Decode API, mirroring ``conv_attn/flash_conv_attention_inference.py``:
``forward_inference`` (the pybind function of fwd_inference_bindings.cpp:20-23) and
``fwd_conv_attn_inference`` (the Python wrapper at :33-93)."""
from . import _native


def forward_inference(Q, K, V, conv_kernel, k_splits, scale, pad_q, pad_k, causal, num_k_blocks=None,
                      offset_causal=False):
    """(O_splits [B,H,k_splits,d], M_splits, L_splits [B,H,k_splits]) fp32 with the merged,
    normalised result in split 0 (fwd_inference.cu:359-368).  ``causal`` is accepted and has no
    effect, exactly as in the reference kernel (fwd_inference.cu:36 is never read);
    ``num_k_blocks`` is accepted for signature compatibility and ignored.  ``offset_causal=True``
    (an addition) applies the training forward's mask with query row r placed at position
    Nk - rows + r, so that the result equals the last row of the causal training forward."""
    return _native.decode(Q, K, V, conv_kernel, k_splits, scale, pad_q, pad_k, bool(offset_causal), False)


def fwd_conv_attn_inference(Q, K, V, conv_kernel, k_splits, scale, pad_q, pad_k, causal, offset_causal=False):
    """(O [B,H,1,d], M [B,H,1], L [B,H,1]) for the last query row
    (flash_conv_attention_inference.py:33-93).  The reference front-pads Q to 16 rows with
    zeros; zero rows contribute nothing, so Q is passed as is."""
    if Q.shape[2] > 16:
        raise ValueError(f"Q sequence length must be <= 16 for inference, got {Q.shape[2]}")
    return _native.decode(Q, K, V, conv_kernel, k_splits, scale, pad_q, pad_k, bool(offset_causal), True)


def forward_inference_paged(Q, K_pool, V_pool, block_table, conv_kernel, k_splits, scale, pad_q, pad_k,
                            seq_lens=None, max_seq_len=None, offset_causal=False):
    """Decode over a paged key/value cache (an addition: the reference cache is contiguous).
    ``K_pool``/``V_pool`` bf16 [n_pages, H, page_size, d]; ``block_table`` int32 [B, max_pages] maps
    page p of sequence b to a pool page; ``seq_lens`` int32 [B] (optional) gives each sequence's
    cache length, bounded by ``max_seq_len`` (default: max_pages * page_size).  Returns
    (O_splits, M_splits, L_splits) as ``forward_inference``; equals ``forward_inference`` on the
    gathered cache."""
    return _native.decode_paged(Q, K_pool, V_pool, block_table, conv_kernel, k_splits, scale, pad_q, pad_k, seq_lens, max_seq_len,
                                bool(offset_causal))


def kv_append_paged(K_pool, V_pool, block_table, seq_lens, K_new, V_new):
    """Write ``K_new``/``V_new`` (bf16 [B,H,n_new,d]) at positions seq_lens[b] .. seq_lens[b]+n_new-1 of
    each sequence of a paged cache.  ``seq_lens`` is read, not advanced; the pages must already be in
    ``block_table``."""
    _native.kv_append_paged(K_pool, V_pool, block_table, seq_lens, K_new, V_new)
