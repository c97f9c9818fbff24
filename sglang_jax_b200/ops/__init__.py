"""Hot ops of the model forward.

Every op has two implementations: the hand-written sm_100a kernel (module
`native`, a C-ABI shared library loaded with ctypes) and a plain-PyTorch statement
(module `reference`).  bf16 CUDA tensors take the native path; CPU tensors and other
dtypes take the reference path.  On a machine with a GPU the native library is
mandatory: if it cannot be loaded the first bf16 CUDA call raises instead of
quietly running the reference.
"""

from __future__ import annotations

import torch

from . import reference

_FORCE_REFERENCE = False


def set_force_reference(flag: bool):
    """Route every op through the PyTorch statements (debugging / `--disable-custom-kernels`)."""
    global _FORCE_REFERENCE
    _FORCE_REFERENCE = bool(flag)


def use_native(x: torch.Tensor) -> bool:
    return (not _FORCE_REFERENCE) and x.is_cuda and x.dtype == torch.bfloat16


def use_native_wide(x: torch.Tensor) -> bool:
    """Ops whose kernels exist for bf16 and for fp32."""
    return (not _FORCE_REFERENCE) and x.is_cuda and x.dtype in (torch.bfloat16, torch.float32)


def varlen_attention(q, k, v, seq_lens, scale: float):
    """Bidirectional attention over packed sequences (encoders, diffusion transformers)."""
    if use_native(q) and q.shape[-1] <= 128 and q.shape[1] % k.shape[1] == 0 and q.shape[1] // k.shape[1] <= 16 \
            and k.dtype == q.dtype and v.dtype == q.dtype:
        return _native().varlen_attention(q, k, v, seq_lens, scale)
    return reference.varlen_attention(q, k, v, seq_lens, scale)


def use_native_sampling(logits: torch.Tensor) -> bool:
    return (not _FORCE_REFERENCE) and logits.is_cuda and logits.dim() == 2 \
        and logits.dtype in (torch.float32, torch.bfloat16)


def _native():
    from . import native
    return native


def rmsnorm(x, w, eps, gemma=False):
    if use_native(x) and w.dtype == x.dtype:
        return _native().rmsnorm(x, w, eps, gemma)
    return reference.rmsnorm(x, w, eps, gemma)


def fused_add_rmsnorm(x, residual, w, eps, gemma=False):
    if use_native(x) and w.dtype == x.dtype:
        return _native().fused_add_rmsnorm(x, residual, w, eps, gemma)
    return reference.fused_add_rmsnorm(x, residual, w, eps, gemma)


def silu_and_mul(x):
    if use_native(x):
        return _native().silu_and_mul(x)
    return reference.silu_and_mul(x)


def gelu_and_mul(x, approximate="tanh"):
    if approximate == "tanh" and use_native_wide(x):
        return _native().gelu_tanh_and_mul(x)
    return reference.gelu_and_mul(x, approximate)


def sigmoid_gate(o, gate):
    """`o * sigmoid(gate)`, `[T, F]` each."""
    return (_native() if use_native_wide(o) else reference).sigmoid_gate(o, gate)


def clipped_swiglu(x, limit: float, alpha: float = 1.702, shift: float = 1.0):
    """`g * sigmoid(alpha g) * (u + shift)` of `x = [gate | up]`, `g = min(gate, limit)`, `u = clamp(up, -limit, limit)`."""
    return (_native() if use_native_wide(x) else reference).clipped_swiglu(x, limit, alpha, shift)


def swiglu(x):
    """`silu(gate) * up` of `x = [gate | up]`, any width, bf16 or fp32."""
    return clipped_swiglu(x, float("inf"), 1.0, 0.0)


def token_side_gate(z, table, ids, offset: int):
    """`gelu_tanh(z) * table[ids, offset : offset + dim]`, `z [T, dim]`."""
    return (_native() if use_native_wide(z) else reference).token_side_gate(z, table, ids, offset)


# ---- residual stream in fp32 (projections in the model's type)
def embed_scaled(ids, table, scale, positions=None, turns=None, out=None):
    """`table[ids] * scale` as `(fp32 stream, the same in the table's type)`.  `turns` (double, `[ceil(width / 2)]`): adds
    the sinusoidal vector of `positions`, channels 2i and 2i + 1 being sine and cosine of `turns[i]` turns a position.  With
    `out` (fp32) the stream goes there, and nothing is made of it in the table's type."""
    return (_native() if use_native_wide(table) else reference).embed_scaled(ids, table, scale, positions, turns, out)


def embed_pair(ids, table, pairs, mul_prev: int, mul_cur: int, slot_ids, fb):
    """`table[ids] + pairs[(previous id * mul_prev + id * mul_cur) mod buckets]` as `(fp32 stream, the same in the table's
    type)`; `pairs [buckets + 1, W]`, the last row is for a sequence's first token.  `slot_ids` int32: the id of the token in
    every slot of the KV pool, read for the predecessor of a portion's first token and written at the step's slots."""
    args = (ids, table, pairs, mul_prev, mul_cur, slot_ids, fb.positions, fb.out_cache_loc,
            None if fb.forward_mode.is_decode() else fb.cu_q_lens, fb.req_pool_indices, fb.page_table, fb.page_size)
    return (_native() if use_native_wide(table) else reference).embed_pair(*args)


def sum_norm(y, x, alpha, scale, weight, eps, **kw):
    """`x <- weight * z / rms(z)` in place on the fp32 stream with `z = alpha x + scale * (y_gate y + sum_j weights[t, j] c_j)`;
    `c_j` is row `pair_row[t, j]` of `expert_out` (negative: nothing), or x itself where `ids[t, j] >= experts`.  Returns x in
    y's type, or with `next_weight` (and `next_eps`) `next_weight * x / rms(x)`."""
    return (_native() if use_native_wide(y) else reference).sum_norm(y, x, alpha, scale, weight, eps, **kw)


def stream_add(y, x, expert_out=None, weights=None, pair_row=None):
    """`x += y` in place on the fp32 stream, with `expert_out` also `sum_j weights[t, j] * expert_out[pair_row[t, j]]`
    (negative rows: nothing); returns x in y's type."""
    return (_native() if use_native_wide(y) else reference).stream_add(y, x, expert_out, weights, pair_row)


def postnorm_add_norm(y, x, channel_scale, eps, next_scale, next_eps):
    """`x += channel_scale * y / rms(y)` in place on the fp32 stream; returns `next_scale * x / rms(x)` in y's type."""
    return (_native() if use_native_wide(y) else reference).postnorm_add_norm(y, x, channel_scale, eps, next_scale, next_eps)


def postnorm_add(y, x, channel_scale, eps):
    """`x += channel_scale * y / rms(y)` in place on the fp32 stream; returns x in y's type."""
    return (_native() if use_native_wide(y) else reference).postnorm_add(y, x, channel_scale, eps)


def rmsnorm_stream(x, weight, eps, dtype):
    """`x / rms(x) * weight` of the fp32 stream, in `dtype`."""
    return (_native() if use_native_wide(x) else reference).rmsnorm_stream(x, weight, eps, dtype)


def layernorm_stream(x, weight, bias, eps, dtype):
    """Layer norm of the fp32 stream, in `dtype`."""
    return (_native() if use_native_wide(x) else reference).layernorm_stream(x, weight, bias, eps, dtype)


def layernorm_add(y, x, out, weight, bias, eps, next_weight, next_bias, next_eps, **kw):
    """`r = x + LN(y + sum_j weights[t, j] * expert_out[pair_row[t, j]])` on fp32 streams (negative rows: nothing); `out <- r`,
    or with `history [>= n, T, W]` and `coefs [n]`: `history[n - 1] <- r` and `out <- sum_j coefs[j] * history[j]`.  `out` may be
    x.  Returns the next layer norm of `out` in y's type."""
    return (_native() if use_native_wide(y) else reference).layernorm_add(y, x, out, weight, bias, eps, next_weight, next_bias,
                                                                          next_eps, **kw)


def squared_relu(x):
    """`max(x, 0)^2`."""
    return (_native() if use_native_wide(x) else reference).squared_relu(x)


def softcap(x, cap: float):
    """`cap * tanh(x / cap)` in fp32; `x [T, V]` with any row stride."""
    return (_native() if use_native_wide(x) else reference).softcap(x, cap)


# ---- state-space duality (see `native.ssd_mix`)
def ssd_mix(proj, *a, **kw):
    return (_native() if use_native_wide(proj) else reference).ssd_mix(proj, *a, **kw)


# ---- gated delta rule (see `native.delta_scan`)
def delta_scan(proj, *a, **kw):
    return (_native() if use_native_wide(proj) else reference).delta_scan(proj, *a, **kw)


def delta_gate(o, gate, weight, eps, act: str = "silu", **kw):
    """`rmsnorm(o) * weight * act(gate)` per head, act silu or sigmoid (`kw`: see `native.delta_gate`)."""
    return (_native() if use_native_wide(gate) else reference).delta_gate(o, gate, weight, eps, act, **kw)


def delta_supported(x, conv_state, state, dim: int, vdim: int, taps: int) -> bool:
    """Whether `delta_scan` runs as kernels for these inputs and pools (the statements of `ops/linear_attention.py` otherwise)."""
    return (use_native_wide(x) and conv_state.dtype == x.dtype and state.dtype == torch.float32 and conv_state.is_contiguous()
            and state.is_contiguous() and 1 <= dim <= 256 and vdim >= 1 and 2 <= taps <= 16)


def linear_part(x, w):
    """`x @ w^T` of a column range of a wider product."""
    if use_native(x) and w.dtype == torch.bfloat16:
        return _native().linear_part(x, w)
    return reference.linear(x, w)


# ---- windowed attention over `PackedKVPool` rows (see `native.attn_prep`)
def attn_prep(proj, *a, **kw):
    return (_native() if use_native_wide(proj) else reference).attn_prep(proj, *a, **kw)


def attn_prep_rows(proj, *a, **kw):
    return (_native() if use_native_wide(proj) else reference).attn_prep_rows(proj, *a, **kw)


def window_attention(q, gate, cache, fb, rows, lens, dim, v_dim, scale, window, keep_first, **terms):
    """Every query token on its own: query n sees the first `lens[n]` tokens of page-table row `rows[n]`, of those the last
    `window` (0: all) and the first `keep_first`.  `softcap` (0: none), `slope` and `sink` (fp32 per head, or None): scores are
    `softcap * tanh(score / softcap) - slope * distance`, and `exp(sink)` joins the denominator.  `chunked`: instead of the last
    keys those in the query's own run of `window` positions, counted from the sequence's start.  `sigmoid_bias` (fp32 per head,
    or None): a key's weight is `sigmoid(score + bias)`, and nothing is normalised.  The result is multiplied by `out_scale` and
    the gate and goes to `out [N, heads, v_dim]` (any token stride), if given."""
    n = _native()
    args = (q, gate, cache, fb.page_table, rows, lens, dim, v_dim, fb.page_size, scale, window, keep_first)
    if n.window_decode_supported(q, cache, dim, v_dim, fb.page_size):
        return n.window_decode(*args, max_seq_len=fb.max_seq_len, **terms)
    return n.window_attn_any(*args, **terms)


def window_extend_supported(q, cache, dim, v_dim) -> bool:
    return use_native(q) and _native().window_extend_supported(q, cache, dim, v_dim)


def window_extend(q, gate, cache, fb, plan, out, dim, v_dim, scale, window, keep_first, **terms):
    return _native().window_extend(q, gate, cache, fb.page_table, plan, out, dim, v_dim, scale, window, keep_first, **terms)


def low_rank_up(x, w):
    """Second product of a low-rank pair; `x` may be a column range of a wider output.  A library GEMM on the GPU."""
    return reference.linear(x, w)


def router_logits(x, weight, bias=None):
    """`x weight^T + bias` in fp32, whatever the operands' type."""
    if use_native(x):
        from . import moe_native
        if moe_native.router_logits_supported(x, weight, bias):
            return moe_native.router_logits(x, weight, bias)
    return reference.linear(x.float(), weight.float(), bias.float() if bias is not None else None)


def route_by_logit(x, weight, bias, top_k):
    """The `top_k` experts with the largest logits `x weight^T + bias` (fp32) and the softmax over them."""
    if use_native_wide(x) and weight.shape[0] <= 512 and top_k <= 16 and weight.dtype == x.dtype:
        from . import moe_native
        return moe_native.route_by_logit(x, weight, bias, top_k)
    return reference.route_by_logit(x, weight, bias, top_k)


def route_by_score(x, weight, correction, top_k, scale, choices: int, gated: bool = False, scoring: str = "softmax",
                   groups: tuple[int, int] | None = None):
    """`s = softmax(x weight[:choices]^T)` (fp32; or "sigmoid" of each), the `top_k` choices with the largest `s + correction`,
    weighted by `scale * s`; `groups = (count, keep)`: only those in the `keep` of `count` groups of neighbours whose two largest
    sum to most.  `gated`: the row behind them is a gate per token, whose sigmoid comes third (else None); further rows are
    padding."""
    args = (x, weight, correction, top_k, scale, choices, gated, scoring, groups)
    if use_native_wide(x) and choices <= 512 and top_k <= 16 and weight.dtype == x.dtype:
        from . import moe_native
        return moe_native.route_by_score(*args)
    return reference.route_by_score(*args)


# ---- latent attention (see `native.latent_prep`)
def latent_prep(proj, *a, **kw):
    return (_native() if use_native_wide(proj) else reference).latent_prep(proj, *a, **kw)


def head_product(x, w):
    """`x [T, H, K]` times `w [H, K, N]` per head, summed in fp32 -> `[T, H, N]` in x's type."""
    if use_native(x) and _native().head_product_supported(x, w):
        return _native().head_product(x, w)
    return reference.head_product(x, w)


def mla_prep_supported(q, *a) -> bool:
    return use_native(q) and _native().mla_prep_supported(q, *a)


def mla_prep(*a):
    return _native().mla_prep(*a)


def latent_rotate(q, *a):
    (_native() if use_native_wide(q) else reference).latent_rotate(q, *a)


def latent_attention(q_lat, q_pe, cache, fb, scale, rows=None, lens=None, window: int = 0, sink=None):
    """Absorbed attention of every query token over the cache rows it sees: `q_lat [T, H, R]`, `q_pe [T, H, rot]`,
    `cache [pages, P, >= R + rot]` -> `[T, H, R]`.  `rows`, `lens` (int32 `[T]`): page-table row and number of visible
    tokens of each query; None = the step's own tokens.  `window` (0: all): of those only the last; `sink` fp32 `[H]`: joins
    the softmax's denominator."""
    R = q_lat.shape[-1]
    if not use_native_wide(q_lat):
        assert rows is None
        decode = fb.forward_mode.is_decode()
        return reference.mla_paged_attention(q_lat, q_pe, cache[..., :R + q_pe.shape[-1]], fb.page_table,
                                             fb.req_pool_indices, fb.seq_lens, fb.page_size, scale, R,
                                             None if decode else fb.cu_q_lens, None if decode else fb.extend_prefix_lens,
                                             window=window, sink=sink)
    native = _native()
    if rows is None:
        if fb.forward_mode.is_decode():
            rows, lens = fb.req_pool_indices, fb.seq_lens
        else:
            from ..layers.extend_plan import extend_plan
            plan = extend_plan(fb, False)
            rows, lens = plan.token_rows, plan.token_lens
    if native.mla_decode_supported(q_lat, q_pe, cache, R, fb.page_size):
        return native.mla_decode(q_lat, q_pe, cache, fb.page_table, rows, lens, fb.page_size, scale, fb.max_seq_len,
                                 exact=True, window=window, sink=sink)
    return native.latent_attn_any(q_lat, q_pe, cache, fb.page_table, rows, lens, fb.page_size, scale, window, sink)


def latent_extend_supported(q, dim, rot, v_dim, rank) -> bool:
    return use_native(q) and _native().latent_extend_supported(q, dim, rot, v_dim, rank)


def latent_gather(*a):
    return _native().latent_gather(*a)


def latent_extend(*a, **kw):
    return _native().latent_extend(*a, **kw)


def linear(x, w, bias=None):
    if w.dtype != x.dtype and w.is_floating_point() and w.dtype.itemsize >= 2:
        # a per-module dtype (`--dtype-config`): compute in the weight's dtype, hand back the activations' dtype
        return reference.linear(x.to(w.dtype), w, bias.to(w.dtype) if bias is not None else None).to(x.dtype)
    if use_native(x) and w.dtype == torch.bfloat16:
        from ..parallel import state as ps
        comm = ps.get_state().fused_comm
        if comm is not None and comm.pending_gather is not None:
            # `x` may be a fused all-gather nobody has waited for yet: the GEMM waits per chunk of rows
            return comm.consume_linear(x, w, bias)
        return _native().linear(x, w, bias)
    return reference.linear(x, w, bias)


def linear_swiglu_supported(x, w) -> bool:
    """Whether `linear_swiglu` computes `silu_and_mul(linear(x, w))` for these operands: prefill sizes, whole blocks of K, and no fused
    all-gather that somebody has to wait for."""
    if not (use_native(x) and w.dtype == torch.bfloat16 and x.dim() == 2 and w.is_contiguous() and x.stride(1) == 1):
        return False
    from ..parallel import state as ps
    comm = ps.get_state().fused_comm
    return (x.shape[0] > 256 and x.shape[1] % 64 == 0 and w.shape[0] % 16 == 0 and x.stride(0) % 8 == 0 and x.stride(0) >= x.shape[1]
            and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0 and (comm is None or comm.pending_gather is None))


def linear_swiglu(x, w):
    """`silu(gate) * up`, gate and up the halves of `x w^T`, from the fp32 sums (no rounding in between)."""
    return _native().gemm_pair(x, w, gated=True)


def rope_qknorm_kvwrite(qkv, positions, cos_sin, q_norm_w, k_norm_w, eps, num_q_heads, num_kv_heads,
                        head_dim, kv_buffer, out_cache_loc, page_size, is_neox=True, rotary_dim=None,
                        gemma_norm=False):
    if use_native(qkv) and (kv_buffer is None or kv_buffer.dtype == torch.bfloat16):
        return _native().rope_qknorm_kvwrite(qkv, positions, cos_sin, q_norm_w, k_norm_w, eps, num_q_heads,
                                             num_kv_heads, head_dim, kv_buffer, out_cache_loc, page_size,
                                             is_neox, rotary_dim, gemma_norm)
    return reference.rope_qknorm_kvwrite(qkv, positions, cos_sin, q_norm_w, k_norm_w, eps, num_q_heads,
                                         num_kv_heads, head_dim, kv_buffer, out_cache_loc, page_size,
                                         is_neox, rotary_dim, gemma_norm)


def rope_parts_supported(q, k, v, positions, cos_sin, q_norm_w, k_norm_w, kv_buffer, *a) -> bool:
    """Whether queries, keys and values that lie apart need not be concatenated for `rope_qknorm_kvwrite`."""
    return use_native(q) and kv_buffer.dtype == torch.bfloat16 and \
        _native().rope_parts_supported(q, k, v, positions, cos_sin, q_norm_w, k_norm_w, kv_buffer, *a)


def rope_parts(*a):
    return _native().rope_parts(*a)


def paged_attention(q, kv_buffer, page_table, req_pool_indices, seq_lens, page_size, scale,
                    cu_q_lens=None, prefix_lens=None, sliding_window=0, soft_cap=0.0, sinks=None,
                    custom_mask=None, max_q_len=0, max_seq_len=0):
    compact_mask = custom_mask is None or (custom_mask.dim() == 3 and cu_q_lens is not None)
    if use_native(q) and kv_buffer.dtype == torch.bfloat16 and sinks is None and compact_mask \
            and q.shape[-1] in (64, 128):
        return _native().paged_attention(q, kv_buffer, page_table, req_pool_indices, seq_lens, page_size,
                                         scale, cu_q_lens, prefix_lens, sliding_window, soft_cap,
                                         max_q_len, max_seq_len, tail_mask=custom_mask)
    return reference.paged_attention(q, kv_buffer, page_table, req_pool_indices, seq_lens, page_size, scale,
                                     cu_q_lens, prefix_lens, sliding_window, soft_cap, sinks, custom_mask)


def embedding(ids, table, vocab_start=0, masked=False):
    if use_native(table) and ids.dtype == torch.int32:
        return _native().embedding(ids, table, vocab_start, masked)
    return reference.embedding(ids, table, vocab_start, masked)


def argmax(logits):
    """Greedy pick per row; the first maximal index wins."""
    if (not _FORCE_REFERENCE) and logits.is_cuda and logits.dtype in (torch.float32, torch.bfloat16):
        return _native().argmax(logits)
    return torch.argmax(logits, dim=-1).to(torch.int32)


def topk_route(router_logits, top_k, scoring="softmax", renormalize=True, correction_bias=None,
               num_expert_group=0, topk_group=0, routed_scaling_factor=1.0):
    if (not _FORCE_REFERENCE) and router_logits.is_cuda and router_logits.shape[-1] <= 512 and top_k <= 16 \
            and router_logits.dtype in (torch.float32, torch.bfloat16):
        from . import moe_native
        return moe_native.topk_route(router_logits, top_k, scoring, renormalize, correction_bias,
                                     num_expert_group, topk_group, routed_scaling_factor)
    return reference.topk_route(router_logits, top_k, scoring, renormalize, correction_bias,
                                num_expert_group, topk_group, routed_scaling_factor)


def fused_experts(x, w13, w2, topk_weights, topk_ids, expert_start=0, workspace=None, add=None):
    """Routed-expert FFN: `w13 [E_local, 2I, H]` (gate rows then up rows), `w2 [E_local, H, I]`."""
    if use_native(x) and w13.dtype == torch.bfloat16 and x.shape[-1] % 8 == 0 and w2.shape[-1] % 8 == 0:
        from . import moe_native
        return moe_native.fused_experts(x, w13, w2, topk_weights, topk_ids, expert_start, workspace, add)
    y = reference.moe_forward(x, w13, w2, topk_weights, topk_ids, expert_start)
    return y if add is None else (y.float() + add.float()).to(y.dtype)


def mla_tokens_supported(q_pe, cache, heads: int, rank: int, page_size: int) -> bool:
    """Whether single query tokens with latent queries `[T, heads, rank]` can go through `mla_tokens`."""
    probe = q_pe.new_empty(0, heads, rank)
    return use_native(q_pe) and _native().mla_decode_supported(probe, q_pe, cache, rank, page_size)


def mla_tokens(q_latent, q_pe, cache, fb, scale, rows, lens):
    """Absorbed attention of query tokens on their own, weights as sums of two bf16 numbers: query n sees the first `lens[n]` tokens
    of page-table row `rows[n]`."""
    return _native().mla_decode(q_latent, q_pe, cache, fb.page_table, rows, lens, fb.page_size, scale, fb.max_seq_len, exact=True)


def mla_paged_attention(q_latent, q_pe, kv_buffer, page_table, req_pool_indices, seq_lens, page_size, scale,
                        kv_lora_rank, cu_q_lens=None, prefix_lens=None, allowed=None, max_seq_len=0):
    """Absorbed-MLA attention over the latent cache `[pages, P, kv_lora_rank + rope_dim]`."""
    if use_native(q_latent) and cu_q_lens is None and allowed is None and req_pool_indices.dtype == torch.int32 \
            and _native().mla_decode_supported(q_latent, q_pe, kv_buffer, kv_lora_rank, page_size):
        return _native().mla_decode(q_latent, q_pe, kv_buffer, page_table, req_pool_indices, seq_lens, page_size,
                                    scale, max_seq_len)
    return reference.mla_paged_attention(q_latent, q_pe, kv_buffer, page_table, req_pool_indices, seq_lens,
                                         page_size, scale, kv_lora_rank, cu_q_lens, prefix_lens, allowed)
