"""ctypes bindings of the MoE kernels (`csrc/moe.cu`, grouped GEMM in `csrc/gemm_sm100.cu`)."""

from __future__ import annotations

from ctypes import c_float, c_int, c_longlong, c_size_t, c_void_p

import torch

from . import native

_bound = False


def _lib():
    global _bound
    L = native.lib()
    if not _bound:
        L.sglb_topk_route.argtypes = [c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int,
                                      c_int, c_int, c_float, c_void_p]
        L.sglb_router_logits.argtypes = [c_void_p, c_void_p, c_longlong, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p]
        L.sglb_gemm_pair_grouped.argtypes = [c_void_p] * 7 + [c_int] * 6 + [c_void_p]
        L.sglb_moe_align.argtypes = [c_void_p, c_int, c_int, c_int, c_int, c_int, c_void_p, c_void_p, c_void_p, c_void_p,
                                     c_void_p, c_void_p, c_void_p, c_void_p]
        L.sglb_moe_gather.argtypes = [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_void_p]
        L.sglb_moe_combine.argtypes = [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p, c_void_p]
        L.sglb_grouped_gemm_bf16.argtypes = [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                                             c_int, c_int, c_int, c_int, c_void_p, c_size_t, c_void_p, c_void_p]
        L.sglb_route_by_logit.argtypes = [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int,
                                          c_int, c_int, c_void_p]
        L.sglb_route_by_score.argtypes = [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int,
                                          c_int, c_int, c_int, c_float, c_int, c_int, c_int, c_int, c_void_p]
        L.sglb_grouped_gemm_any.argtypes = [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                                            c_int, c_int, c_int, c_int, c_int, c_void_p]
        L.sglb_grouped_gemm_fp8.argtypes = [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                                            c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_void_p, c_size_t,
                                            c_void_p, c_void_p]
        _bound = True
    return L


_SCORING = {"softmax": 0, "sigmoid": 1, "tanh": 2}


def topk_route(router_logits, top_k, scoring="softmax", renormalize=True, correction_bias=None,
               num_expert_group=0, topk_group=0, routed_scaling_factor=1.0):
    T, E = router_logits.shape
    router_logits = router_logits.contiguous()
    w = torch.empty((T, top_k), dtype=torch.float32, device=router_logits.device)
    ids = torch.empty((T, top_k), dtype=torch.int32, device=router_logits.device)
    bias = correction_bias.float().contiguous() if correction_bias is not None else None
    rc = _lib().sglb_topk_route(router_logits.data_ptr(), router_logits.element_size(),
                                bias.data_ptr() if bias is not None else None, w.data_ptr(), ids.data_ptr(), T, E,
                                top_k, _SCORING[scoring], int(renormalize), int(num_expert_group or 0),
                                int(topk_group or 0), float(routed_scaling_factor), native._stream())
    native._check(rc, "topk_route")
    return w, ids


def router_logits_supported(x, weight, bias=None) -> bool:
    return (x.dim() == weight.dim() == 2 and x.dtype == weight.dtype == torch.bfloat16 and weight.is_contiguous()
            and x.shape[1] == weight.shape[1] > 0 and x.shape[1] % 32 == 0 and weight.shape[0] > 0
            and x.stride(1) == 1 and x.stride(0) % 8 == 0 and x.stride(0) >= x.shape[1] and x.data_ptr() % 16 == 0
            and weight.data_ptr() % 16 == 0 and x.device == weight.device
            and (bias is None or (bias.dtype == torch.bfloat16 and bias.is_contiguous() and bias.shape == weight.shape[:1]
                                  and bias.device == x.device)))


def router_logits(x, weight, bias=None):
    """`x [T, K] @ weight [E, K]^T (+ bias)` in fp32 arithmetic from bf16 operands."""
    T, K = x.shape
    out = torch.empty((T, weight.shape[0]), dtype=torch.float32, device=x.device)
    native._check(_lib().sglb_router_logits(out.data_ptr(), x.data_ptr(), x.stride(0), weight.data_ptr(), native._p(bias), T,
                                            weight.shape[0], K, native._stream()), "router_logits")
    return out


# rows of a token tile in the lists of `moe_align`, where a kernel does not want others
TILE_ROWS = 128


class MoeWorkspace:
    """Index buffers of one MoE layer call, sized for `max_pairs` routed (token, expert) pairs and tiles of at least 32 rows."""

    def __init__(self, max_pairs: int, num_local_experts: int, device):
        self.max_pairs = max_pairs
        i32 = dict(dtype=torch.int32, device=device)
        self.offsets = torch.zeros(num_local_experts + 1, **i32)
        self.pair_row = torch.empty(max_pairs, **i32)
        self.row_token = torch.empty(max_pairs, **i32)
        self.tile_group = torch.empty(max_pairs // 32 + num_local_experts + 1, **i32)
        self.tile_row0 = torch.empty(max_pairs // 32 + num_local_experts + 1, **i32)
        self.tile_rows = TILE_ROWS
        self.counts = torch.zeros(2, **i32)


def moe_align(topk_ids, expert_start, num_local_experts, ws: MoeWorkspace, expert_hist=None, tile_rows: int = TILE_ROWS):
    T, k = topk_ids.shape
    assert tile_rows >= 32
    ws.tile_rows = tile_rows
    rc = _lib().sglb_moe_align(topk_ids.data_ptr(), T * k, k, expert_start, num_local_experts, tile_rows, ws.offsets.data_ptr(),
                               ws.pair_row.data_ptr(), ws.row_token.data_ptr(), ws.tile_group.data_ptr(),
                               ws.tile_row0.data_ptr(), ws.counts.data_ptr(),
                               expert_hist.data_ptr() if expert_hist is not None else None, native._stream())
    native._check(rc, "moe_align")


def moe_gather(x, ws: MoeWorkspace, max_rows: int):
    H = x.shape[-1]
    out = torch.empty((max_rows, H), dtype=x.dtype, device=x.device)
    rc = _lib().sglb_moe_gather(out.data_ptr(), x.data_ptr(), ws.row_token.data_ptr(), ws.counts.data_ptr(),
                                max_rows, H, native._stream())
    native._check(rc, "moe_gather")
    return out


def on_pairs(rows: int, K: int, experts: int, expected: int | None = None) -> bool:
    """Whether a grouped product of `rows` rows at most (`expected` of them, where others may be other ranks') runs on pairs of SMs
    (`csrc/gemm_pair.cu`): its maps want whole blocks of 64 lanes.  Up to 256 rows the other kernel shares the bytes of all experts
    out evenly over all SMs, which is good while most of few experts are chosen.  Both products of 768 x 2048, pairs against that, 64
    experts: 37 / 66 us at 8 rows, 96 / 88 at 56, 125 / 118 at 128, 135 / 137 at 256; 128 experts: 117 / 134 at 64 rows, 206 / 232 at 256.
    Whole layers at other sizes, rows spread evenly: 16 experts of 1408 x 4096 98 / 92 at 32 rows, 103 / 140 at 256, 48 of them 149 / 165 and
    263 / 343; 80 of 768 x 2048 81 / 96 at 64 rows, 128 / 158 at 256, 112 of them 93 / 116 and 162 / 216.  So from some 48 experts on and for
    wider ones the line is on the safe side: what it sends to the other kernel there would be faster in pairs."""
    return K % 64 == 0 and (rows > 256 or experts >= 128 or 2 * (rows if expected is None else expected) <= experts)


def pair_tile(rows: int, experts: int) -> int:
    """Rows of a token tile for `rows` pairs over `experts`: an expert's rows in one tile where 256 hold them (with a quarter to
    spare, as tokens are not spread evenly: a second tile reads all of the weights again), else in few of equal size.
    Both products of 64 experts of 768 x 2048, tiles of 64 / 128 / 192 / 256: 182 / 158 / 154 / 154 us at 1024 tokens x 8, 304 / 232 / 215
    / 223 at 2500, 387 / 271 / 248 / 243 at 3000; in 128-row tiles of single SMs with the activation of its own 180, 275 and 315."""
    mean = max(rows // max(experts, 1), 1)
    n = -(-mean // 256)
    return min(256, -(-mean * 5 // (4 * n * 32)) * 32)


def expert_tile(pairs: int, hidden: int, inner: int, local: int, experts: int) -> int:
    """Rows of a token tile for both products of `local` of all `experts` on pairs of SMs, 0 where they run elsewhere.  `pairs` (token,
    choice) pairs of the step are spread over all experts, those of other ranks too: this rank's rows are its share of them."""
    rows = -(-pairs * local // max(experts, 1))
    if on_pairs(pairs, hidden, local, rows) and on_pairs(pairs, inner, local, rows):
        return pair_tile(rows, local)
    return 0


def grouped_gemm_pair(x_sorted, w, ws: MoeWorkspace, rows: int, gated: bool = False):
    """`grouped_gemm` on pairs of SMs; `gated`: `w [E_local, 2 N, K]` holds gate, then up rows, the result is `silu(gate) * up` of the
    fp32 sums."""
    E, N, K = w.shape
    N //= 2 if gated else 1
    out = torch.empty((rows, N), dtype=x_sorted.dtype, device=x_sorted.device)
    rc = _lib().sglb_gemm_pair_grouped(x_sorted.data_ptr(), w.data_ptr(), out.data_ptr(), ws.offsets.data_ptr(), ws.tile_group.data_ptr(),
                                       ws.tile_row0.data_ptr(), ws.counts.data_ptr() + 4, rows, N, K, E, int(gated), ws.tile_rows,
                                       native._stream())
    native._check(rc, "gemm_pair_grouped")
    return out


def grouped_gemm(x_sorted, w, ws: MoeWorkspace, rows: int):
    """`x_sorted [rows, K]` (rows sorted by expert), `w [E_local, N, K]` -> `[rows, N]`."""
    E, N, K = w.shape
    if on_pairs(rows, K, E):
        return grouped_gemm_pair(x_sorted, w, ws, rows)
    assert ws.tile_rows == TILE_ROWS or rows <= 256
    out = torch.empty((rows, N), dtype=x_sorted.dtype, device=x_sorted.device)
    sc = native.gemm_scratch(x_sorted.device)
    rc = _lib().sglb_grouped_gemm_bf16(x_sorted.data_ptr(), w.data_ptr(), out.data_ptr(), ws.offsets.data_ptr(),
                                       ws.tile_group.data_ptr(), ws.tile_row0.data_ptr(),
                                       ws.counts.data_ptr() + 4, rows, N, K, E, sc.workspace.data_ptr(), sc.bytes,
                                       sc.counters.data_ptr(), native._stream())
    native._check(rc, "grouped_gemm")
    return out


def grouped_gemm_fp8(xq_sorted, scale_x, wq, scale_w, ws: MoeWorkspace, rows: int):
    """e4m3 grouped GEMM on the tcgen05 `kind::f8f6f4` path: `xq_sorted [rows, K]` with per-row scales
    `scale_x [rows]`, `wq [E_local, N, K]` with per-output-channel scales `scale_w [E_local, N]` -> bf16 `[rows, N]`."""
    E, N, K = wq.shape
    assert xq_sorted.dtype == torch.float8_e4m3fn and wq.dtype == torch.float8_e4m3fn
    assert scale_x.dtype == torch.float32 and scale_w.dtype == torch.float32
    assert scale_x.numel() >= rows and scale_w.numel() == E * N and K % 16 == 0
    out = torch.empty((rows, N), dtype=torch.bfloat16, device=xq_sorted.device)
    sc = native.gemm_scratch(xq_sorted.device)
    rc = _lib().sglb_grouped_gemm_fp8(xq_sorted.data_ptr(), wq.data_ptr(), scale_x.data_ptr(), scale_w.data_ptr(),
                                      out.data_ptr(), ws.offsets.data_ptr(), ws.tile_group.data_ptr(),
                                      ws.tile_row0.data_ptr(), ws.counts.data_ptr() + 4, rows, N, K, E,
                                      sc.workspace.data_ptr(), sc.bytes, sc.counters.data_ptr(), native._stream())
    native._check(rc, "grouped_gemm_fp8")
    return out


def fused_experts_fp8(x, w13_q, w13_scale, w2_q, w2_scale, topk_weights, topk_ids, expert_start: int = 0,
                      ws: MoeWorkspace | None = None, add=None, out=None):
    """W8A8 e4m3 routed-expert FFN: align -> gather -> per-token quantise -> grouped fp8 GEMM (gate|up) ->
    fused SiLU*mul + per-token quantise -> grouped fp8 GEMM (down) -> weighted combine.  Weights are per-channel
    quantised (`w13_q [E_local, 2I, H]`, `w13_scale [E_local, 2I]`, `w2_q [E_local, H, I]`, `w2_scale [E_local, H]`)."""
    T, H = x.shape
    k = topk_ids.shape[1]
    E_local = w13_q.shape[0]
    pairs = T * k
    if ws is None or ws.max_pairs < pairs:
        ws = MoeWorkspace(pairs, E_local, x.device)
    moe_align(topk_ids, expert_start, E_local, ws)
    xs = moe_gather(x, ws, pairs)
    valid = ws.counts[0:1]
    xq, sx = native.quant_fp8_rows(xs, valid_rows=valid)
    h = grouped_gemm_fp8(xq, sx, w13_q, w13_scale, ws, pairs)
    aq, sa = native.quant_fp8_rows(h, gated=True, valid_rows=valid)
    y = grouped_gemm_fp8(aq, sa, w2_q, w2_scale, ws, pairs)
    return moe_combine(y, topk_weights, ws, T, add=add, out=out)


def grouped_gemm_fp8_block(xq_sorted, sx, wq, sw, ws: MoeWorkspace, rows: int):
    """Block-scaled e4m3 grouped GEMM: `xq_sorted [rows, K]` with group scales `sx [K/128, >=rows]`, `wq [E, N, K]`
    with `sw [E, N/128, K/128]` -> bf16 `[rows, N]` (`csrc/gemm_fp8_block.cu`)."""
    E, N, K = wq.shape
    out = torch.empty((rows, N), dtype=torch.bfloat16, device=xq_sorted.device)
    L = _lib()
    L.sglb_grouped_gemm_fp8_block.argtypes = [c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_void_p, c_void_p,
                                              c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_void_p]
    rc = L.sglb_grouped_gemm_fp8_block(xq_sorted.data_ptr(), wq.data_ptr(), sx.data_ptr(), sx.shape[1], sw.data_ptr(),
                                       out.data_ptr(), ws.offsets.data_ptr(), ws.tile_group.data_ptr(),
                                       ws.tile_row0.data_ptr(), ws.counts.data_ptr() + 4, rows, N, K, E,
                                       native._stream())
    native._check(rc, "grouped_gemm_fp8_block")
    return out


def fused_experts_fp8_block(x, w13_q, w13_scale, w2_q, w2_scale, topk_weights, topk_ids, expert_start: int = 0,
                            ws: MoeWorkspace | None = None, add=None, out=None):
    """Routed-expert FFN on 128 x 128 block-scaled e4m3 weights (DeepSeek-V3 format) with per-token-group-128
    activation scales: align -> gather -> group quantise -> grouped block GEMM (gate|up) -> SiLU*mul -> group
    quantise -> grouped block GEMM (down) -> weighted combine."""
    T, H = x.shape
    k = topk_ids.shape[1]
    E_local = w13_q.shape[0]
    pairs = T * k
    if ws is None or ws.max_pairs < pairs:
        ws = MoeWorkspace(pairs, E_local, x.device)
    moe_align(topk_ids, expert_start, E_local, ws)
    xs = moe_gather(x, ws, pairs)
    valid = ws.counts[0:1]
    xq, sx = native.quant_fp8_group128(xs, valid_rows=valid)
    h = grouped_gemm_fp8_block(xq, sx, w13_q, w13_scale, ws, pairs)
    a = native.silu_and_mul(h)
    aq, sa = native.quant_fp8_group128(a, valid_rows=valid)
    y = grouped_gemm_fp8_block(aq, sa, w2_q, w2_scale, ws, pairs)
    return moe_combine(y, topk_weights, ws, T, add=add, out=out)


def moe_combine(y_sorted, topk_weights, ws: MoeWorkspace, T: int, add=None, out=None):
    k = topk_weights.shape[1]
    H = y_sorted.shape[1]
    if out is None:
        out = torch.empty((T, H), dtype=y_sorted.dtype, device=y_sorted.device)
    rc = _lib().sglb_moe_combine(out.data_ptr(), y_sorted.data_ptr(), topk_weights.data_ptr(), ws.pair_row.data_ptr(),
                                 T, k, H, add.data_ptr() if add is not None else None, native._stream())
    native._check(rc, "moe_combine")
    return out


def fused_experts(x, w13, w2, topk_weights, topk_ids, expert_start: int = 0, ws: MoeWorkspace | None = None,
                  add=None, out=None, experts: int | None = None):
    """Routed-expert FFN with the native kernels: align -> gather -> grouped GEMM (gate|up) -> SiLU*mul ->
    grouped GEMM (down) -> weighted combine.  `w13 [E_local, 2I, H]`, `w2 [E_local, H, I]`; `experts`: of all ranks (None: these)."""
    T, H = x.shape
    k = topk_ids.shape[1]
    E_local = w13.shape[0]
    pairs = T * k
    if ws is None or ws.max_pairs < pairs:
        ws = MoeWorkspace(pairs, E_local, x.device)
    tile = expert_tile(pairs, H, w2.shape[2], E_local, experts or E_local)
    if tile:
        moe_align(topk_ids, expert_start, E_local, ws, tile_rows=tile)
        y = grouped_gemm_pair(grouped_gemm_pair(moe_gather(x, ws, pairs), w13, ws, pairs, gated=True), w2, ws, pairs)
    else:
        moe_align(topk_ids, expert_start, E_local, ws)
        y = grouped_gemm(native.silu_and_mul(grouped_gemm(moe_gather(x, ws, pairs), w13, ws, pairs)), w2, ws, pairs)
    return moe_combine(y, topk_weights, ws, T, add=add, out=out)


# tokens up to which the router is one launch; above, its product is a library GEMM with fp32 results
ROUTE_FUSED_TOKENS = 256


def route_by_logit(x, weight, bias, top_k):
    """`z = x weight^T + bias` in fp32, the `top_k` largest (ties: the lower index) and their softmax."""
    T, K = x.shape
    E = weight.shape[0]
    x = x.contiguous()
    assert weight.is_contiguous() and weight.dtype == x.dtype and (bias is None or bias.dtype == x.dtype)
    w = torch.empty((T, top_k), dtype=torch.float32, device=x.device)
    ids = torch.empty((T, top_k), dtype=torch.int32, device=x.device)
    z = None
    if T > ROUTE_FUSED_TOKENS:
        z = torch.mm(x, weight.t()) if x.dtype == torch.float32 else torch.mm(x, weight.t(), out_dtype=torch.float32)
    p = native._p
    native._check(_lib().sglb_route_by_logit(p(z), p(x), p(weight), p(bias), p(w), p(ids), T, E, K, top_k, native._f32(x),
                                             native._stream()), "route_by_logit")
    return w, ids


def route_by_score(x, weight, correction, top_k, scale, choices, gated: bool = False, scoring: str = "softmax", groups=None):
    """`s = softmax(x weight[:choices]^T)` in fp32 (or "sigmoid" of each), the `top_k` largest `s + correction` (ties: the lower
    index) and `scale * s` of those; `groups = (count, keep)`: among the best groups only (`ops.route_by_score`).  `gated`: the
    sigmoid of the next row's product is returned too (`[T]`, else None)."""
    T, K = x.shape
    E = choices
    x = x.contiguous()
    assert weight.is_contiguous() and weight.dtype == x.dtype
    assert correction is None or (correction.dtype == torch.float32 and correction.numel() == E)
    w = torch.empty((T, top_k), dtype=torch.float32, device=x.device)
    ids = torch.empty((T, top_k), dtype=torch.int32, device=x.device)
    gate = torch.empty(T, dtype=torch.float32, device=x.device) if gated else None
    z = None
    if T > ROUTE_FUSED_TOKENS or (K % 8 == 0 and weight.shape[0] % 8 == 0):     # (a split product beats one CTA per token)
        z = torch.mm(x, weight.t()) if x.dtype == torch.float32 else torch.mm(x, weight.t(), out_dtype=torch.float32)
    p = native._p
    native._check(_lib().sglb_route_by_score(p(z), p(x), p(weight), p(correction), p(w), p(ids), p(gate), T, weight.shape[0], E, K,
                                             top_k, float(scale), int(scoring == "sigmoid"), *(groups or (0, 0)),
                                             native._f32(x), native._stream()), "route_by_score")
    return w, ids, gate


def grouped_gemm_any(x, row_token, w, ws: MoeWorkspace, rows: int):
    """Grouped product of any sizes in bf16 or fp32 on the CUDA cores, fp32 accumulation: row r of the result is row
    `row_token[r]` (None: r) of `x` times its expert's `w [E_local, N, K]`."""
    E, N, K = w.shape
    assert x.is_contiguous() and w.is_contiguous() and x.dtype == w.dtype and x.shape[1] == K
    out = torch.empty((rows, N), dtype=x.dtype, device=x.device)
    native._check(_lib().sglb_grouped_gemm_any(x.data_ptr(), native._p(row_token), w.data_ptr(), out.data_ptr(),
                                               ws.offsets.data_ptr(), ws.tile_group.data_ptr(), ws.tile_row0.data_ptr(),
                                               ws.counts.data_ptr() + 4, rows, N, K, E, native._f32(x), native._stream()),
                  "grouped_gemm_any")
    return out


def sorted_experts(x, w13, w2, topk_ids, expert_start, ws: MoeWorkspace, act):
    """Outputs of the routed experts, one row per (token, choice) pair in the workspace's order (`ws.pair_row`)."""
    pairs, E_local = topk_ids.numel(), w13.shape[0]
    moe_align(topk_ids, expert_start, E_local, ws)
    if x.dtype == torch.bfloat16 and x.shape[1] % 8 == 0 and w2.shape[2] % 8 == 0:
        return grouped_gemm(act(grouped_gemm(moe_gather(x, ws, pairs), w13, ws, pairs)), w2, ws, pairs)
    return grouped_gemm_any(act(grouped_gemm_any(x.contiguous(), ws.row_token, w13, ws, pairs)), None, w2, ws, pairs)
