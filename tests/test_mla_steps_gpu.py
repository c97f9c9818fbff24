"""Steps of `MLAAttention` on the GPU: preparation of latents and queries, extends by tiles and by tokens."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from sglang_jax_b200 import ops
from sglang_jax_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H,dim,rot,rank,split,rope", [(1, 1, 8, 8, 8, False, True), (37, 3, 40, 16, 136, False, True),
                                                         (37, 3, 40, 16, 136, True, True), (130, 16, 128, 64, 512, False, True),
                                                         (5, 16, 128, 64, 512, False, False)])
@pytest.mark.parametrize("gemma", [False, True])
def test_mla_prep(T, H, dim, rot, rank, split, rope, gemma):
    torch.manual_seed(T + rank)
    dev, bf = "cuda", torch.bfloat16
    q = torch.randn(T, H, dim + rot, device=dev, dtype=bf)
    lat = torch.randn(T, rank + rot, device=dev, dtype=bf)
    w = torch.randn(rank, device=dev, dtype=bf)
    cache = torch.zeros(T // 4 + 2, 8, rank + rot + 8, device=dev, dtype=bf)
    loc = torch.randperm(cache.shape[0] * 8, device=dev)[:T].int()
    pos = torch.randint(0, 300, (T,), device=dev, dtype=torch.int32)
    cs = ref.build_cos_sin_cache(rot, 300, 1e4, device=dev) if rope else None
    assert ops.mla_prep_supported(q, lat, cache, w, cs, pos, loc, rank, split)
    want_q, pe = q.clone(), lat[:, None, rank:]
    if rope:
        want_q[..., dim:] = ref.apply_rope(q[..., dim:], pos, cs, split)
        pe = ref.apply_rope(pe, pos, cs, split)
    x = lat[:, :rank].double()
    c = x / (x.pow(2).mean(-1, keepdim=True) + 1e-6).sqrt() * (w.double() + (1.0 if gemma else 0.0))
    want = torch.zeros_like(cache).flatten(0, 1)
    want[loc.long(), :rank + rot] = torch.cat([c.to(bf), pe[:, 0]], -1)
    ops.mla_prep(q, lat, w, 1e-6, gemma, cs, split, pos, loc, cache)
    # one rounding of fp32 arithmetic each: a last place of bf16 apart at most
    torch.testing.assert_close(q, want_q, rtol=2 ** -7, atol=1e-6)
    torch.testing.assert_close(cache.flatten(0, 1), want, rtol=2 ** -7, atol=1e-6)


@pytest.mark.parametrize("news,prefixes", [([1], [0]), ([31, 1], [5, 200]), ([32], [0]), ([257, 3, 0, 64], [0, 70, 9, 129]),
                                           ([300, 40], [1, 64])])
@pytest.mark.parametrize("page", [16, 64])
def test_mla_extend(news, prefixes, page):
    """Long sequences by tiles, short ones token by token, against the statements in 64 bits over the same cache."""
    from sglang_jax_b200.models.deepseek_v3 import MLAAttention
    torch.manual_seed(sum(news))
    dev, bf = torch.device("cuda"), torch.bfloat16
    cfg = SimpleNamespace(hidden_size=256, num_attention_heads=4, qk_nope_head_dim=64, qk_rope_head_dim=32, v_head_dim=96,
                          kv_lora_rank=128, q_lora_rank=None, rms_norm_eps=1e-6, max_position_embeddings=1024)
    with torch.device(dev):
        m = MLAAttention(cfg, 0, bf)
    for p in m.parameters():
        p.data.normal_(0, 0.06)
    m.kv_a_layernorm.weight.data.add_(1.0)
    m.absorb()
    n, pre = np.asarray(news), np.asarray(prefixes)
    B, T, total = len(n), int(n.sum()), n + pre
    pages = [-(-int(t) // page) for t in total]
    order = torch.randperm(sum(pages)) + 1
    table = torch.zeros(B, max(pages) + 1, dtype=torch.int32)
    at = 0
    for b in range(B):
        table[b, :pages[b]] = order[at:at + pages[b]].int()
        at += pages[b]
    cache = torch.randn(sum(pages) + 1, page, 160, device=dev, dtype=bf)
    pos = np.concatenate([np.arange(a, a + c) for a, c in zip(pre, n)]).astype(np.int32)
    seq = np.repeat(np.arange(B), n)
    loc = table.numpy()[seq, pos // page] * page + pos % page
    t = lambda v: torch.from_numpy(np.asarray(v, np.int32)).to(dev)
    mode = SimpleNamespace(is_decode=lambda: False)
    fb = SimpleNamespace(positions=t(pos), out_cache_loc=t(loc), page_table=table.to(dev), req_pool_indices=t(np.arange(B)),
                         seq_lens=t(total), page_size=page, extend_seq_lens_cpu=n, extend_prefix_lens_cpu=pre,
                         extend_seq_lens=t(n), extend_prefix_lens=t(pre), cu_q_lens=t(np.concatenate([[0], np.cumsum(n)])),
                         num_tokens=T, max_seq_len=int(total.max()), forward_mode=mode, extras={},
                         token_to_kv_pool=SimpleNamespace(get_kv_buffer=lambda _: cache))
    x = torch.randn(T, 256, device=dev, dtype=bf)
    seen = {}
    extend = m._extend
    m._extend = lambda q, *a: seen.setdefault("o", extend(seen.setdefault("q", q), *a))
    got = m(x, fb)
    q, rows = seen["q"].double(), cache.flatten(0, 1).double()
    up = m.w_up.double()
    want = torch.zeros(T, 4, 96, device=dev, dtype=torch.float64)
    for i in range(T):
        b, s = seq[i], int(pos[i]) + 1
        slots = (table[b].long()[:, None] * page + torch.arange(page)).flatten()[:s].to(dev)
        c, pe = rows[slots, :128], rows[slots, 128:]
        ql = torch.einsum("hn,hnr->hr", q[i, :, :64], up[:, :64])
        p = torch.softmax((ql @ c.t() + q[i, :, 64:] @ pe.t()) * m.scaling, -1)
        want[i] = torch.einsum("hr,hvr->hv", p @ c, up[:, 64:])
    # keys and values (or latent queries and sums) are rounded to bf16 once, 2^-9 of each at most; so is the result
    err = (got.view(T, 4, 96).double() - want).norm() / want.norm()
    assert err < 6e-3, float(err)


def _one_rounding(got, x, w):
    """`got` against `x [T, H, K] . w [H, K, N]`: one rounding to bf16 (eight significant bits: 2^-8 of the value), and fp32 sums of at most 64
    steps of the tensor core, 2^-22 each of what has been added up.  Two partial sums rounded to bf16 do not pass at K = 512."""
    want = torch.einsum("thk,hkn->thn", x.double(), w.double())
    size = torch.einsum("thk,hkn->thn", x.double().abs(), w.double().abs())
    return ((got.double() - want).abs() <= want.abs() * 2 ** -8 * (1 + 2 ** -8) + size * 2 ** -16 + 1e-30).all()


# the kernels' rule on a B200: CTAs of 16 tokens (four warps, K up to 128: up to 1036 of them; eight: 518), tiles of 32 x 64 with a ring of three
# stages (K up to 192) and of five, tiles of 128 x 128
@pytest.mark.parametrize("T,H,K,N", [(1, 1, 8, 8), (7, 16, 128, 512), (16, 16, 512, 128), (17, 3, 40, 136), (65, 16, 520, 72), (33, 16, 128, 512),
                                     (64, 128, 512, 128), (65, 128, 512, 128), (129, 16, 200, 520), (40, 128, 192, 136), (260, 16, 128, 512),
                                     (1000, 16, 512, 128), (131, 128, 72, 24)])
def test_head_product(T, H, K, N):
    torch.manual_seed(T + K)
    bf = torch.bfloat16
    wide = torch.randn(T, H, K + 24, device="cuda", dtype=bf)
    rows = torch.randn(H, N + 8, K, device="cuda", dtype=bf) * K ** -0.5
    x, w = wide[..., 8:8 + K], rows[:, 8:].transpose(1, 2)           # strides of a wider projection, rows of a taller one
    from sglang_jax_b200.ops import native
    assert native.head_product_supported(x, w)
    got = ops.head_product(x, w)
    assert got.shape == (T, H, N) and got.is_contiguous() and _one_rounding(got, x, w)
    assert _one_rounding(ops.head_product(wide[..., 7:7 + K], w), wide[..., 7:7 + K], w)      # not aligned: the general statement
    assert ops.head_product(x[:0], w).shape == (0, H, N)


@pytest.mark.parametrize("T", [1, 7, 96])
@pytest.mark.parametrize("heads", [16, 128])
def test_absorbed_products_sum_in_fp32(T, heads, monkeypatch):
    """The products before and behind latent decode keep fp32 sums whatever the process lets a library do."""
    from sglang_jax_b200.models.deepseek_v3 import MLAAttention
    cfg = SimpleNamespace(hidden_size=64, num_attention_heads=heads, qk_nope_head_dim=128, qk_rope_head_dim=64, v_head_dim=128,
                          kv_lora_rank=512, q_lora_rank=None, rms_norm_eps=1e-6, max_position_embeddings=1024)
    torch.manual_seed(T)
    with torch.device("cuda"):
        m = MLAAttention(cfg, 0, torch.bfloat16)
    m.kv_b_proj.weight.data.normal_(0, 512 ** -0.5)
    m.absorb()
    q = torch.randn(T, heads, 192, device="cuda", dtype=torch.bfloat16)
    o_lat = torch.randn(T, heads, 512, device="cuda", dtype=torch.bfloat16)
    monkeypatch.setattr(torch.backends.cuda.matmul, "allow_bf16_reduced_precision_reduction", True)

    def library(*a, **k):
        raise AssertionError("a library product, whose partial sums that flag lets into bf16")

    monkeypatch.setattr(torch, "bmm", library)
    up = m.kv_b_proj.weight.view(heads, 256, 512)
    assert _one_rounding(m._latent_query(q), q[..., :128], up[:, :128])
    assert _one_rounding(m._value_up(o_lat), o_lat, up[:, 128:].transpose(1, 2))


@pytest.mark.parametrize("group", [1, 3])
def test_mla_extend_in_groups_of_heads(group, monkeypatch):
    """Where the expanded keys and values of all heads are too much at a time, the heads go in groups (the last one shorter): each is
    computed by itself, so the bits are the same."""
    from sglang_jax_b200.models.deepseek_v3 import MLAAttention
    torch.manual_seed(group)
    bf, page, n, pre = torch.bfloat16, 16, [40, 5, 300], [70, 20, 0]
    cfg = SimpleNamespace(hidden_size=256, num_attention_heads=4, qk_nope_head_dim=64, qk_rope_head_dim=32, v_head_dim=96,
                          kv_lora_rank=128, q_lora_rank=None, rms_norm_eps=1e-6, max_position_embeddings=1024)
    with torch.device("cuda"):
        m = MLAAttention(cfg, 0, bf)
    for p in m.parameters():
        p.data.normal_(0, 0.06)
    m.absorb()
    t = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    total = [a + b for a, b in zip(n, pre)]
    table = (torch.randperm(3 * 20, device="cuda") + 1).int().view(3, 20)
    cache = torch.randn(61, page, 160, device="cuda", dtype=bf)
    q = torch.randn(sum(n), 4, 96, device="cuda", dtype=bf)
    pos = t([i for a, b in zip(pre, n) for i in range(a, a + b)])

    def run():
        fb = SimpleNamespace(positions=pos, page_table=table, req_pool_indices=t([0, 1, 2]), seq_lens=t(total), page_size=page,
                             extend_seq_lens_cpu=np.asarray(n), extend_prefix_lens_cpu=np.asarray(pre), extend_seq_lens=t(n),
                             extend_prefix_lens=t(pre), cu_q_lens=t([0, 40, 45, 345]), num_tokens=sum(n), max_seq_len=max(total), extras={})
        return m._extend(q, cache, fb)

    want, groups = run(), []
    long = sum(a for a, b in zip(total, n) if b >= 32)     # tokens of which keys and values are expanded
    monkeypatch.setattr(m, "EXPAND_BYTES", group * long * (64 + 96) * 2)
    extend = ops.latent_extend
    monkeypatch.setattr(ops, "latent_extend", lambda q, *a: groups.append(q.shape[1]) or extend(q, *a))
    assert torch.equal(run(), want) and groups == ([1] * 4 if group == 1 else [3, 1])
