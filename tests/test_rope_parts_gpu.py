"""Norm, rotation and cache write of queries, keys and values, and the fused gated product, on the GPU."""

import pytest
import torch

from sglang_jax_b200 import ops
from sglang_jax_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,Hq,Hkv,D", [(1, 16, 4, 128), (3, 1, 1, 64), (300, 5, 2, 128), (37, 3, 1, 256), (700, 64, 8, 128)])
@pytest.mark.parametrize("rd,neox", [(1.0, True), (0.5, True), (0.25, True), (1.0, False), (0.5, False), (0.0, True)])
@pytest.mark.parametrize("norm,gemma", [(False, False), (True, False), (True, True)])
def test_rope_parts(T, Hq, Hkv, D, rd, neox, norm, gemma):
    torch.manual_seed(T + D)
    dev, bf, P = "cuda", torch.bfloat16, 16
    rd = int(D * rd)
    qg = torch.randn(T, Hq, 2 * D, device=dev, dtype=bf)                      # a gate behind every query
    q, k, v = qg[..., :D], torch.randn(T, Hkv, D, device=dev, dtype=bf), torch.randn(T, Hkv, D, device=dev, dtype=bf)
    pos = torch.randint(0, 500, (T,), device=dev, dtype=torch.int32)
    cs = ref.build_cos_sin_cache(rd, 500, 1e4, device=dev) if rd else None
    qw, kw = ((torch.randn(D, device=dev, dtype=bf) * 0.2 + (0.0 if gemma else 1.0)) if norm else None for _ in range(2))
    loc = torch.randperm(T + 40, device=dev)[:T].int()
    cache = torch.zeros((T + 40) // P + 1, 2, Hkv, P, D, device=dev, dtype=bf)
    got_kv, want_kv, fused_kv = cache.clone(), cache.clone(), cache.clone()
    qkv = torch.cat([q.flatten(1), k.flatten(1), v.flatten(1)], -1)
    want = ref.rope_qknorm_kvwrite(qkv, pos, cs, qw, kw, 1e-6, Hq, Hkv, D, want_kv, loc, P, neox, rd or None, gemma)
    args = (pos, cs, qw, kw)
    assert ops.rope_parts_supported(q, k, v, *args, got_kv, loc, neox, rd or None)
    got = ops.rope_parts(q, k, v, *args, 1e-6, got_kv, loc, P, neox, rd or None, gemma)
    fused = ops.rope_qknorm_kvwrite(qkv, *args, 1e-6, Hq, Hkv, D, fused_kv, loc, P, neox, rd or None, gemma)
    assert torch.equal(fused, got) and torch.equal(fused_kv, got_kv)
    # the norm's rounding to bf16 may fall the other way (2^-8 of a value at most); a rotation adds two such values and rounds again
    for a, b in ((got, want), (got_kv, want_kv)):
        assert (a.float() - b.float()).abs().max() <= 2 ** -6 * max(b.float().abs().max().item(), 1.0)
        assert (a.float() - b.float()).norm() <= 2e-3 * b.float().norm()
    assert torch.equal(got_kv[:, 1], want_kv[:, 1])


@pytest.mark.parametrize("T,K,I", [(257, 64, 8), (300, 192, 136), (1000, 2048, 768)])
def test_linear_swiglu(T, K, I):
    torch.manual_seed(T)
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(2 * I, K, device="cuda", dtype=torch.bfloat16) * K ** -0.5
    assert ops.linear_swiglu_supported(x, w) and not ops.linear_swiglu_supported(x[:256], w)
    h = x.double() @ w.double().t()
    want = torch.nn.functional.silu(h[:, :I]) * h[:, I:]
    err = lambda y: ((y.double() - want).norm() / want.norm()).item()
    assert err(ops.linear_swiglu(x, w)) < 2 ** -8                             # one rounding to bf16
    assert err(ops.linear_swiglu(x, w)) <= err(ops.silu_and_mul(ops.linear(x, w)))


@pytest.mark.parametrize("form", ["heads", "odd rows", "odd table", "odd cache"])
def test_rows_as_callers_have_them(form):
    """Rows by heads, and tensors that begin off a 16-byte boundary: the same results as plain ones."""
    T, Hq, Hkv, D, P, dev, bf = 37, 3, 1, 64, 16, "cuda", torch.bfloat16
    torch.manual_seed(5)
    odd = lambda t: torch.empty(t.numel() + 1, device=dev, dtype=t.dtype)[1:].view_as(t).copy_(t)
    qkv, pos = torch.randn(T, (Hq + 2 * Hkv) * D, device=dev, dtype=bf), torch.randint(0, 90, (T,), device=dev, dtype=torch.int32)
    cs, loc = ref.build_cos_sin_cache(D, 90, 1e4, device=dev), torch.randperm(64, device=dev)[:T].int()
    w = torch.randn(2, D, device=dev, dtype=bf)
    cache = torch.zeros(4, 2, Hkv, P, D, device=dev, dtype=bf)
    run = lambda x, table, kv: ops.rope_qknorm_kvwrite(x, pos, table, w[0], w[1], 1e-6, Hq, Hkv, D, kv, loc, P)
    want = run(qkv, cs, cache)
    x = {"heads": qkv.view(T, -1, D), "odd rows": odd(qkv)}.get(form, qkv)
    other = odd(torch.zeros_like(cache)) if form == "odd cache" else torch.zeros_like(cache)
    got = run(x, odd(cs) if form == "odd table" else cs, other)
    if form in ("odd table", "odd cache"):               # the general statement: sums in another order, last places of bf16
        assert (got.float() - want.float()).norm() <= 2e-3 * want.float().norm()
        assert (other.float() - cache.float()).norm() <= 2e-3 * cache.float().norm()
    else:
        assert torch.equal(got, want) and torch.equal(other, cache)


# heads that fill a CTA's pass, several tokens to a CTA (some of its lanes idle, the last CTA with fewer tokens), passes of uneven shares; tokens
# from where on the CTAs are enough for several each (592 on a B200)
@pytest.mark.parametrize("Hq,Hkv,D", [(1, 1, 128), (8, 1, 64), (3, 1, 256), (14, 1, 128), (16, 4, 128), (16, 2, 256), (7, 5, 64), (30, 1, 64)])
@pytest.mark.parametrize("T", [1, 591, 1187, 2961])
def test_rope_spreads_heads_over_threads(Hq, Hkv, D, T):
    torch.manual_seed(T + Hq)
    dev, bf, P = "cuda", torch.bfloat16, 16
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, device=dev, dtype=bf)
    pos = torch.randint(0, 500, (T,), device=dev, dtype=torch.int32)
    cs = ref.build_cos_sin_cache(D // 2, 500, 1e4, device=dev)
    w = torch.randn(2, D, device=dev, dtype=bf) * 0.2 + 1.0
    loc = torch.randperm(T + 40, device=dev)[:T].int()
    loc[::7] = -1                                        # tokens whose keys and values go nowhere
    cache = torch.zeros((T + 40) // P + 1, 2, Hkv, P, D, device=dev, dtype=bf)
    got = ops.rope_qknorm_kvwrite(qkv, pos, cs, w[0], w[1], 1e-6, Hq, Hkv, D, cache, loc, P, True, D // 2)
    kept, want_kv = loc >= 0, torch.zeros_like(cache)
    want = ref.rope_qknorm_kvwrite(qkv, pos, cs, w[0], w[1], 1e-6, Hq, Hkv, D, None, loc, P, True, D // 2)
    ref.rope_qknorm_kvwrite(qkv[kept], pos[kept], cs, w[0], w[1], 1e-6, Hq, Hkv, D, want_kv, loc[kept], P, True, D // 2)
    # sums in another order: a norm's rounding to bf16 may fall the other way, and a rotation adds two such values and rounds again
    for a, b in ((got, want), (cache, want_kv)):
        assert (a.float() - b.float()).abs().max() <= 2 ** -6 * max(b.float().abs().max().item(), 1.0)
        assert (a.float() - b.float()).norm() <= 2e-3 * b.float().norm()
    assert torch.equal(cache[:, 1], want_kv[:, 1])
