"""Routing, permutation and products of an MoE layer on the GPU, at the edges of their tiles and splits."""

import numpy as np
import pytest
import torch

from sglang_jax_b200 import ops
from sglang_jax_b200.ops import moe_native

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def randn(*s, seed=0, std=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed + sum(s))
    return torch.empty(s, device="cuda", dtype=BF).normal_(0, std, generator=g)


@pytest.mark.parametrize("T,E,K", [(1, 1, 32), (7, 64, 2048), (16, 20, 96), (17, 256, 7168), (512, 128, 2048), (513, 24, 288),
                                   (2100, 130, 2048)])
def test_router_logits(T, E, K):
    x, w, bias = randn(T, K, seed=1), randn(E, K, seed=2, std=4 * K ** -0.5), randn(E, seed=3)
    want = x.double() @ w.double().t()
    got = ops.router_logits(x, w)
    assert got.dtype == torch.float32
    # 32 products at a time from zero, K / 32 rounded additions behind them: an ordinary fp32 sum
    scale = x.double().abs() @ w.double().abs().t()
    assert ((got - want).abs() <= 4e-7 * scale + 1e-30).all()
    torch.testing.assert_close(ops.router_logits(x, w, bias), got + bias.float(), rtol=1e-6, atol=1e-6)
    wide = randn(T, K + 8, seed=5)
    torch.testing.assert_close(ops.router_logits(wide[:, 8:], w), ops.router_logits(wide[:, 8:].contiguous(), w), rtol=0, atol=0)


@pytest.mark.parametrize("T,k,E,e0,local", [(1, 1, 1, 0, 1), (7, 8, 64, 0, 64), (512, 8, 128, 32, 96), (513, 8, 64, 0, 64),
                                            (4096, 8, 512, 0, 512), (3001, 3, 33, 5, 20), (600, 10, 16, 12, 4)])
@pytest.mark.parametrize("tile", [32, 128, 256])
def test_moe_align(T, k, E, e0, local, tile):
    rs = np.random.RandomState(T + E)
    ids = np.sort(rs.rand(T, E).argsort(1)[:, :k], 1).astype(np.int32) if k <= E else None
    ids[:, :1] = np.minimum(ids[:, :1], 1 + E // 4)                           # some experts hold more than others
    ws = moe_native.MoeWorkspace(T * k, local, "cuda")
    hist = torch.zeros(local, dtype=torch.int32, device="cuda")
    moe_native.moe_align(torch.from_numpy(ids).cuda(), e0, local, ws, hist, tile_rows=tile)
    flat = ids.ravel() - e0
    mine = (flat >= 0) & (flat < local)
    count = np.bincount(flat[mine], minlength=local)
    off = np.concatenate([[0], np.cumsum(count)])
    assert np.array_equal(ws.offsets.cpu().numpy(), off) and np.array_equal(hist.cpu().numpy(), count)
    row, token = ws.pair_row.cpu().numpy(), ws.row_token.cpu().numpy()
    assert (row[~mine] == -1).all() and np.array_equal(np.sort(row[mine]), np.arange(off[-1]))
    assert (row[mine] >= off[flat[mine]]).all() and (row[mine] < off[flat[mine] + 1]).all()
    assert np.array_equal(token[row[mine]], np.nonzero(mine)[0] // k)
    tiles = [(e, off[e] + r) for e in range(local) for r in range(0, count[e], tile)]
    n = ws.counts.cpu().numpy()
    assert n[0] == off[-1] and n[1] == len(tiles)
    got = list(zip(ws.tile_group.cpu().numpy()[:n[1]], ws.tile_row0.cpu().numpy()[:n[1]]))
    assert got == tiles


@pytest.mark.parametrize("T,k,H", [(1, 1, 8), (3, 7, 1032), (5, 8, 2048), (4, 16, 2056), (2, 9, 24)])
@pytest.mark.parametrize("shared", [False, True])
def test_moe_combine(T, k, H, shared):
    y, w = randn(T * k, H), torch.rand(T, k, device="cuda")
    ws = moe_native.MoeWorkspace(T * k, 1, "cuda")
    ws.pair_row.copy_(torch.randperm(T * k, device="cuda"))
    ws.pair_row[::5] = -1                                                     # pairs of other ranks
    add = randn(T, H, seed=9) if shared else None
    rows = ws.pair_row.view(T, k).long()
    want = ((w * (rows >= 0)).unsqueeze(-1).double() * y[rows.clamp_min(0)].double()).sum(1) + (add.double() if shared else 0.0)
    got = moe_native.moe_combine(y, w, ws, T, add=add)
    torch.testing.assert_close(got.double(), want, rtol=2 ** -8, atol=1e-5)   # one rounding to bf16


@pytest.mark.parametrize("T,k,E,H,I", [(1, 8, 64, 256, 128), (8, 8, 128, 128, 64), (4, 8, 64, 64, 192), (20, 8, 64, 256, 128), (300, 1, 3, 128, 64),
                                       (257, 8, 64, 256, 200), (1024, 8, 8, 192, 320), (33, 8, 64, 512, 128),
                                       (700, 2, 128, 64, 264)])
def test_fused_experts(T, k, E, H, I):
    """Products on pairs of SMs (whole blocks of 64 lanes) and the general ones against fp32 arithmetic."""
    torch.backends.cuda.matmul.allow_tf32 = False
    x, w13, w2 = randn(T, H), randn(E, 2 * I, H, std=H ** -0.5), randn(E, H, I, std=I ** -0.5)
    p = torch.softmax(randn(T, E, seed=4).float() * 2, -1)
    w, ids = p.topk(k, -1)
    ids = ids.int().contiguous()
    got = moe_native.fused_experts(x, w13, w2, w.contiguous(), ids)
    want = torch.zeros(T, H, device="cuda")
    for e in range(E):
        h = x.float() @ w13[e].float().t()
        y = (torch.nn.functional.silu(h[:, :I]) * h[:, I:]) @ w2[e].float().t()
        want += ((ids == e).float() * w).sum(-1, keepdim=True) * y
    # activations and expert outputs rounded to bf16 (gate and up too where I is no multiple of 64), 2^-9 each
    assert (got.float() - want).norm() / want.norm() < 6e-3
    from sglang_jax_b200.ops import native
    native.check_status()
