"""Kernels that read their inputs where a wider product or a checkpoint's row order leaves them, against the same kernels on
inputs laid out plainly: the arithmetic is the same, so the results are the same bits."""

import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device="cuda")


# value heads, key heads, key and value width, taps, type
DELTA = [(4, 2, 128, 128, 4, torch.bfloat16), (6, 3, 20, 12, 3, torch.bfloat16), (2, 2, 64, 32, 4, torch.float32),
         (8, 1, 48, 96, 2, torch.bfloat16)]


@pytest.mark.parametrize("H,K,D,V,taps,dtype", DELTA)
@pytest.mark.parametrize("lens", [None, (1, 33, 0, 70, 1)])
def test_grouped_columns_give_the_same_bits(H, K, D, V, taps, dtype, lens):
    from sglang_jax_b200.ops import native
    torch.manual_seed(H * 100 + D)
    r, B = H // K, 5
    T = B if lens is None else sum(lens)
    q, k = torch.randn(2, T, K, D).unbind(0)
    v, z = torch.randn(2, T, H, V).unbind(0)
    b, a = torch.randn(2, T, H).unbind(0)
    flat = lambda *t: torch.cat([x.reshape(T, -1) for x in t], -1).to(dtype).cuda()
    plain = flat(q, k, v, b, a)
    group = 2 * D + 2 * r * V
    rows = flat(torch.cat([q, k, v.reshape(T, K, r * V), z.reshape(T, K, r * V)], -1))
    ba = flat(torch.cat([b.reshape(T, K, r), a.reshape(T, K, r)], -1))
    wide = torch.cat([rows, ba], -1)                  # both at the same row stride, neither contiguous
    channels = 2 * K * D + H * V
    conv_w = (torch.randn(channels, taps) * 0.5).to(dtype).cuda()
    a_log, dt = torch.rand(H).cuda(), torch.randn(H).cuda()
    conv0 = torch.randn(B + 1, channels, taps - 1).to(dtype).cuda()
    state0 = torch.randn(B + 1, H, D, V).cuda() * 0.1
    slots = torch.arange(1, B + 1).cuda()
    ragged = {}
    if lens is not None:
        cu = [0]
        for n in lens:
            cu.append(cu[-1] + n)
        ragged = dict(cu=_i32(cu), prefix=_i32([0, 7, 0, 5, 9]))
    got = []
    for proj, off, kw in ((plain, (channels, channels + H), {}), (wide[:, :rows.shape[1]], (0, r), dict(ba=wide[:, rows.shape[1]:],
                                                                                                   grouped=group))):
        conv, state = conv0.clone(), state0.clone()
        o = native.delta_scan(proj, -1, *off, conv_w, a_log, dt, conv, state, slots, H, K, D, V, **ragged, **kw)
        got.append((o, conv, state))
    assert all(torch.equal(x, y) for x, y in zip(*got))
    w = torch.randn(V).to(dtype).cuda()
    want = native.delta_gate(got[0][0], flat(z), w.float(), 1e-6)
    assert torch.equal(native.delta_gate(got[0][0], wide[:, 2 * D + r * V:], w, 1e-6, group=r, step=group), want)


@pytest.mark.parametrize("M,K,N,ld,off", [(1, 128, 2048, 6416, 6144), (300, 128, 256, 400, 16), (65, 72, 40, 200, 8),
                                          (130, 96, 64, 100, 4)])
def test_column_range_of_a_wider_product(M, K, N, ld, off):
    """bf16 operands, fp32 sums: what is left is the rounding of the result, at most 2^-8 of it, and the order of the sum."""
    from sglang_jax_b200.ops import native
    torch.manual_seed(M)
    x = torch.randn(M, ld).bfloat16().cuda()[:, off:off + K]
    w = torch.randn(N, K).bfloat16().cuda()
    want = x.double() @ w.double().t()
    assert ((native.linear_part(x, w).double() - want).abs() <= want.abs() * 2 ** -8 + 1e-4 * K ** 0.5).all()
