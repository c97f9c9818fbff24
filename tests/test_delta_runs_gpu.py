"""Rows a warp takes in the delta rule's preparation: one at a time, eight or sixteen give the same bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


# heads, key heads, type; tokens of the sequences: together enough for runs of 8 (from 18944 rows x heads on) or 16 (75776), alone not
@pytest.mark.parametrize("H,K,dtype,lens", [(16, 8, torch.bfloat16, (500, 33, 1, 0, 7, 270, 8)),
                                            (16, 16, torch.float32, (590, 2, 9)), (16, 8, torch.bfloat16, (700, 701, 15, 780, 17, 760, 300))])
def test_sequences_together_and_alone(H, K, dtype, lens):
    from sglang_jax_b200.ops import native
    torch.manual_seed(sum(lens))
    D, taps, B, T = 128, 4, len(lens), sum(lens)
    channels = (2 * K + H) * D
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    proj = torch.randn(T, channels + 2 * H, device="cuda").to(dtype)
    conv_w = (torch.randn(channels, taps, device="cuda") * 0.5).to(dtype)
    a_log, dt = torch.rand(H, device="cuda"), torch.randn(H, device="cuda")
    conv0 = torch.randn(B + 1, channels, taps - 1, device="cuda").to(dtype)
    state0 = torch.randn(B + 1, H, D, D, device="cuda") * 0.1
    prefix = [5 * (i % 2) for i in range(B)]

    def run(rows, slots, ns, pre):
        conv, state = conv0.clone(), state0.clone()
        cu = [0]
        for n in ns:
            cu.append(cu[-1] + n)
        o = native.delta_scan(rows, -1, channels, channels + H, conv_w, a_log, dt, conv, state, slots, H, K, D, D, cu=i32(cu),
                              prefix=i32(pre))
        return o, conv, state

    o, conv, state = run(proj, torch.arange(1, B + 1, device="cuda"), lens, prefix)
    at = 0
    for i, n in enumerate(lens):
        if n:
            a, c, s = run(proj[at:at + n].contiguous(), torch.tensor([i + 1], device="cuda"), [n], [prefix[i]])
            assert torch.equal(a, o[at:at + n]) and torch.equal(c[i + 1], conv[i + 1]) and torch.equal(s[i + 1], state[i + 1])
        at += n
