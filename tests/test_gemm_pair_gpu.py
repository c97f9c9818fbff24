"""Products of prefill sizes on pairs of SMs (csrc/gemm_pair.cu)."""

import pytest
import torch

from sglang_jax_b200.ops import native

pytestmark = pytest.mark.gpu


def operands(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    r = lambda *s: torch.empty(s, device="cuda", dtype=torch.bfloat16).normal_(0, 1, generator=g)
    return r(M, K), r(N, K)


def close(got, want, K):
    # fp32 sums in another order (a few 2^-24 of the terms' magnitude each), then one rounding to bf16, 2^-9 of the value
    torch.testing.assert_close(got.float(), want, rtol=2 ** -8, atol=2e-4 * K ** 0.5)


# one token; tiles that end inside, at and behind 32 tokens; N smaller than one CTA's rows, of one half, no multiple of a tile; one block
# of K, an odd number of blocks; more tiles than pairs; bands of token tiles with a shorter last one
@pytest.mark.parametrize("M,N,K", [(1, 8, 64), (31, 136, 128), (33, 256, 192), (257, 264, 320), (293, 4096, 1024), (700, 1000, 2048),
                                   (2500, 3072, 704), (2600, 520, 12288)])
@pytest.mark.parametrize("tile", [0, 32, 160, 256])
def test_pair(M, N, K, tile):
    torch.backends.cuda.matmul.allow_tf32 = False
    x, w = operands(M, N, K)
    bias = w[:, 0].contiguous()
    want = x.float() @ w.float().t()
    close(native.gemm_pair(x, w, tile=tile), want, K)
    close(native.gemm_pair(x, w, bias, tile=tile), want + bias.float(), K)
    wide = torch.full((M, K + 72), float("nan"), device="cuda", dtype=torch.bfloat16)
    wide[:, 8:K + 8] = x
    assert torch.equal(native.gemm_pair(wide[:, 8:K + 8], w, tile=tile), native.gemm_pair(x, w, tile=tile))
    if N % 16 == 0:
        g, u = want[:, :N // 2], want[:, N // 2:]
        got = native.gemm_pair(x, w, gated=True, tile=tile)
        # silu and the product pass on the sums' errors: each times the other factor
        act = torch.nn.functional.silu(g) * u
        slack = 2e-4 * K ** 0.5 * (u.abs() * 1.1 + torch.nn.functional.silu(g).abs() + 1.0)
        assert ((got.float() - act).abs() <= 2 ** -8 * act.abs() + slack).all()
    native.check_status()


@pytest.mark.parametrize("M,N,K", [(257, 256, 64), (300, 136, 4096), (1030, 2048, 200)])
def test_linear_takes_either_kernel(M, N, K):
    """The general kernel (any K) and the one on pairs give the same products."""
    x, w = operands(M, N, K)
    got, general = native.linear(x, w), native.linear(x, w, force_mode=0)
    close(got, x.float() @ w.float().t(), K)
    assert (got != general).float().mean() < 0.01
    native.check_status()


# a side of every line of the rule: short K, tiles that fill one wave of single SMs, few columns for many tokens
@pytest.mark.parametrize("M,N,K", [(257, 264, 64), (300, 136, 192), (1000, 4096, 192), (2048, 4096, 512), (300, 10240, 1536), (1025, 56, 256),
                                   (1024, 56, 2048), (1025, 64, 2048), (2500, 1000, 2048)])
def test_products_of_either_choice(M, N, K):
    x, w = operands(M, N, K)
    bias = w[:, 0].contiguous()
    want = x.float() @ w.float().t()
    close(native.linear(x, w), want, K)
    close(native.linear(x, w, bias), want + bias.float(), K)
    wide = torch.full((M, K + 72), float("nan"), device="cuda", dtype=torch.bfloat16)
    wide[:, 8:K + 8] = x
    assert torch.equal(native.linear_part(wide[:, 8:K + 8], w), native.linear(x, w))
    native.check_status()
