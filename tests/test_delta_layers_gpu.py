"""Layers with a delta rule (Gated DeltaNet, KDA) on the GPU, prefill and decode, against the PyTorch statements of the same layer."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from sglang_jax_b200 import ops
from sglang_jax_b200.ops import native

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _layer(kind, heads, kv, dim, dtype, seed):
    from sglang_jax_b200.layers.linear_attention import GatedDeltaNet, KimiDeltaAttention
    cfg = SimpleNamespace(hidden_size=256, rms_norm_eps=1e-6, linear_num_value_heads=heads, linear_num_key_heads=kv, linear_key_head_dim=dim,
                          linear_value_head_dim=dim, linear_conv_kernel_dim=4,
                          linear_attn_config=dict(num_heads=heads, head_dim=dim, short_conv_kernel_size=4))
    torch.manual_seed(seed)
    with torch.device("cuda"):
        m = (KimiDeltaAttention if kind == "kda" else GatedDeltaNet)(cfg, 0, dtype)
        for name, p in m.named_parameters():
            p.data.copy_(torch.rand(p.shape) + 0.5 if "A_log" in name or "norm" in name else
                         torch.randn(p.shape) * (1.0 if "dt_bias" in name else 0.5 if "conv" in name else 256 ** -0.5))
            assert p.is_cuda
    return m


def _batch(new, cached, decode, pool, tracks):
    i32 = lambda v: torch.tensor(np.asarray(v, np.int32), device="cuda")
    new, cached = np.asarray(new), np.asarray(cached)
    return SimpleNamespace(forward_mode=SimpleNamespace(is_decode=lambda: decode), cu_q_lens=i32(np.concatenate([[0], np.cumsum(new)])),
                           extend_prefix_lens=i32(cached), extend_prefix_lens_cpu=cached, extend_seq_lens_cpu=new, batch_size=len(new),
                           req_pool_indices=i32(np.arange(len(new))[::-1].copy()), positions=i32(np.zeros(int(new.sum()))),
                           extras={"recurrent_pool": pool, "recurrent_tracks": tracks})


def _pool(m, B, conv_dtype, seed):
    torch.manual_seed(seed)
    heads, dim = (m.nh, m.hd) if hasattr(m, "nh") else (m.nv, m.dk)
    return SimpleNamespace(conv_state=torch.randn(1, B + 3, m.conv_dim, 3, device="cuda").to(conv_dtype),
                           recurrent_state=torch.randn(1, B + 3, heads, dim, dim, device="cuda") * 0.1)


def _both(m, x, new, cached, decode, conv_dtype, tol, tracks=None):
    """The layer as it runs and by its statements, from the same caches."""
    got = []
    for reference in (False, True):
        pool = _pool(m, len(new), conv_dtype, 3)
        ops.set_force_reference(reference)
        try:
            y = m(x, _batch(new, cached, decode, pool, tracks))
        finally:
            ops.set_force_reference(False)
        got.append((y, pool.conv_state, pool.recurrent_state))
    native.check_status()
    for a, b in zip(*got):
        assert (a.double() - b.double()).norm() <= tol * b.double().norm()


# the statements round queries, keys, values and read-outs to bf16 (2^-9 of each on average), some 0.006 in all; a column read from the wrong
# place is of the size of the result
def _tol(dtype):
    return 1.5e-2 if dtype == BF else 1e-4


CASES = [("gdn", 8, 4, 64, BF), ("gdn", 6, 2, 32, BF), ("kda", 8, 8, 64, BF), ("kda", 3, 3, 32, BF), ("gdn", 8, 8, 32, torch.float32),
         ("kda", 8, 8, 32, torch.float32)]


@pytest.mark.parametrize("kind,heads,kv,dim,dtype", CASES)
@pytest.mark.parametrize("weights", ["as loaded", "one moved", "one quantised"])
def test_layer_equals_its_statements(kind, heads, kv, dim, dtype, weights):
    from sglang_jax_b200.utils.quantization import QuantizedWeight, quantize_tensor
    m = _layer(kind, heads, kv, dim, dtype, heads + dim)
    together = heads % 8 == 0                              # all projections have rows of whole 16-byte units
    first = m._joint.linears[0]
    if weights == "one moved":
        first.weight.data = first.weight.data.clone()
    elif weights == "one quantised":
        q, s = quantize_tensor(first.weight.data, torch.int8, "per_channel")
        first.set_quantized(QuantizedWeight(q, s, None, None, dtype))
    assert (m._joint.weight() is not None) == (together and weights == "as loaded")
    conv_w = m._conv_weight() if kind == "kda" else m.conv1d_weight
    for new, cached, decode in (([40, 1, 0, 33, 70], [0, 9, 5, 64, 0], False), ([1] * 5, [40, 10, 5, 97, 70], True)):
        x = torch.randn(sum(new), 256, device="cuda").to(dtype)
        pool = _pool(m, 5, dtype, 3)
        assert ops.delta_supported(x, pool.conv_state[0], pool.recurrent_state[0], dim, dim, 4) and conv_w.dtype == dtype
        # checkpoints inside and at the end of a sequence, in slots of their own
        _both(m, x, new, cached, decode, dtype, _tol(dtype), None if decode else {0: (32, 6), 4: (70, 7)})


@pytest.mark.parametrize("kind", ["gdn", "kda"])
def test_decode_with_windows_in_fp32(kind, monkeypatch):
    """Windows kept in fp32 beside bf16 inputs: the in-place kernels of `csrc/linear_attn.cu`."""
    m = _layer(kind, 4, 4, 64, BF, 2)
    calls = []
    step = native.delta_rule_step
    monkeypatch.setattr(native, "delta_rule_step", lambda *a, **k: calls.append(1) or step(*a, **k))
    _both(m, torch.randn(5, 256, device="cuda").to(BF), [1] * 5, [40, 10, 5, 97, 70], True, torch.float32, _tol(BF))
    assert len(calls) == 1                                 # (the statements do not call it)
