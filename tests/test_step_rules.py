"""Which calls take which kernel, and what a layer keeps: the rules on the host, without a GPU."""

import pytest
import torch

from sglang_jax_b200 import ops
from sglang_jax_b200.ops import moe_native

BF = torch.bfloat16


@pytest.mark.parametrize("rows,weight,bias,ok", [
    ((4, 64), (8, 64), None, True), ((4, 64), (8, 64), (8,), True), ((0, 64), (8, 64), None, True),
    # a kernel would read past a narrower weight or a shorter bias, and skip what is wider
    ((4, 64), (8, 32), None, False), ((4, 64), (8, 96), None, False), ((4, 64), (8, 64), (7,), False), ((4, 64), (8, 64), (1,), False),
    ((4, 64), (64,), None, False), ((4, 0), (8, 0), None, False), ((4, 64), (0, 64), None, False), ((4, 40), (8, 40), None, False)])
def test_router_logits_takes_operands_that_fit(rows, weight, bias, ok):
    zeros = lambda s: None if s is None else torch.zeros(s, dtype=BF)
    assert moe_native.router_logits_supported(zeros(rows), zeros(weight), zeros(bias)) == ok


def test_router_logits_refuses_what_a_product_refuses():
    with pytest.raises(RuntimeError):
        ops.router_logits(torch.zeros(4, 64, dtype=BF), torch.zeros(8, 32, dtype=BF))


# ---- weights of several projections in one allocation
def _delta_net(width=64):
    from types import SimpleNamespace
    from sglang_jax_b200.layers.linear_attention import GatedDeltaNet
    m = GatedDeltaNet(SimpleNamespace(hidden_size=width, rms_norm_eps=1e-6, linear_num_value_heads=8, linear_num_key_heads=4,
                                      linear_key_head_dim=16, linear_value_head_dim=16, linear_conv_kernel_dim=4), 0, BF)
    for p in m.parameters():
        p.data.normal_()
    return m


def _kept(*linears):
    """Bytes of the allocations that the layers' weights keep alive beyond their own."""
    return sum(w.untyped_storage().nbytes() - w.numel() * w.element_size() for w in (lin.weight for lin in linears))


def test_a_quantised_projection_releases_its_dense_weight():
    from sglang_jax_b200.utils.quantization import QuantizedWeight, quantize_tensor
    m = _delta_net()
    x = torch.randn(5, 64).to(BF)
    y, parts = m._joint(x)
    assert y.shape[1] == sum(p.shape[1] for p in parts) and torch.equal(parts[1], m.in_proj_ba(x)) and torch.equal(parts[0], m.in_proj_qkvz(x))
    before = m.in_proj_ba.weight.clone()
    q, s = quantize_tensor(m.in_proj_qkvz.weight.data, torch.int8, "per_channel")
    m.in_proj_qkvz.set_quantized(QuantizedWeight(q, s, None, None, BF))
    assert m.in_proj_qkvz.weight is None and _kept(m.in_proj_ba) == 0
    assert torch.equal(m.in_proj_ba.weight, before) and m._joint(x) is None and m.in_proj_ba(x).shape == (5, 16)


def test_a_projection_of_another_type_leaves_the_allocation():
    from sglang_jax_b200.configs.dtype_config import DtypeConfig, apply_dtype_config
    m = _delta_net()
    before = m.in_proj_qkvz.weight.clone()
    assert list(apply_dtype_config(m, DtypeConfig({"in_proj_ba": "float32"}, torch.bfloat16))) == ["in_proj_ba.weight"]
    assert _kept(m.in_proj_qkvz, m.in_proj_ba) == 0 and m.in_proj_ba.weight.dtype == torch.float32
    assert torch.equal(m.in_proj_qkvz.weight, before) and m._joint(torch.zeros(1, 64, dtype=BF)) is None


def test_a_layer_goes_when_its_last_reference_does():
    import gc
    import weakref
    gc.disable()
    try:
        m = _delta_net()
        watch = weakref.ref(m.in_proj_qkvz)
        del m
        assert watch() is None                   # no cycle through the shared allocation waits for a collection
    finally:
        gc.enable()


def test_copies_share_nothing_with_the_original():
    import copy
    m = _delta_net()
    c = copy.deepcopy(m)
    c.in_proj_qkvz.leave_joint()
    assert m._joint(torch.zeros(1, 64, dtype=BF)) is not None and torch.equal(c.in_proj_ba.weight, m.in_proj_ba.weight)


def test_projections_stay_together_where_nothing_changes():
    from sglang_jax_b200.configs.dtype_config import DtypeConfig, apply_dtype_config
    m = _delta_net()
    assert apply_dtype_config(m, DtypeConfig({}, torch.bfloat16)).keys().isdisjoint({"in_proj_qkvz.weight", "in_proj_ba.weight"})
    m.in_proj_ba.weight_loader(m.in_proj_ba.weight, torch.ones(16, 64))
    assert m._joint(torch.ones(1, 64, dtype=BF))[1][1].eq(64).all()


def test_a_watched_projection_is_called():
    """Hooks of a layer see its call: it is not passed by for a product over several layers."""
    from sglang_jax_b200.layers.linear_attention import KimiDeltaAttention
    m, x, seen = _delta_net(), torch.randn(3, 64).to(BF), []
    for add in ("register_forward_hook", "register_forward_pre_hook"):
        handle = getattr(m.in_proj_ba, add)(lambda *a: seen.append(add))
        assert m._joint(x) is None
        KimiDeltaAttention._up(m.in_proj_ba, x)
        assert seen.pop() == add and not seen
        handle.remove()
        assert m._joint(x) is not None


# ---- expert products under expert parallelism
@pytest.mark.parametrize("pairs,local,experts,tile", [
    (8192, 32, 256, 64), (8192, 256, 256, 64), (8192, 32, 32, 256),       # 32 rows an expert on one of eight ranks are 32 on a single one
    (16384, 16, 128, 160), (16384, 128, 128, 160),
    (64, 64, 512, 32), (64, 64, 64, 0),                                   # 8 rows for 64 experts: most of them idle
    (260, 8, 64, 32), (260, 8, 8, 64)])
def test_expert_tiles_follow_this_ranks_rows(pairs, local, experts, tile):
    assert moe_native.expert_tile(pairs, 2048, 768, local, experts) == tile
    assert moe_native.expert_tile(pairs, 2040, 768, local, experts) == moe_native.expert_tile(pairs, 2048, 760, local, experts) == 0
