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
