"""Carry images of the forward: the walk with the state on chip and the two steps through memory, on both sides of the rule
that picks one (units = batch x KV heads, chunks of 128 tokens), against the fp64 oracle."""

import pytest
import torch

from oal_b200 import synthetic
from tests.helpers import assert_close, oracle_dense, run_operator


# (units: batch, query heads, KV heads; tokens): one, two and three chunks, odd counts, a partial last chunk; three units and a
# length at which one unit takes the two steps
@pytest.mark.gpu
@pytest.mark.parametrize("batch,hq,hkv,n", [(1, 2, 1, 129), (1, 2, 1, 384), (1, 2, 1, 1700), (3, 2, 1, 641), (3, 1, 1, 513)])
def test_carry_of_every_chunk(batch, hq, hkv, n):
    case = synthetic.qwen_head_case(11, batch=batch, n=n, hq=hq, hkv=hkv, g=4, bf16=True)
    ref = oracle_dense(case)
    # 2e-2: the bar of the bf16 mode (operands of 8 bits, differences of sums)
    assert_close(run_operator(case, precision="bf16_tensorcore", io_dtype=torch.bfloat16), ref, 2e-2, label=f"{batch}x{hkv}x{n}")
