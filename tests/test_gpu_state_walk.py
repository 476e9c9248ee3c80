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
    case = synthetic.qwen_head_case(11, batch=batch, n=n, hq=hq, hkv=hkv, g=8, bf16=True)
    ref = oracle_dense(case)
    # 2e-2: the bar of the bf16 mode (operands of 8 bits, differences of sums)
    assert_close(run_operator(case, precision="bf16_tensorcore", io_dtype=torch.bfloat16), ref, 2e-2, label=f"{batch}x{hkv}x{n}")


@pytest.mark.gpu
@pytest.mark.parametrize("batch,n", [(1, 200), (1, 1700), (3, 513)])
def test_forward_without_backward(batch, n):
    """A call without gradients writes less for a backward to read; its results are the same bits."""
    from oal_b200 import prepare_grouped_hd_block_gemm, run_prepared_grouped_hd_block_gemm

    case = synthetic.qwen_head_case(12, batch=batch, n=n, hq=2, hkv=1, g=8, bf16=True)
    q, k, v = (t.cuda().bfloat16() for t in (case.q, case.k, case.v))
    factor, groups = case.factor.cuda(), case.dim_groups.cuda()
    results = []
    for grad in (False, True):
        args = [t.detach().clone().requires_grad_(grad) for t in (q, k, v, factor)]
        prepared = prepare_grouped_hd_block_gemm(*args[:3], groups, args[3], precision="bf16_tensorcore")
        results.append(run_prepared_grouped_hd_block_gemm(prepared, *args))
    for a, b in zip(*results):
        assert torch.equal(a, b.detach())
