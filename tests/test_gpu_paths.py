"""Launch rules of the tensor-core path at their edges: both forms of the per-head prologue, the shares of the
key/value side, sequences whose chunks meet no state."""

import pytest
import torch

from oal_b200 import _lib, synthetic
from oal_b200.hd_block_gemm import make_problem
from tests.helpers import assert_close, oracle_dense, run_operator

pytestmark = pytest.mark.gpu

TOL_BF16 = 2e-2      # the tolerance of bf16 inputs and outputs with fp32 accumulation


def _case(b, n, hq, hkv, g):
    """Per-head partitions into g groups, no outlier channels (with one or two groups they would share one)."""
    gen = torch.Generator().manual_seed(100 * g + n)
    case = synthetic.mixed_case(n, batch=b, hq=hq, hkv=hkv, n=n, d=64, dv=64, gmax=g, aux_grads=False)
    case.dim_groups = torch.stack([torch.randperm(64, generator=gen) % g for _ in range(hq)]).to(torch.int32)
    case.factor = torch.rand(hq, (g + 1) * (g + 2) // 2, generator=gen) * 0.9 + 0.1
    case.q, case.k, case.v, case.grad_out = (t.bfloat16().float() for t in (case.q, case.k, case.v, case.grad_out))
    return case


# one chunk (prologue alone), two and three chunks (prologue in two launches, or one with the side streams off);
# register extents of the rotations: 9 columns up to 8 groups, 17 above; one, several and all heads per key/value CTA
@pytest.mark.parametrize("b,n,hq,hkv", [(1, 128, 3, 1), (1, 129, 14, 2), (2, 300, 4, 4), (40, 129, 4, 1)])
@pytest.mark.parametrize("g", [1, 8, 9, 16])
def test_prologue_forms_agree_and_match_the_dense_statement(b, n, hq, hkv, g):
    case = _case(b, n, hq, hkv, g)
    beside = run_operator(case, precision="bf16_tensorcore", io_dtype=torch.bfloat16)
    _lib.load().oal_set_overlap(0)
    try:
        in_line = run_operator(case, precision="bf16_tensorcore", io_dtype=torch.bfloat16)
    finally:
        _lib.load().oal_set_overlap(1)
    for key in beside:
        assert torch.equal(beside[key], in_line[key]), key
    assert_close(beside, oracle_dense(case), TOL_BF16, label=f"{b, n, hq, hkv, g}")


def test_token_major_output_stays_limited_to_eight_groups():
    for groups, legal in ((8, True), (9, False)):
        p = make_problem((1, 2, 1, 64, 64, 64), groups=groups, io_dtype=torch.bfloat16, out_dtype=torch.bfloat16,
                         precision="bf16_tensorcore", chunk=128, scale=1.0, floor=1e-38, flags=_lib.FLAG_OUT_TOKEN_MAJOR)
        if legal:
            assert _lib.workspace_bytes(p, 1) > 0
        else:
            with pytest.raises(ValueError, match="at most 8 groups"):
                _lib.workspace_bytes(p, 1)
