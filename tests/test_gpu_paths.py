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


# the first chunk of a sequence (nothing from the state kernels): full, partial and one-block tiles, rep 7 / 1 / 3
@pytest.mark.parametrize("n,hq,hkv,g", [(128, 14, 2, 8), (33, 2, 2, 1), (100, 3, 1, 16)])
def test_numerators_of_the_first_chunk_value_by_value(n, hq, hkv, g):
    case = _case(1, n, hq, hkv, g)
    num = run_operator(case, precision="bf16_tensorcore", io_dtype=torch.bfloat16, need=())["num"].double()
    q, k, v = (t[0].double() for t in (case.q, case.k, case.v))
    k, v = (t.repeat_interleave(hq // hkv, 0) for t in (k, v))
    rows, cols = torch.tril_indices(g + 1, g + 1)
    lower = torch.zeros(hq, g + 1, g + 1, dtype=torch.double)
    lower[:, rows, cols] = case.factor.double()
    per_dim = case.scale * lower[:, 1:].gather(1, case.dim_groups.long()[..., None].expand(-1, -1, g + 1))    # [hq, 64, r]
    u = lower[:, 0, None, None] + torch.einsum("hid,hdr,hjd->hijr", q, per_dim, k)
    w = ((u ** 2).sum(-1) + case.kernel_eps).tril()
    # Weights enter as bf16 value + remainder (2^-17 of w) and u_r = c_r + sum_d l_r[d] q_d k_d from products with one
    # factor rounded the same way: |du_r| <= 2^-17 a_r, a_r the sum of magnitudes, so dw <= 2^-16 |u| |a|; both norms over r
    # are those of any rotation of the terms, |a| <= |L_0| + sum_d |l[d]| |q_d k_d|.  Doubled for the fp32 roundings.
    a = lower[:, 0].norm(dim=-1)[:, None, None] + torch.einsum("hid,hd,hjd->hij", q.abs(), per_dim.norm(dim=-1), k.abs())
    bound = (2.0 ** -16 * w + 2.0 ** -15 * w.sqrt() * a).tril() @ v.abs()
    assert ((num[0] - w @ v).abs() <= bound).all()


@pytest.mark.parametrize("n,hq,hkv,g", [(128, 14, 2, 9), (100, 2, 2, 12), (128, 4, 1, 16)])
def test_key_value_gradients_above_eight_groups_are_as_exact_as_their_dtype(n, hq, hkv, g):
    """One chunk, every product as value + remainder (2^-16): what is left is the rounding of the results to bf16, at most
    2^-9 of each value and so of the 2-norm."""
    case = _case(2, n, hq, hkv, g)
    res, ref = run_operator(case, precision="bf16_tensorcore", io_dtype=torch.bfloat16), oracle_dense(case)
    for key in ("dq", "dk", "dv"):
        assert (res[key].double() - ref[key]).norm() <= 1.01 * 2.0 ** -9 * ref[key].norm(), key
