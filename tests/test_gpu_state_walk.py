"""Carry images of the forward: the walk with the state on chip and the two steps through memory, on both sides of the rule
that picks one (units = batch x KV heads, chunks of 128 tokens), against the fp64 oracle."""

import ctypes

import pytest
import torch

from oal_b200 import _lib, synthetic
from oal_b200.hd_block_gemm import make_problem
from oal_b200.hd_block_gemm_autograd import build_group_tables
from tests.helpers import assert_close, oracle_dense, run_operator, saved_state_parts


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


# (units, chunks, whether the walk is the faster route): one and two units soon leave most SMs idle
@pytest.mark.gpu
@pytest.mark.parametrize("units,chunks,walk", [(1, 4, True), (1, 20, False), (2, 6, True), (2, 20, False), (3, 16, True), (8, 20, True)])
def test_route_of_the_carry_images(units, chunks, walk):
    from oal_b200 import prepare_grouped_hd_block_gemm, run_prepared_grouped_hd_block_gemm

    case = synthetic.qwen_head_case(13, batch=1, n=128 * chunks, hq=units, hkv=units, g=8, bf16=True, with_grad=False)
    q, k, v = (t.cuda().bfloat16() for t in (case.q, case.k, case.v))
    factor = case.factor.cuda()
    prepared = prepare_grouped_hd_block_gemm(q, k, v, case.dim_groups.cuda(), factor, precision="bf16_tensorcore")
    _lib.profile_enable(True)
    try:
        _lib.profile_report()
        run_prepared_grouped_hd_block_gemm(prepared, q, k, v, factor)
        kernels = _lib.profile_report()
    finally:
        _lib.profile_enable(False)
    assert ("state_walk" in kernels) == walk and ("state_scan" in kernels) != walk


@pytest.mark.gpu
@pytest.mark.parametrize("batch,hq,hkv,n", [(1, 2, 1, 300), (1, 4, 2, 641), (3, 2, 1, 1024)])
def test_both_routes_leave_the_same_bits(batch, hq, hkv, n):
    """The walk, and the increments of oal_forward_local_state scanned by the forward that reuses them: the same sums in the
    same order."""
    lib, dev = _lib.load(), torch.device("cuda")
    case = synthetic.qwen_head_case(14, batch=batch, n=n, hq=hq, hkv=hkv, g=8, bf16=True)
    q, k, v = (t.to(dev, torch.bfloat16) for t in (case.q, case.k, case.v))
    gen = torch.Generator().manual_seed(5)
    a, b, c = (t.to(dev) for t in (torch.rand(hq, generator=gen) + 1, torch.rand(hq, 8, generator=gen) * 0.1, torch.eye(8).expand(hq, 8, 8).contiguous()))
    tables = build_group_tables(case.dim_groups.to(dev).unsqueeze(0).expand(hq, -1), 8)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    results = []
    for reuse in (False, True):
        problem = make_problem((batch, hq, hkv, n, 64, 64), groups=8, io_dtype=torch.bfloat16, out_dtype=torch.bfloat16,
                               precision="bf16_tensorcore", chunk=128, scale=case.scale, floor=1e-38,
                               grad_mask=_lib.GRAD_REUSE_STATE_STAGE if reuse else 0)
        num = torch.empty(batch, hq, n, 64, device=dev)
        out, den = torch.empty_like(num, dtype=torch.bfloat16), torch.empty(batch, hq, n, device=dev)
        saved = torch.full((_lib.workspace_bytes(problem, 2),), 0x5A if reuse else 0xA5, dtype=torch.uint8, device=dev)
        ws = torch.empty(_lib.workspace_bytes(problem, 0), dtype=torch.uint8, device=dev)
        status = torch.zeros(1, dtype=torch.int32, device=dev)
        if reuse:
            total = torch.empty(batch * hkv, _lib.STATE_ROWS, _lib.E_PAD, device=dev)
            _lib.check(lib.oal_forward_local_state(ctypes.byref(problem), _lib.ptr(k), _lib.ptr(v), _lib.ptr(total), _lib.ptr(ws),
                                                   ws.numel(), _lib.ptr(status), stream))
        _lib.check(lib.oal_forward(ctypes.byref(problem), *(_lib.ptr(t) for t in (q, k, v, tables.dim_perm, tables.group_start, a, b, c,
                                                                                out, num, den, saved)), None, _lib.ptr(ws), ws.numel(),
                                   _lib.ptr(status), stream))
        torch.cuda.synchronize()
        assert int(status) == 0
        parts = saved_state_parts(saved.cpu(), batch=batch, q_heads=hq, kv_heads=hkv, n=n, groups=8)
        results.append(dict(parts, out=out, num=num, den=den))
    for name, want in results[0].items():
        assert torch.equal(results[1][name], want), name
