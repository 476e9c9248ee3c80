"""A preparation as a value: copies, pickles and changed copies run what their fields say."""

import copy
import dataclasses
import io
import pickle

import pytest
import torch

import oal_b200

pytestmark = pytest.mark.gpu


def _prepared(n=150, **options):
    gen = torch.Generator().manual_seed(7)
    q, k, v = (torch.randn(1, h, n, 64, generator=gen).bfloat16().cuda() for h in (4, 2, 2))
    groups = (torch.arange(64) % 4).to(torch.int32).cuda()
    factor = (torch.rand(4, 15, generator=gen) * 0.9 + 0.1).cuda()
    make = lambda **more: oal_b200.prepare_grouped_hd_block_gemm(q, k, v, groups, factor, precision="bf16_tensorcore", **options, **more)
    return make, (q, k, v, factor)


def test_copies_and_pickles_run_the_same_call():
    make, live = _prepared()
    prepared = make()
    want = oal_b200.run_prepared_grouped_hd_block_gemm(prepared, *live)
    for other in (copy.copy(prepared), copy.deepcopy(prepared), pickle.loads(pickle.dumps(prepared))):
        for got, x in zip(oal_b200.run_prepared_grouped_hd_block_gemm(other, *live), want):
            assert torch.equal(got, x)


@pytest.mark.parametrize("general", [False, True])
def test_a_plan_with_the_sizes_of_another_build_gets_room_enough(general):
    """Stored sizes only ever raise what a call allocates: a forward call cannot check the length of its saved state."""
    from oal_b200.hd_block_gemm_adapters import run_grouped_coefficients

    make, live = _prepared()
    q, k, v, factor = (t.clone().requires_grad_(True) for t in live)
    groups = (torch.arange(64) % 4).to(torch.int32).cuda()
    prepared = oal_b200.prepare_grouped_hd_block_gemm(q, k, v, groups, factor, precision="bf16_tensorcore")
    plan = dataclasses.replace(prepared.plan, forward_workspace_bytes=16, backward_workspace_bytes=16, saved_state_bytes=16)
    coefficients = [t.cuda().requires_grad_(True) for t in (torch.ones(4), torch.full((4, 4), 0.5), torch.eye(4).expand(4, 4, 4).clone())]
    results = []
    for each in (prepared, dataclasses.replace(prepared, plan=plan)):
        inputs = (q, k, v, *coefficients) if general else (q, k, v, factor)
        out = (run_grouped_coefficients(*inputs, tables=each.tables, plan=each.plan, scale=each.scale,
                                        normalization_floor=each.normalization_floor) if general
               else oal_b200.run_prepared_grouped_hd_block_gemm(each, *inputs))
        results.append([*out, *torch.autograd.grad(out[0].float().sum(), inputs)])
    for got, want in zip(results[1], results[0]):
        assert torch.equal(got, want)


def test_a_sequence_parallel_call_with_the_sizes_of_another_build_gets_room_enough():
    from oal_b200.sequence_parallel import sequence_parallel_attention

    make, live = _prepared()
    q, k, v, factor = (t.clone().requires_grad_(True) for t in live)
    groups = (torch.arange(64) % 4).to(torch.int32).cuda()
    prepared = make()
    plan = dataclasses.replace(prepared.plan, forward_workspace_bytes=16, backward_workspace_bytes=16, saved_state_bytes=16)
    results = []
    for each in (prepared, dataclasses.replace(prepared, plan=plan)):
        out = sequence_parallel_attention(q, k, v, groups, factor, prepared=each)
        results.append([*out, *torch.autograd.grad(out[0].float().sum(), (q, k, v, factor))])
    for got, want in zip(results[1], results[0]):
        assert torch.equal(got, want)


def test_a_changed_copy_runs_its_own_options():
    make, live = _prepared()
    prepared = make()
    for change in (dict(kernel_eps=0.5), dict(scale=0.3)):
        changed = dataclasses.replace(prepared, **change)
        for got, x in zip(oal_b200.run_prepared_grouped_hd_block_gemm(changed, *live),
                          oal_b200.run_prepared_grouped_hd_block_gemm(make(**change), *live)):
            assert torch.equal(got, x)
    assert not torch.equal(oal_b200.run_prepared_grouped_hd_block_gemm(changed, *live)[0],
                           oal_b200.run_prepared_grouped_hd_block_gemm(prepared, *live)[0])


def test_a_layer_is_copied_and_saved_after_its_first_call():
    from oal_b200 import attention_shell as shell

    geo = shell.ModelGeometry(num_query_heads=4, num_kv_heads=2, hidden_size=256, head_dim=64)
    groups = (torch.arange(64) % 4).to(torch.int32).expand(4, 64).clone()
    torch.manual_seed(1)
    layer = shell.OalAttentionLayer(0, groups, torch.full((4, 15), 0.5), cache=shell.PreparedCallCache(), geometry=geo,
                                    dtype=torch.bfloat16).cuda()
    x, rope = torch.randn(1, 130, 256, device="cuda").bfloat16(), shell.rope_tables(130, 64, device="cuda")
    want = layer(x, rope)
    file = io.BytesIO()
    torch.save(layer, file)
    file.seek(0)
    for other in (copy.deepcopy(layer), torch.load(file, weights_only=False)):
        assert torch.equal(other(x, rope), want)


def test_transforms_that_the_operator_does_not_support_raise():
    """Forward-mode tangents, vmap and functional gradients never come back as plain outputs."""
    import torch.autograd.forward_ad as fw

    make, (q, k, v, factor) = _prepared()
    prepared = make()
    with fw.dual_level():
        dual = fw.make_dual(factor, torch.ones_like(factor))
        with pytest.raises((RuntimeError, NotImplementedError)):
            oal_b200.run_prepared_grouped_hd_block_gemm(prepared, q, k, v, dual)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda x: oal_b200.run_prepared_grouped_hd_block_gemm(prepared, x, k, v, factor)[0])(q.expand(2, *q.shape))
    trained = oal_b200.prepare_grouped_hd_block_gemm(q, k, v, (torch.arange(64) % 4).to(torch.int32).cuda(),
                                                     factor.clone().requires_grad_(), precision="bf16_tensorcore")
    for call in (prepared, trained):      # refused as another gradient mode, and as a transform
        with pytest.raises((RuntimeError, ValueError)):
            torch.func.grad(lambda x: oal_b200.run_prepared_grouped_hd_block_gemm(call, q, k, v, x)[0].float().sum())(factor)
    assert torch.isfinite(oal_b200.run_prepared_grouped_hd_block_gemm(prepared, q, k, v, factor)[0]).all()
