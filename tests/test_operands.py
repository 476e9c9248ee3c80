"""What the launch code makes of live tensors before the kernels read them by address."""

import pytest
import torch

from oal_b200.hd_block_gemm_autograd import _pad_last


@pytest.mark.parametrize("d", [5, 48, 64])
def test_operands_are_row_major_whatever_the_strides_of_the_live_tensor(d):
    t = torch.randn(2, 7, 3, d)
    for live in (t, t.transpose(1, 2), t[:, ::2], t[:1].expand(4, 7, 3, d), t.permute(3, 1, 2, 0).contiguous().permute(3, 1, 2, 0)):
        got = _pad_last(live)
        assert got.is_contiguous() and got.shape == (*live.shape[:3], 64)
        assert torch.equal(got[..., :d], live) and not got[..., d:].any()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_prepared_call_on_live_tensors_of_other_strides(dtype):
    import oal_b200

    gen = torch.Generator().manual_seed(1)
    base = [torch.randn(2, h, 150, 64, generator=gen).to("cuda", dtype) for h in (4, 2, 2)]
    groups = (torch.arange(64) % 4).to(torch.int32).cuda()
    factor = (torch.rand(4, 15, generator=gen) * 0.9 + 0.1).cuda()
    precision = "bf16_tensorcore" if dtype == torch.bfloat16 else "fp32_ieee"

    def run(tensors, train):
        leaves = [t.detach().requires_grad_(train) for t in tensors] + [factor.clone().requires_grad_(train)]
        rows = [t.detach().contiguous().requires_grad_(train) for t in tensors]
        prepared = oal_b200.prepare_grouped_hd_block_gemm(*rows, groups, leaves[3], precision=precision)
        out = oal_b200.run_prepared_grouped_hd_block_gemm(prepared, *leaves)
        if train:
            out[0].backward(torch.ones_like(out[0]))
        return [o.detach() for o in out] + [t.grad for t in leaves if train]

    other = [t.transpose(1, 2).contiguous().transpose(1, 2) for t in base]
    for train in (False, True):
        # explicit coefficients where the row-major call takes the packed factor: equal up to fp32 rounding of the
        # coefficients, which a bf16 output may round apart by one unit
        for got, want in zip(run(other, train), run(base, train)):
            assert (got.float() - want.float()).norm() <= 4e-3 * want.float().norm()
