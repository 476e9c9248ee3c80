"""Exact fp32 mode at the sizes where its launch rules change: CTAs per owner tile (clusters), group
capacities of the kernels, tile edges, unaligned tensors."""

import pytest
import torch

from oal_b200 import synthetic
from tests.helpers import assert_close, oracle_dense, run_operator

pytestmark = pytest.mark.gpu

# every output is a chain of three fp32 sums over at most N pairs, 64 dimensions and 16 groups with relative error
# 2^-24 per step; errors of independent roundings grow with the square root of the length, sqrt(600) * 2^-24 = 1.5e-6,
# and gradients cancel by a factor of a few in the normalised maximum
TOL = 1e-5


# (B, Hq, Hkv, N, G): a tile shared by 1, 2, 4 and 8 CTAs; more CTAs than tiles to walk (the first and last tiles);
# one query head per KV head and several; 4, 8 and 16 groups of capacity at their edges; N at both sides of a tile edge
@pytest.mark.parametrize("shape", [
    (1, 2, 1, 64, 4), (1, 3, 3, 128, 5), (1, 2, 2, 255, 8), (1, 4, 2, 257, 9), (1, 2, 1, 577, 3),
    (2, 14, 2, 513, 16), (5, 16, 4, 129, 2), (10, 16, 2, 100, 1),
])
def test_cluster_and_group_capacity_edges(shape):
    b, hq, hkv, n, g = shape
    gen = torch.Generator().manual_seed(n)
    case = synthetic.mixed_case(n, batch=b, hq=hq, hkv=hkv, n=n, d=64, dv=64, gmax=g)
    groups = torch.stack([torch.randperm(64, generator=gen) % g for _ in range(hq)]).to(torch.int32)
    case.dim_groups = groups
    case.factor = torch.rand(hq, (g + 1) * (g + 2) // 2, generator=gen) * 0.9 + 0.1
    assert_close(run_operator(case, precision="fp32_ieee"), oracle_dense(case), TOL, label=str(shape))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_tensors_off_a_four_element_boundary(dtype):
    import oal_b200

    gen = torch.Generator().manual_seed(3)
    groups = (torch.arange(64) % 4).to(torch.int32).cuda()
    factor = (torch.rand(2, 15, generator=gen) * 0.9 + 0.1).cuda()

    def run(offset):
        gen.manual_seed(4)
        leaves = []
        for heads in (2, 1, 1):
            flat = torch.zeros(heads * 70 * 64 + 8, device="cuda", dtype=dtype)
            t = flat[offset:offset + heads * 70 * 64].view(1, heads, 70, 64)
            t.copy_(torch.randn(t.shape, generator=gen))
            leaves.append(t.requires_grad_())
        out = oal_b200.oal_attention(*leaves, groups, factor, precision="fp32_ieee")
        return [out, *torch.autograd.grad(out, leaves, torch.ones_like(out))]

    for got, want in zip(run(1), run(0)):
        assert torch.equal(got, want)
