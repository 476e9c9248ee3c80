"""What the launch code makes of live tensors before the kernels read them by address."""

import ctypes

import pytest
import torch

from oal_b200 import _lib
from oal_b200.hd_block_gemm import make_problem
from oal_b200.hd_block_gemm_autograd import _pad_last, on_boundary


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


def _off(t, elements=1):
    """The same values in a contiguous tensor that starts ``elements`` elements into its storage."""
    flat = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    view = flat[elements:elements + t.numel()].view(t.shape)
    view.copy_(t)
    return view


def test_operands_start_on_a_16_byte_boundary():
    t = torch.randn(1, 2, 3, 64).bfloat16()
    for elements in (1, 4, 7):
        live = _off(t, elements)
        assert live.is_contiguous() and live.data_ptr() % 16
        for got in (on_boundary(live), _pad_last(live)):
            assert got.data_ptr() % 16 == 0 and torch.equal(got, t)
    assert _pad_last(t) is t or _pad_last(t).data_ptr() == t.data_ptr()
    assert on_boundary(None) is None


@pytest.mark.parametrize("name,places", [          # positions in the C signature
    ("oal_forward", (1, 2, 3, 9, 10, 12, 13, 14)),
    ("oal_forward_packed", (1, 2, 3, 10, 11, 13, 14)),
    ("oal_backward", (1, 2, 3, 9, 11, 12, 13, 15, 16, 17, 21, 22)),
    ("oal_backward_packed", (1, 2, 3, 9, 11, 12, 13, 15, 16, 17, 19)),
    ("oal_forward_local_state", (1, 2, 3, 4)),
    ("oal_backward_local_state", (1, 7, 9, 10, 11, 13, 14)),
    ("oal_forward_static_scratch", (1, 2, 3, 9, 10, 12)),
    ("oal_rope_pack", range(8)),
    ("oal_rope_unpack_grad", range(8)),
])
def test_c_abi_refuses_tensors_off_a_16_byte_boundary(name, places):
    """Every tensor that the kernels touch in 16-byte pieces; refused before anything is launched."""
    function = getattr(_lib.load(), name)
    problem = make_problem((1, 2, 1, 128, 64, 64), groups=2, io_dtype=torch.bfloat16, out_dtype=torch.bfloat16,
                           precision="bf16_tensorcore", chunk=128, scale=1.0, floor=1e-38, grad_mask=15)
    scalars = {ctypes.c_int: 2, ctypes.c_float: 1e-6, ctypes.c_size_t: 1 << 40}
    for place in places:
        args = []
        for i, t in enumerate(function.argtypes):
            if t in scalars:
                args.append(scalars[t])
            elif i == 0 and not name.startswith("oal_rope"):
                args.append(ctypes.byref(problem))
            elif i == len(function.argtypes) - 1 or t == ctypes.POINTER(ctypes.c_int64):
                args.append(None)                                   # stream, ticket
            else:
                args.append(ctypes.cast(ctypes.c_void_p((1 << 20) + 2 * (i == place)), t))
        assert function(*args) == -1, place
        assert b"16-byte boundary" in _lib.load().oal_last_error_string(), place


@pytest.mark.gpu
def test_bf16_tensors_off_a_16_byte_boundary():
    import oal_b200

    gen = torch.Generator().manual_seed(3)
    q, k, v, dout = (torch.randn(1, h, 200, 64, generator=gen).to("cuda", torch.bfloat16) for h in (4, 2, 2, 4))
    dnum = torch.randn(q.shape, generator=gen).cuda()
    groups = (torch.arange(64) % 4).to(torch.int32).cuda()
    factor = (torch.rand(4, 15, generator=gen) * 0.9 + 0.1).cuda()
    coefs = [torch.ones(4), torch.ones(4, 4), torch.eye(4).expand(4, 4, 4).clone()]

    def run(place, explicit):
        leaves = [place(t).requires_grad_() for t in (q, k, v)]
        if explicit:
            out, num, _ = oal_b200.grouped_coefficient_attention(*leaves, groups, *(c.cuda().requires_grad_() for c in coefs),
                                                                 precision="bf16_tensorcore")
        else:
            prepared = oal_b200.prepare_grouped_hd_block_gemm(*leaves, groups, factor, precision="bf16_tensorcore")
            out, num, _ = oal_b200.run_prepared_grouped_hd_block_gemm(prepared, *leaves, factor)
        torch.autograd.backward([out, num], [place(dout), place(dnum)])
        free = oal_b200.oal_attention(*(place(t) for t in (q, k, v)), groups, factor)
        return [out.detach(), num.detach(), free, *(t.grad for t in leaves)]

    for explicit in (False, True):
        for got, want in zip(run(_off, explicit), run(lambda t: t.clone(), explicit)):
            assert torch.equal(got, want)


@pytest.mark.gpu
def test_layer_prologue_off_a_16_byte_boundary():
    from oal_b200.attention_shell import _RopePackFunction, rope_tables

    gen = torch.Generator().manual_seed(4)
    flats = [torch.randn(2, 33, h * 64, generator=gen).to("cuda", torch.bfloat16) for h in (4, 2, 2)]
    cos, sin = rope_tables(33, 64, device=torch.device("cuda"))

    def run(place):
        leaves = [place(t).requires_grad_() for t in flats]
        outs = _RopePackFunction.apply(*leaves, place(cos), place(sin), 4, 2)
        torch.autograd.backward(outs, [place(torch.ones_like(o)) for o in outs])
        return [*(o.detach() for o in outs), *(t.grad for t in leaves)]

    for got, want in zip(run(_off), run(lambda t: t.clone())):
        assert torch.equal(got, want)
