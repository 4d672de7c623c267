"""SwiGLU in the epilogue of the gate_up GEMM against the GEMM followed by the SwiGLU kernel.

Both forms accumulate every element over K in the same order and round at the same places (gate, up, silu, product),
so all bits are compared exactly.
"""
import pytest
import torch

from tests import helpers as H

pytestmark = pytest.mark.gpu


def _weights(n, k, seed):
    from sharq_b200.quantize import quantize_weight_shared_nvfp4

    return quantize_weight_shared_nvfp4(H.config0_w(n, k, seed).cuda())


def _amax_bits(h):
    return h.float().abs().max().reshape(1).view(torch.int32)


@pytest.mark.parametrize("m", [1, 127, 129, 256, 300, 777])
@pytest.mark.parametrize("f,k", [(128, 128), (384, 640), (1152, 1024)])
def test_gemm_swiglu_equals_gemm_then_swiglu(m, f, k):
    from sharq_b200 import ops

    x = H.config0_x(m, k, m).cuda()
    qw, sfs, sfd, scale = _weights(2 * f, k, f)
    a = ops.scaled_sparse_residual_quantize_x(x, 2 * f)
    ops.set_gemm_tile_n(512)  # same accumulation order
    try:
        gate_up = ops.sharq_linear_gemm(*a[:5], qw, sfs, sfd, a[5].reshape(1), alpha_host=40.0 * float(scale))
    finally:
        ops.set_gemm_tile_n(0)
    want = ops.swiglu(gate_up)
    h, amax = ops.linear_gemm_swiglu(*a[:5], qw, sfs, sfd, a[5].reshape(1), alpha_host=40.0 * float(scale))
    ops.check_device_errors()
    assert torch.equal(h, want)
    assert torch.equal(amax.max().reshape(1), _amax_bits(want))
    if f % 128 == 0:
        p = ops.absmax_sparse_residual_quantize_x(h, 128, amax)
        q = ops.scaled_sparse_residual_quantize_x(want, 128)
        assert all(torch.equal(u, v) for u, v in zip(p, q))


def test_grouped_gemm_swiglu_equals_grouped_gemm_then_swiglu():
    from sharq_b200 import ops

    f, k, groups = 256, 384, 4
    unit_group = torch.tensor([0, 0, 2, -1, 3, -1], dtype=torch.int32, device="cuda")  # group 1 and two units have no rows
    x = H.config0_x(unit_group.numel() * 256, k, 5).cuda()
    weights = [_weights(2 * f, k, 10 + g)[:3] for g in range(groups)]
    p = ops.grouped_sparse_residual_quantize_x(x, unit_group, groups)
    alpha = (p[5] * torch.tensor([0.002, 0.003, 0.004, 0.5], device="cuda")).contiguous()
    want = ops.swiglu(ops.linear_gemm_grouped(*p[:5], weights, unit_group, alpha))
    h, amax = ops.linear_gemm_grouped_swiglu(*p[:5], weights, unit_group, alpha)
    ops.check_device_errors()
    rows = (unit_group >= 0).repeat_interleave(256)
    assert torch.equal(h[rows], want[rows])
    for g in range(groups):
        mine = (unit_group == g).repeat_interleave(256)
        assert int(amax[g]) == (int(_amax_bits(want[mine])) if bool(mine.any()) else 0)


def test_swiglu_of_every_bf16_gate():
    """All 65536 bf16 gates (NaN, infinities, subnormals among them) against ATen's silu and product."""
    from sharq_b200 import ops

    gate = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).cuda().view(512, 128)
    up = torch.full_like(gate, 1.5)
    got = ops.swiglu(torch.cat((gate, up), dim=1))
    want = torch.nn.functional.silu(gate) * up
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.nan_to_num(0.25), want.nan_to_num(0.25))
