"""The residual add in the epilogue of the fused GEMM and of the expert combine against a separate bf16 add, bit for bit."""
import pytest
import torch

from tests import helpers as H

pytestmark = pytest.mark.gpu


# a split launch, 128-wide tiles, CTA pairs with ragged rows; columns that do and do not allow 16-byte stores
@pytest.mark.parametrize("m", [3, 200, 700])
@pytest.mark.parametrize("n", [264, 300, 4096])
def test_gemm_residual_equals_a_separate_add(m, n):
    from sharq_b200 import ops
    from sharq_b200.quantize import quantize_weight_shared_nvfp4

    k = 1152
    x, r = H.config0_x(m, k, m).cuda(), H.config0_x(m, n, n).cuda()
    bias = H.config0_x(1, n, 3).cuda().reshape(n)
    qw, sfs, sfd, scale = quantize_weight_shared_nvfp4(H.config0_w(n, k, n).cuda())
    a = ops.scaled_sparse_residual_quantize_x(x, n)
    alpha = (a[5] * scale).reshape(1)
    plain = ops.sharq_linear_gemm(*a[:5], qw, sfs, sfd, alpha, bias=bias)
    fused = ops.sharq_linear_gemm(*a[:5], qw, sfs, sfd, alpha, bias=bias, residual=r)
    ops.check_device_errors()
    assert torch.equal(fused, r + plain)


def test_combine_residual_equals_a_separate_add():
    from sharq_b200 import ops
    from sharq_b200.decoder import moe_grouping

    tokens, width = 37, 264
    selected = torch.rand(tokens, 4, generator=torch.Generator().manual_seed(0)).topk(2, dim=1).indices.cuda()
    dest, src_row, _ = moe_grouping(selected, 4)
    y, r = H.config0_x(src_row.numel(), width, 1).cuda(), H.config0_x(tokens, width, 2).cuda()
    w = H.config0_x(tokens, 2, 3).cuda()
    assert torch.equal(ops.moe_combine(y, dest, selected, w, residual=r), r + ops.moe_combine(y, dest, selected, w))
