"""The bias of the two-call and the dense NVFP4 linear in the GEMM epilogue against a separate bf16 add, bit for bit."""
import pytest
import torch

from tests import helpers as H

pytestmark = pytest.mark.gpu


# a split launch, 128-wide tiles, CTA pairs with ragged rows; columns that do and do not allow 16-byte stores
@pytest.mark.parametrize("m", [3, 200, 700])
@pytest.mark.parametrize("n", [264, 300, 4608])
def test_dense_gemm_bias_equals_a_separate_add(m, n):
    from sharq_b200 import ops
    from sharq_b200.quantize import quantize_activation_nvfp4, quantize_weight_nvfp4

    k = 1152
    a, sfa, sx = quantize_activation_nvfp4(H.config0_x(m, k, m).cuda())
    b, sfb, sw = quantize_weight_nvfp4(H.config0_w(n, k, n).cuda())
    c, bias = H.config0_x(m, n, n).cuda(), H.config0_x(1, n, 3).cuda().reshape(n)
    scale = (sx * sw).reshape(1)
    got = ops.matmul_tensor_scale(a, b, sfa, sfb, scale, bias=bias)
    assert torch.equal(got, ops.matmul_tensor_scale(a, b, sfa, sfb, scale) + bias)
    got = ops.matmul_accum_tensor_scale(a, b, sfa, sfb, scale, c, 1.0, bias=bias)
    assert torch.equal(got, ops.matmul_accum_tensor_scale(a, b, sfa, sfb, scale, c, 1.0) + bias)
    ops.check_device_errors()
