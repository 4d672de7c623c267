"""A bias of another GPU is refused before anything is launched.

The operands are fake tensors (a device and a shape, no memory), so the check is reached without a GPU; with one the
test is skipped, so that no kernel can be launched on their pointers.
"""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from sharq_b200 import _lib

M, N, K = 4, 256, 256


@pytest.mark.skipif(torch.cuda.is_available(), reason="fake operands have no memory")
@pytest.mark.parametrize("op", ["dense_gemm", "linear_gemm", "linear_forward"])
def test_bias_of_another_device_is_refused(op):
    native = _lib.native()

    def sf(rows):
        return (rows // 128 + 1) * 128 * K // 16

    with FakeTensorMode():
        def u8(*shape):
            return torch.empty(shape, dtype=torch.uint8, device="cuda:0")

        q, w, sfa, sfw = u8(M, K // 2), u8(N, K // 2), u8(sf(M)), u8(sf(N))
        flag = torch.empty(1, dtype=torch.int32, device="cuda:0")
        alpha = torch.empty(1, device="cuda:0")
        bias = torch.empty(N, dtype=torch.bfloat16, device="cuda:1")
        with pytest.raises(RuntimeError, match="bias must be on the same device"):
            if op == "dense_gemm":
                native.dense_gemm(q, w, sfa, sfw, 1.0, alpha, None, 0.0, bias, None, flag, True)
            elif op == "linear_gemm":
                native.linear_gemm(u8(M * K // 4), u8(128 * K // 16), sfa, q, sfa, w, sfw, sfw, alpha, 1.0, bias, None, None, flag,
                                   True)
            else:
                native.linear_forward(torch.empty(M, K, dtype=torch.bfloat16, device="cuda:0"), w, sfw, sfw, 1.0, bias, flag, True)
