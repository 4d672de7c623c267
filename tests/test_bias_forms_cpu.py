"""The forms of bias that the two-call and the dense NVFP4 linear take: the GEMM epilogue gets those it can read, torch's add
the rest.  Runs on the CPU with the GEMMs stubbed."""
import pytest
import torch

from sharq_b200 import ops
from sharq_b200.qlinear import QLinearLayer

N, K, M = 256, 128, 3
ONE = torch.ones(())


@pytest.fixture(autouse=True)
def gemms(monkeypatch):
    """Every GEMM gives ones, plus the bias as the binding would take it."""
    def gemm(bias=None):
        if bias is not None and not (bias.dtype == torch.bfloat16 and bias.is_contiguous() and bias.numel() == N):
            raise RuntimeError("bias must be a contiguous CUDA bfloat16 tensor with N elements")
        y = torch.ones(M, N, dtype=torch.bfloat16)
        return y if bias is None else y + bias.reshape(N)

    monkeypatch.setattr(ops, "matmul_tensor_scale", lambda *a, out=None, bias=None: gemm(bias))
    monkeypatch.setattr(ops, "matmul_accum_tensor_scale", lambda *a, bias=None: gemm(bias))
    monkeypatch.setattr(ops, "sparse_matmul_tensor_scale", lambda *a, **kw: gemm())


FORMS = {
    "plain": lambda b: b,
    "strided": lambda b: torch.stack((b, -b), dim=1)[:, 0],
    "expanded": lambda b: b[:1].expand(N),
    "one element": lambda b: b[:1],
    "row": lambda b: b.reshape(1, N),
    "column": lambda b: b[:M].reshape(M, 1),
    "float32": lambda b: b.float(),
    "float16": lambda b: b.half(),
}


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("tag,extra_fusion", [("NVFP4", True), ("SHARQ", True), ("SHARQ", False)])
def test_every_bias_that_torch_adds_is_added(form, tag, extra_fusion):
    byte = torch.zeros(1, dtype=torch.uint8)
    lin = QLinearLayer.from_quantized(K, N, byte, byte, byte, 1.0, extra_fusion=extra_fusion, fused_gemm=False)
    lin.scale_w = byte
    lin.bias = FORMS[form](torch.arange(N).to(torch.bfloat16))
    prepared = ("NVFP4", byte, byte, ONE) if tag == "NVFP4" else ("SHARQ", byte, byte, byte, torch.zeros(M, 1), byte, ONE)
    got = lin.apply_prepared(prepared)
    y = torch.ones(M, N, dtype=torch.bfloat16) * (1 if tag == "NVFP4" or extra_fusion else 2)
    want = y + lin.bias
    assert got.dtype == want.dtype and torch.equal(got, want)
