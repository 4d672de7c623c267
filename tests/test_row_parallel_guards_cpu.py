"""Every condition under which RowParallelSharqLinear.forward runs its steps one by one, each as the only reason to do so: the layer has
nothing else that the one native call could not stand for.  Operators stubbed."""
import types

import pytest
import torch

from sharq_b200 import ops, qlinear, tp
from sharq_b200.qlinear import QLinearLayer
from sharq_b200.tp import RowParallelSharqLinear
from tests.test_row_parallel_forward import K, _layer

BIAS = torch.full((K,), 4.0, dtype=torch.bfloat16)


@pytest.fixture(autouse=True)
def operators(monkeypatch):
    def joint(*args, **kw):
        raise AssertionError("a step was passed by")

    def gemm(x, *args, bias=None, **kw):
        return 2 * x if bias is None else 2 * x + bias

    monkeypatch.setattr(ops, "sharq_linear_forward", joint)
    monkeypatch.setattr(ops, "scaled_sparse_residual_quantize_x", lambda x, n: (x, None, None, x, None, torch.ones(())))
    monkeypatch.setattr(ops, "sharq_linear_gemm", gemm)
    monkeypatch.setattr(ops, "sparse_matmul_tensor_scale", lambda x, *a, **kw: x)
    monkeypatch.setattr(ops, "matmul_accum_tensor_scale", lambda q, w, sf, sfw, scale, c, beta, **kw: q + beta * c)
    monkeypatch.setattr(qlinear, "quantize_activation_nvfp4", lambda x: (x, None, torch.ones(())))
    monkeypatch.setattr(ops, "matmul_tensor_scale", gemm)


def _run(layer):
    x = torch.ones(3, K, dtype=torch.bfloat16)
    return layer(x), x


def test_an_overridden_reduce():
    cls = type("Doubled", (RowParallelSharqLinear,), {"reduce": lambda self, y: 2 * y})
    y, x = _run(_layer(cls=cls))
    assert torch.equal(y, 4 * x)


def test_a_replaced_apply_prepared_reduced():
    layer = _layer()
    layer.apply_prepared_reduced = lambda prepared: 5 * prepared[1]
    y, x = _run(layer)
    assert torch.equal(y, 5 * x)


def test_a_reduce_hook():
    y, x = _run(_layer(hook=lambda v: 3 * v))
    assert torch.equal(y, 6 * x)


def test_more_than_one_rank(monkeypatch):
    monkeypatch.setattr(tp, "sum_buffer", lambda *a: None)
    monkeypatch.setattr(tp.dist, "all_reduce", lambda t, **kw: t.mul_(2))
    layer = _layer()
    layer.world = 2
    y, x = _run(layer)
    assert torch.equal(y, 4 * x)


def test_a_bias_behind_the_sum():
    y, x = _run(_layer(bias=BIAS))
    assert torch.equal(y, 2 * x + BIAS)


def test_a_bias_of_the_local_linear():
    layer = _layer()
    layer.local.bias = BIAS
    y, x = _run(layer)
    assert torch.equal(y, 2 * x + BIAS)


def test_two_gemms():
    y, x = _run(_layer(fused=False))
    assert torch.equal(y, 2 * x)


def test_a_dense_nvfp4_linear():
    layer = _layer()
    layer.local.quant_type, layer.local.scale_w = "NVFP4", None
    y, x = _run(layer)
    assert torch.equal(y, 2 * x)


@pytest.mark.parametrize("name", ["prepare_input", "apply_prepared"])
@pytest.mark.parametrize("how", ["subclass", "instance"])
def test_a_replaced_step_of_the_local_linear(name, how):
    def prepare_input(self, x, out_features_hint=None):
        return ("SHARQ", 3 * x, None, None, x, None, torch.ones(()))

    def apply_prepared(self, prepared, out=None, scatter=None, residual=None):
        return 6 * prepared[1]

    step = {"prepare_input": prepare_input, "apply_prepared": apply_prepared}[name]
    if how == "subclass":
        layer = _layer(type("Mine", (QLinearLayer,), {name: step}))
    else:
        layer = _layer()
        setattr(layer.local, name, types.MethodType(step, layer.local))
    y, x = _run(layer)
    assert torch.equal(y, 6 * x)
