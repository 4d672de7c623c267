"""RowParallelSharqLinear.forward as one native call: taken only while every step that it stands for is the class's own (CPU, operators
stubbed), and the same bits as the steps for every form of input (GPU)."""
import types

import pytest
import torch

from sharq_b200 import ops
from sharq_b200.qlinear import QLinearLayer
from sharq_b200.tp import RowParallelSharqLinear
from tests import helpers as H

K, N = 128, 256


def _layer(local_cls=QLinearLayer, cls=RowParallelSharqLinear, bias=None, hook=None, fused=True):
    byte = torch.zeros(1, dtype=torch.uint8)
    layer = cls.__new__(cls)
    torch.nn.Module.__init__(layer)
    layer.world, layer.rank, layer.group, layer.reduce_hook, layer.bias = 1, 0, None, hook, bias
    layer.local = local_cls.from_quantized(K, N, byte, byte, byte, 1.0, fused_gemm=fused)
    return layer


class _Steps(QLinearLayer):
    def prepare_input(self, x, out_features_hint=None):
        return ("mine", x)

    def apply_prepared(self, prepared, out=None, scatter=None, residual=None):
        return 2 * prepared[1]


class _Doubled(RowParallelSharqLinear):
    def reduce(self, y):
        return 2 * y


@pytest.mark.parametrize("case", ["steps", "instance", "reduce", "hook", "bias", "not a linear"])
def test_replaced_steps_are_kept(monkeypatch, case):
    def joint(*args, **kw):
        raise AssertionError("a step was passed by")

    monkeypatch.setattr(ops, "sharq_linear_forward", joint)
    x = torch.ones(3, K, dtype=torch.bfloat16)
    bias = torch.full((K,), 4.0, dtype=torch.bfloat16)
    layer = _layer(QLinearLayer if case == "instance" else _Steps, _Doubled if case == "reduce" else RowParallelSharqLinear,
                   bias if case == "bias" else None, (lambda y: 3 * y) if case == "hook" else None)
    if case == "instance":
        layer.local.prepare_input, layer.local.apply_prepared = (lambda v: ("mine", v)), (lambda p, **kw: 2 * p[1])
    if case == "not a linear":
        del layer.local
        layer.local = types.SimpleNamespace(prepare_input=lambda v: ("mine", v), apply_prepared=lambda p: 2 * p[1])
    want = {"reduce": 4 * x, "hook": 6 * x, "bias": 2 * x + bias}.get(case, 2 * x)
    assert torch.equal(layer(x), want)


def test_untouched_is_one_call(monkeypatch):
    monkeypatch.setattr(ops, "sharq_linear_forward", lambda x, *a, **kw: 3 * x)
    x = torch.ones(2, 3, K, dtype=torch.bfloat16)
    assert torch.equal(_layer()(x), 3 * x)


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["plain", "three", "columns", "rows", "float", "one"])
def test_same_bits_as_the_steps(form):
    k, n = 1152, 264
    x = H.config0_x(37, 2 * k, 1).cuda()
    x = {"plain": x[:, :k].contiguous(), "three": x[:36, :k].reshape(4, 9, k), "columns": x[:, 1:k + 1], "rows": x[::2, :k],
         "float": x[:, :k].float(), "one": x[:1, :k]}[form]
    layer = RowParallelSharqLinear(H.config0_w(n, k, 2).cuda())
    want = layer.apply_prepared_reduced(layer.local.prepare_input(x.reshape(-1, k).to(torch.bfloat16)))
    got = layer(x)
    ops.check_device_errors()
    assert got.shape == (*x.shape[:-1], n) and torch.equal(got.reshape(-1, n), want)
