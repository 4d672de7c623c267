"""A call that does the work of several methods of a layer is not taken when one of them was replaced: by a subclass, on the
class itself (as a profiler's wrappers do) or on the instance.  Runs on the CPU with the operators stubbed."""
import types

import pytest
import torch

from sharq_b200 import decoder, ops
from sharq_b200.decoder import DecoderConfig, SharqDecoderLayer
from sharq_b200.qlinear import QLinearLayer
from sharq_b200.tp import RowParallelSharqLinear

F = 128


def _byte():
    return torch.zeros(1, dtype=torch.uint8)


def _linear(cls=QLinearLayer, n=2 * F, k=F):
    return cls.from_quantized(k, n, _byte(), _byte(), _byte(), 1.0)


def _unexpected(*args, **kw):
    raise AssertionError("the replaced method was passed by")


@pytest.fixture(autouse=True)
def fused_operators_refuse(monkeypatch):
    monkeypatch.setattr(ops, "sharq_linear_forward", _unexpected)
    monkeypatch.setattr(ops, "linear_gemm_swiglu_pays", lambda *a: True)
    monkeypatch.setattr(ops, "linear_gemm_swiglu", _unexpected)
    monkeypatch.setattr(ops, "sharq_linear_gemm", lambda *a, **kw: "gemm")


def _replace(monkeypatch, how, name, method):
    """A QLinearLayer whose method `name` is `method`."""
    if how == "subclass":
        return _linear(type("Sub", (QLinearLayer,), {name: method}))
    lin = _linear()
    if how == "class":
        monkeypatch.setattr(QLinearLayer, name, method)
    else:
        setattr(lin, name, types.MethodType(method, lin) if how == "bound" else lambda *a, **kw: method(lin, *a, **kw))
    return lin


HOW = ["subclass", "class", "bound", "function"]


@pytest.mark.parametrize("how", HOW)
@pytest.mark.parametrize("name", ["prepare_input", "apply_prepared"])
def test_forward_runs_a_replaced_step(monkeypatch, how, name):
    x = torch.ones(3, F, dtype=torch.bfloat16)
    lin = _replace(monkeypatch, how, name, lambda self, v, *a, **kw: ("mine", v) if name == "prepare_input" else 2 * v[1])
    if name == "prepare_input":
        monkeypatch.setattr(type(lin), "apply_prepared", lambda self, v: 2 * v[1])
    else:
        monkeypatch.setattr(type(lin), "prepare_input", lambda self, v: ("mine", v))
    assert torch.equal(lin(x), 2 * x)


def test_forward_of_an_untouched_linear_is_one_call(monkeypatch):
    monkeypatch.setattr(ops, "sharq_linear_forward", lambda x, *a, **kw: 3 * x)
    x = torch.ones(3, F, dtype=torch.bfloat16)
    assert torch.equal(_linear()(x), 3 * x)


@pytest.mark.parametrize("how", HOW)
def test_gate_up_and_down_steps_are_kept(monkeypatch, how):
    prep = ("SHARQ", _byte(), _byte(), _byte(), torch.zeros(4, 1), _byte(), torch.ones(()))
    if how != "class":
        gate_up = _replace(monkeypatch, how, "apply_prepared", lambda self, p, **kw: "mine")
        down = types.SimpleNamespace(quant_type="SHARQ", prepare_input_swiglu=lambda gu: ("prepared", gu))
        assert gate_up.apply_prepared_swiglu(prep, down) == ("prepared", "mine")
    down = _replace(monkeypatch, how, "prepare_input_swiglu", lambda self, gu, *a: ("mine", gu))
    assert _linear().apply_prepared_swiglu(prep, down) == ("mine", "gemm")


class _Qkv:
    def prepare_input_rmsnorm(self, x, gamma, eps):
        return x

    def apply_prepared(self, prep):
        return torch.cat((prep, prep, prep), dim=1)


class _GateUp:
    """Only the methods that a decoder layer called before the linears had a joint form."""

    def prepare_input_add_rmsnorm(self, x, residual, gamma, eps):
        return x, x + residual

    def apply_prepared(self, prep):
        return torch.cat((prep, prep), dim=1)


class _Down(QLinearLayer):
    def prepare_input_swiglu(self, gate_up, out_features_hint=None):
        return ("mine", gate_up[:, :F])

    def apply_prepared(self, prepared, out=None, scatter=None):
        return 0.5 * prepared[1]


def _layer(bias=None, down_cls=RowParallelSharqLinear, local_cls=_Down):
    layer = SharqDecoderLayer.__new__(SharqDecoderLayer)
    torch.nn.Module.__init__(layer)
    layer.cfg = DecoderConfig(hidden=F, layers=1, heads=1, kv_heads=1, head_dim=F, ffn=F)
    layer.mode, layer.world, layer.reduce_hook, layer.fused_glue = "SHARQ", 1, None, True
    layer.local_heads = layer.local_kv = 1
    layer.input_norm = layer.post_norm = torch.ones(F, dtype=torch.bfloat16)
    layer.qkv, layer.gate_up = _Qkv(), _GateUp()
    layer.o_proj = lambda x: torch.zeros_like(x)
    down = down_cls.__new__(down_cls)
    torch.nn.Module.__init__(down)
    down.world, down.rank, down.group, down.reduce_hook, down.bias = 1, 0, None, None, bias
    down.local = _linear(local_cls, n=F)
    layer.down = down
    return layer


class _Doubled(RowParallelSharqLinear):
    def reduce(self, y):
        return 2 * y


@pytest.mark.parametrize("case", ["local", "bias", "reduce"])
def test_decoder_layer_keeps_replaced_linears(case):
    bias = torch.full((F,), 4.0, dtype=torch.bfloat16) if case == "bias" else None
    layer = _layer(bias, _Doubled if case == "reduce" else RowParallelSharqLinear)
    x = torch.randn(1, 5, F, generator=torch.Generator().manual_seed(0)).to(torch.bfloat16)
    cos, sin = decoder.rope_tables(5, F, 1e4, "cpu")
    d = 0.5 * x.view(5, F)
    want = x.view(5, F) + (d if case == "local" else 2 * d if case == "reduce" else d + bias)
    assert torch.equal(layer(x, cos, sin), want.view(1, 5, F))


def test_moe_override_is_kept():
    class Sub(SharqDecoderLayer):
        def _moe(self, hn):
            return hn

    layer = Sub.__new__(Sub)
    torch.nn.Module.__init__(layer)
    assert not decoder.methods_kept(layer, decoder._LAYER_METHODS, "_moe", "_moe_grouped")
    plain = SharqDecoderLayer.__new__(SharqDecoderLayer)
    torch.nn.Module.__init__(plain)
    assert decoder.methods_kept(plain, decoder._LAYER_METHODS, "_moe", "_moe_grouped")
