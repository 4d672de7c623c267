"""The forms of the scaled prepare at the sizes where one hands over to the next: a scan by every CTA, a scan by clusters, a statistics
launch with 8 elements per lane, and with a group per lane; all against the oracle, byte for byte."""
import numpy as np
import pytest
import torch

from tests import helpers as H
from tests.test_prepare_gpu import _compare
from tests.test_small_launches_gpu import _prepare

pytestmark = pytest.mark.gpu

# one row of the smallest and of an odd K, half a 256-column tile at the end, both sides of every line, more rows than a band
SHAPES = [(1, 128), (1, 4096), (3, 384), (10, 4096), (11, 4096), (64, 4096), (65, 4096), (129, 1152), (160, 4096), (161, 4096), (18, 14336),
          (19, 14336), (8, 18944), (2, 32768), (512, 1152)]


@pytest.mark.parametrize("m,k", SHAPES)
@pytest.mark.parametrize("spread", ["plain", "subnormal"])
def test_scaled_prepare(oracle, m, k, spread):
    x = H.config0_x(m, k, seed=m)
    if spread == "subnormal":  # one value so large that most quotients are subnormal, and the pairs are picked among those
        x = (x.float() * 1e-3).to(torch.bfloat16)
        x[m // 2, k // 3] = 3e38
    got, amax, scale, _ = _prepare(m, k, x, None)
    s = oracle.tensor_scale(oracle.absmax_bf16(H.bits(x)), cuda_mode=True)
    assert scale == s
    if m * k > 64 * 1024:
        assert amax == np.float32(x.float().abs().max())
    _compare(got, oracle.prepare(oracle.scale_bf16(H.bits(x), s, cuda_mode=True)), f"scaled {m}x{k} {spread}")


@pytest.mark.parametrize("m,k", SHAPES)
def test_rmsnorm_prepare(oracle, m, k):
    x, gamma = H.config0_x(m, k, seed=m + 1), H.config0_gamma(k, seed=m)
    got, amax, scale, inv = _prepare(m, k, x, gamma)
    _, amax_rows, _ = oracle.rmsnorm_row_stats(H.bits(x), H.bits(gamma), 1e-6, inv_rms_in=inv)
    assert np.float32(amax_rows.max()) == amax and oracle.tensor_scale(amax, cuda_mode=True) == scale
    _compare(got, oracle.rmsnorm_prepare(H.bits(x), H.bits(gamma), inv, scale), f"rmsnorm {m}x{k}")


# the already scaled input takes the same two forms
@pytest.mark.parametrize("m,k", [(1, 128), (33, 1152), (160, 4096), (161, 4096)])
def test_prepare_of_a_scaled_input(oracle, m, k):
    from sharq_b200 import ops

    x = H.config0_x(m, k, seed=m)
    got = ops.fused_sparse_residual_quantize_x(x.cuda(), 128)
    _compare([t.cpu().numpy().reshape(-1) for t in got], oracle.prepare(H.bits(x)), f"scaled input {m}x{k}")
