"""Launches for few rows: the prepare as one thread-block cluster, and split-K GEMMs whose CTAs sum their partial tiles
through distributed shared memory."""
import pytest
import torch

from tests import helpers as H
from tests import test_prepare_gpu as prepare

pytestmark = pytest.mark.gpu


# one row per CTA, one more than the CTAs, the largest input of the form, the longest row, the next size up
@pytest.mark.parametrize("m,k", [(1, 4096), (16, 4096), (17, 4096), (64, 4096), (8, 32768), (65, 4096)])
def test_small_rmsnorm_prepare_matches_oracle(oracle, m, k):
    prepare.test_rmsnorm_prepare_matches_oracle(oracle, m, k)


@pytest.mark.parametrize("m,k", [(8, 4096), (9, 4096), (33, 1152), (64, 4096), (65, 4096)])
def test_small_scaled_prepare_matches_oracle(oracle, m, k):
    prepare.test_scaled_prepare_matches_oracle(oracle, m, k)


def test_small_add_rmsnorm_prepare_equals_the_prepare_of_the_sum():
    from sharq_b200 import ops

    for m, k in ((5, 4096), (48, 2048)):
        x, r, g = H.config0_x(m, k, m).cuda(), H.config0_x(m, k, m + 1).cuda(), H.config0_gamma(k, m).cuda()
        got = ops.fused_add_rmsnorm_sparse_residual_quantize_x(x, r, g, 1e-6, 128)
        assert torch.equal(got[6], x + r)
        want = ops.fused_rmsnorm_sparse_residual_quantize_x(x + r, g, 1e-6, 128)
        assert all(torch.equal(a, b) for a, b in zip(got[:6], want))


# rows: one, a quadrant of the accumulator and one more, a full tile, two tiles with a ragged second; columns: one tile,
# ragged (also not a multiple of 8), several; K: two stages per CTA, ragged last stage, the most CTAs per cluster
@pytest.mark.parametrize("m", [1, 33, 128, 211])
@pytest.mark.parametrize("n,k", [(128, 1024), (264, 1152), (300, 4224), (1024, 8192)])
def test_split_k_against_one_pass(m, n, k, monkeypatch):
    from sharq_b200 import ops
    from sharq_b200.quantize import quantize_weight_shared_nvfp4

    x, c = H.config0_x(m, k, m).cuda(), H.config0_x(m, n, n).cuda()
    bias = H.config0_x(1, n, 3).cuda().reshape(n)
    qw, sfs, sfd, scale = quantize_weight_shared_nvfp4(H.config0_w(n, k, n).cuda())
    a = ops.scaled_sparse_residual_quantize_x(x, n)
    alpha = (a[5] * scale).reshape(1)

    def run():
        return (ops.sharq_linear_gemm(*a[:5], qw, sfs, sfd, alpha, bias=bias),
                ops.sparse_matmul_tensor_scale(a[0], qw, a[1], a[2], sfs, m, n, k, alpha),
                ops.matmul_accum_tensor_scale(a[3], qw, a[4], sfd, alpha, c, 0.5))

    monkeypatch.setenv("SHARQ_GEMM_SPLIT_K", "1")
    split, again = run(), run()
    monkeypatch.setenv("SHARQ_GEMM_SPLIT_K", "0")
    whole = run()
    ops.check_device_errors()
    for s, t, w in zip(split, again, whole):
        assert torch.equal(s, t)  # a fixed order of additions
        # both round an fp32 sum once (twice with a bias) to bf16: one bf16 step apart at most, and where the sum
        # cancels the orders of addition differ by K * 2^-24 of the terms, far below 2^-10 of the largest element
        d, size = (s.float() - w.float()).abs(), w.float().abs()
        assert bool((d <= size * 2.0 ** -7 + float(size.max()) * 2.0 ** -10).all())
