"""Split GEMMs on both sides of the lines between the ways in which partial tiles meet, in narrow and wide tiles, against one pass over K
(bounds of test_split_k_against_one_pass); a residual is added to the same bits."""
import pytest
import torch

from tests import helpers as H
from tests.test_small_launches_gpu import test_split_k_against_one_pass as against_one_pass

pytestmark = pytest.mark.gpu


# 36, 40 and 17 stages over 8, 8 and 4 CTAs: 4 to 5, 5 and 4 to 5 of them each, so that the receiving slot moves; a last tile of 32, 33 and 65 rows
@pytest.mark.parametrize("m", [32, 33, 64, 65, 80, 81, 128, 160, 161, 193])
@pytest.mark.parametrize("n,k", [(1024, 9216), (520, 10240), (3584, 4352)])
def test_narrow_tiles(m, n, k, monkeypatch):
    against_one_pass(m, n, k, monkeypatch)


# the smallest N whose narrow tiles fill more than half of 148 SMs at two and at three rows of tiles, a K just above the line
@pytest.mark.parametrize("m,n", [(129, 4864), (384, 3200)])
def test_wide_tiles_of_a_long_k(m, n, monkeypatch):
    from sharq_b200 import _lib

    assert _lib.lib().sharq_gemm_tile_n(m, n, 16640, 1, 148) == 256
    against_one_pass(m, n, 16640, monkeypatch)


# rows that are sent from registers, as blocks (room in some layouts), read; a ragged second column tile
@pytest.mark.parametrize("m", [1, 32, 33, 64, 65, 81, 128, 300])
@pytest.mark.parametrize("k", [9216, 10496])
def test_wide_tiles(m, k, monkeypatch):
    from sharq_b200 import ops

    ops.set_gemm_tile_n(256)
    try:
        against_one_pass(m, 520, k, monkeypatch)
    finally:
        ops.set_gemm_tile_n(0)


@pytest.mark.parametrize("m", [1, 33, 65, 129])
@pytest.mark.parametrize("tile_n", [128, 256])
def test_residual(m, tile_n):
    from sharq_b200 import ops
    from sharq_b200.quantize import quantize_weight_shared_nvfp4

    n, k = 1024, 9216
    x, r = H.config0_x(m, k, m).cuda(), H.config0_x(m, n, n).cuda()
    bias = H.config0_x(1, n, 3).cuda().reshape(n)
    qw, sfs, sfd, scale = quantize_weight_shared_nvfp4(H.config0_w(n, k, n).cuda())
    a = ops.scaled_sparse_residual_quantize_x(x, n)
    alpha = (a[5] * scale).reshape(1)
    ops.set_gemm_tile_n(tile_n)
    try:
        plain = ops.sharq_linear_gemm(*a[:5], qw, sfs, sfd, alpha, bias=bias)
        summed = ops.sharq_linear_gemm(*a[:5], qw, sfs, sfd, alpha, bias=bias, residual=r)
    finally:
        ops.set_gemm_tile_n(0)
    ops.check_device_errors()
    assert torch.equal(summed, plain + r)
