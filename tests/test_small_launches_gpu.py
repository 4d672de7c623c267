"""Launches for few rows: the prepare as a statistics launch that leaves a maximum per CTA and a quantisation launch that
overlap, and split-K GEMMs whose CTAs sum their partial tiles through distributed shared memory."""
import ctypes

import numpy as np
import pytest
import torch

from tests import helpers as H
from tests.test_prepare_gpu import _compare

pytestmark = pytest.mark.gpu


def _prepare(m, k, x, gamma, eps=1e-6):
    """The scaled (RMSNorm) prepare with the workspace that takes the two overlapping launches -> outputs, absmax, scale, inv_rms."""
    from sharq_b200 import _lib
    from tests.gpu_util import Buf, call, dptr, sizes5, stream_ptr

    bufs = [Buf(s) for s in sizes5(m, 128, k)]
    ws_bytes = int(_lib.lib().sharq_prepare_workspace_best_bytes(m))
    ws, scale = Buf(ws_bytes), Buf(4)
    xd = x.cuda()
    tail = (m, 128, k, ws.ptr, ws_bytes, *[b.ptr for b in bufs], scale.ptr, stream_ptr())
    if gamma is None:
        call("sharq_scaled_sparse_residual_quantize_x", dptr(xd), *tail)
    else:
        gd = gamma.cuda()
        call("sharq_fused_rmsnorm_sparse_residual_quantize_x", dptr(xd), dptr(gd), ctypes.c_float(eps), *tail)
    wsh = ws.get()
    return ([b.get() for b in bufs], wsh[:4].view(np.float32)[0], scale.get().view(np.float32)[0],
            wsh[256:256 + 4 * m].view(np.float32))


# one row, around one and two CTAs per SM, the longest row, rows of a chunk, the largest number of CTA maxima and one row more
@pytest.mark.parametrize("m,k", [(1, 4096), (17, 4096), (149, 256), (8, 32768), (300, 1152), (4096, 128), (4097, 128)])
def test_rmsnorm_prepare_in_two_launches_matches_oracle(oracle, m, k):
    x, gamma = H.config0_x(m, k, seed=m + k), H.config0_gamma(k, seed=m)
    got, amax, scale, inv = _prepare(m, k, x, gamma)
    inv_cpu, _, _ = oracle.rmsnorm_row_stats(H.bits(x), H.bits(gamma), 1e-6)
    ulp = np.abs(inv.view(np.int32).astype(np.int64) - inv_cpu.view(np.int32).astype(np.int64))
    assert ulp.max() <= 2  # the sum of squares is order-exact, rsqrtf a <= 2 ulp approximation
    _, amax_rows, _ = oracle.rmsnorm_row_stats(H.bits(x), H.bits(gamma), 1e-6, inv_rms_in=inv)
    assert np.float32(amax_rows.max()) == amax and oracle.tensor_scale(amax, cuda_mode=True) == scale
    _compare(got, oracle.rmsnorm_prepare(H.bits(x), H.bits(gamma), inv, scale), f"rmsnorm {m}x{k}")


# around the size up to which every CTA scans the input, a ragged row, more input than CTAs
@pytest.mark.parametrize("m,k", [(16, 4096), (17, 4096), (33, 1152), (65, 4096), (700, 4096)])
def test_scaled_prepare_in_two_launches_matches_oracle(oracle, m, k):
    x = H.config0_x(m, k, seed=m)
    got, _, scale, _ = _prepare(m, k, x, None)
    s = oracle.tensor_scale(oracle.absmax_bf16(H.bits(x)), cuda_mode=True)
    assert scale == s
    _compare(got, oracle.prepare(oracle.scale_bf16(H.bits(x), s, cuda_mode=True)), f"scaled {m}x{k}")


# two launches, the cooperative launch, and two launches again
@pytest.mark.parametrize("m,k", [(5, 4096), (48, 2048), (1100, 4096), (4096, 8192)])
def test_add_rmsnorm_prepare_equals_the_prepare_of_the_sum(m, k):
    from sharq_b200 import ops

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


# full tiles on both sides of the K from which the fused (18 stages of 256), dense (20) and sparse (29) GEMM are split, with a ragged last stage
@pytest.mark.parametrize("m", [128, 300])
@pytest.mark.parametrize("n,k", [(264, 4480), (300, 5248), (264, 7552)])
def test_split_k_of_full_tiles_against_one_pass(m, n, k, monkeypatch):
    test_split_k_against_one_pass(m, n, k, monkeypatch)


# one CTA, more CTAs than the smallest workspace has words; the smallest workspace, a word short of one per CTA, plenty
@pytest.mark.parametrize("m,k", [(1, 128), (100, 4096), (700, 8192)])
@pytest.mark.parametrize("ws_bytes", [256, 259, 260, 8192])
def test_swiglu_prepare_leaves_the_absmax_in_the_first_word(m, k, ws_bytes):
    from sharq_b200 import ops
    from tests.gpu_util import Buf, call, dptr, sizes5, stream_ptr

    gate_up = H.config0_x(m, 2 * k, seed=m).cuda()
    bufs, ws, scale, h = [Buf(s) for s in sizes5(m, 128, k)], Buf(ws_bytes), Buf(4), Buf(m * k * 2)
    call("sharq_swiglu_sparse_residual_quantize_x", dptr(gate_up), m, 128, k, h.ptr, ws.ptr, ws_bytes, *[b.ptr for b in bufs],
         scale.ptr, stream_ptr())
    want_h = ops.swiglu(gate_up)
    want = ops.scaled_sparse_residual_quantize_x(want_h, 128)
    assert ws.get()[:4].view(np.float32)[0] == float(want_h.float().abs().max())
    assert scale.get().view(np.float32)[0] == float(want[5])
    assert np.array_equal(bufs[3].get().ravel(), want[3].cpu().numpy().ravel())


# the largest input that is scanned by the prepare itself and one row more, with and without room for the CTAs' maxima; the
# workspace is written only where there is a statistics pass
@pytest.mark.parametrize("m,k,minimal,scanned", [(16, 4096, False, True), (17, 4096, False, False), (17, 4096, True, True),
                                                 (48, 4096, True, True), (49, 4096, True, False), (13, 14336, True, True)])
def test_small_input_is_scanned_by_the_prepare(oracle, m, k, minimal, scanned):
    from sharq_b200 import _lib
    from tests.gpu_util import Buf, SENTINEL, call, dptr, sizes5, stream_ptr

    x = H.config0_x(m, k, seed=m)
    ws_bytes = 256 if minimal else int(_lib.lib().sharq_prepare_workspace_best_bytes(m))
    bufs, ws, scale, xd = [Buf(s) for s in sizes5(m, 128, k)], Buf(ws_bytes), Buf(4), x.cuda()
    call("sharq_scaled_sparse_residual_quantize_x", dptr(xd), m, 128, k, ws.ptr, ws_bytes, *[b.ptr for b in bufs], scale.ptr,
         stream_ptr())
    assert bool((ws.get()[:4] == SENTINEL).all()) == scanned
    s = oracle.tensor_scale(oracle.absmax_bf16(H.bits(x)), cuda_mode=True)
    assert scale.get().view(np.float32)[0] == s
    _compare([b.get() for b in bufs], oracle.prepare(oracle.scale_bf16(H.bits(x), s, cuda_mode=True)), f"scaled {m}x{k}")
