"""The form that a scaled prepare takes, from shapes alone (CPU), and its bytes beside the lines (GPU)."""
import numpy as np
import pytest

from sharq_b200 import _lib
from tests import helpers as H

SMS = 148
CTA_SCAN, CLUSTER_SCAN, NARROW, WIDE, ONE_LAUNCH = range(5)


def _form(m, k, rms=0, residual=0, ready=0, minimal=False):
    L = _lib.lib()
    ws = L.sharq_prepare_workspace_bytes(m) if minimal else L.sharq_prepare_workspace_best_bytes(m)
    return L.sharq_scaled_prepare_form(m, k, rms, residual, ready, ws, SMS)


@pytest.mark.parametrize("minimal", [False, True])
def test_scans_without_a_statistics_launch(minimal):
    for m, k, form in ((1, 128, CTA_SCAN), (10, 4096, CTA_SCAN), (11, 4096, CLUSTER_SCAN), (64, 4096, CLUSTER_SCAN), (16, 16384, CLUSTER_SCAN)):
        assert _form(m, k, minimal=minimal) == form
    assert _form(65, 4096, minimal=minimal) == (ONE_LAUNCH if minimal else NARROW)


def test_clusters_are_taken_only_where_all_fit_at_once():
    assert _form(2, 18944) == CTA_SCAN and _form(3, 18944) == WIDE and _form(8, 18944) == WIDE
    # a cooperative launch is the other form: every CTA scans
    assert [_form(m, k, minimal=True) for m, k in ((3, 18944), (8, 18944), (2, 32768))] == [CTA_SCAN] * 3


# a CTA takes 8 tasks of 256 columns: 144 and 148 CTAs, then 150 and 160
@pytest.mark.parametrize("k,most", [(4096, 74), (8192, 37)])
def test_narrow_tensor_scale_is_one_cta_per_sm(k, most):
    assert _form(most, k) == NARROW and _form(most + 1, k) == WIDE


def test_narrow_rmsnorm():
    assert [_form(m, 4096, rms=1) for m in (32, 33, 160, 161)] == [WIDE, NARROW, NARROW, WIDE]
    assert _form(1024, 4096, rms=1, residual=1) == ONE_LAUNCH


def test_a_maximum_that_is_there_keeps_a_group_per_lane():
    assert all(_form(m, k, ready=1) == WIDE for m, k in ((1, 128), (33, 4096), (48, 14336), (72, 4096), (128, 1152), (160, 4096)))


@pytest.mark.gpu
@pytest.mark.parametrize("m,k", [(74, 4096), (75, 4096), (37, 8192), (38, 8192)])
def test_bytes_beside_the_narrow_line(oracle, m, k):
    from tests.test_prepare_gpu import _compare
    from tests.test_small_launches_gpu import _prepare

    x = H.config0_x(m, k, seed=m)
    got, amax, scale, _ = _prepare(m, k, x, None)
    s = oracle.tensor_scale(oracle.absmax_bf16(H.bits(x)), cuda_mode=True)
    assert scale == s and amax == np.float32(x.float().abs().max())
    _compare(got, oracle.prepare(oracle.scale_bf16(H.bits(x), s, cuda_mode=True)), f"scaled {m}x{k}")


@pytest.mark.gpu
@pytest.mark.parametrize("m,k", [(3, 18944), (10, 18944), (2, 32768)])
def test_bytes_of_a_scan_by_every_cta(oracle, m, k):
    from tests.gpu_util import Buf, call, dptr, sizes5, stream_ptr
    from tests.test_prepare_gpu import _compare

    x = H.config0_x(m, k, seed=m)
    ws_bytes = int(_lib.lib().sharq_prepare_workspace_bytes(m))
    bufs, ws, scale, xd = [Buf(s) for s in sizes5(m, 128, k)], Buf(ws_bytes), Buf(4), x.cuda()
    call("sharq_scaled_sparse_residual_quantize_x", dptr(xd), m, 128, k, ws.ptr, ws_bytes, *[b.ptr for b in bufs], scale.ptr,
         stream_ptr())
    s = oracle.tensor_scale(oracle.absmax_bf16(H.bits(x)), cuda_mode=True)
    assert scale.get().view(np.float32)[0] == s
    _compare([b.get() for b in bufs], oracle.prepare(oracle.scale_bf16(H.bits(x), s, cuda_mode=True)), f"scaled {m}x{k}")


# a maximum that the SwiGLU kernel left, and an input that needs none
@pytest.mark.gpu
@pytest.mark.parametrize("m,k", [(33, 1152), (72, 4096)])
def test_bytes_without_a_statistics_launch(oracle, m, k):
    import torch

    from sharq_b200 import ops
    from tests.test_prepare_gpu import _compare

    gate_up = H.config0_x(m, 2 * k, seed=m).cuda()
    h = ops.swiglu(gate_up)
    got, want = ops.swiglu_sparse_residual_quantize_x(gate_up, 128), ops.scaled_sparse_residual_quantize_x(h, 128)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    plain = ops.fused_sparse_residual_quantize_x(h, 128)
    _compare([t.cpu().numpy().reshape(-1) for t in plain], oracle.prepare(H.bits(h.cpu())), f"scaled input {m}x{k}")
