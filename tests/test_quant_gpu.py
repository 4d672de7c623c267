"""Bit-exact parity of the weight / dense quantisation kernels with the CPU oracle."""
import numpy as np
import pytest
import torch

from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(1, 32), (130, 256), (256, 4096), (384, 3584)])
def test_quantize_w32_shared(oracle, n, k):
    from tests.gpu_util import Buf, call, dptr, stream_ptr

    w = H.config0_w(n, k, seed=n)
    w = (w.float() / (w.float().abs().max() / 2688.0)).to(torch.bfloat16)
    wd = w.cuda()
    sf = (n // 128 + 1) * 128 * k // 16
    bufs = [Buf(n * k // 2), Buf(sf), Buf(sf)]
    call("sharq_quantize_w32_shared", dptr(wd), n, k, *[b.ptr for b in bufs], stream_ptr())
    got = [b.get() for b in bufs]
    want = oracle.quantize_w32_shared(H.bits(w))
    for name, g, wv in zip(("qw", "sfw_sparse", "sfw_dense"), got, want):
        assert np.array_equal(g, np.asarray(wv).reshape(-1)), name
    # duplicate op reproduces the dense view from the sparse one
    dup = Buf(sf)
    call("sharq_duplicate_sfa32_to_sfa16", bufs[1].ptr, n, 64, k, dup.ptr, stream_ptr())
    assert np.array_equal(dup.get(), want[2])


@pytest.mark.parametrize("rows,k", [(1, 16), (33, 128), (130, 2048), (64, 14336), (16, 3584)])
def test_quantize_dense_nvfp4(oracle, rows, k):
    from tests.gpu_util import Buf, SENTINEL, call, dptr, stream_ptr

    x = H.config0_x(rows, k, seed=rows + 1)
    x = (x.float() / (x.float().abs().max() / 2688.0)).to(torch.bfloat16)
    xd = x.cuda()
    sf = (rows // 128 + 1) * 128 * k // 16
    bufs = [Buf(rows * k // 2), Buf(sf)]
    call("sharq_quantize_nvfp4", dptr(xd), rows, k, *[b.ptr for b in bufs], stream_ptr())
    q, s = [b.get() for b in bufs]
    wq, ws = oracle.quantize_dense_nvfp4(H.bits(x), fill=SENTINEL)  # unwritten bytes stay as they were
    assert np.array_equal(q, wq.reshape(-1))
    assert np.array_equal(s, ws)


def test_compress_sparse_a(oracle):
    from tests.gpu_util import Buf, call, dptr, stream_ptr

    m, k, n = 70, 512, 128
    x = H.outlier_rich_x(m, k, 11)
    dense = oracle.prepare(H.bits(x), debug=True)[0]
    # add corner cases: empty chunks, single survivors at each position, minus zeros
    dense[0, :8] = 0
    dense[1, :4] = [0, 0, 0, 0x23]
    dense[1, 4:8] = [0, 0x51, 0, 0]
    dense[2, :4] = [0x88, 0x08, 0x33, 0x80]
    dd = torch.from_numpy(dense).cuda()
    bufs = [Buf(m * k // 4), Buf(((m + 127) // 128 * 128) * k // 16)]
    call("sharq_compress_sparse_a", dptr(dd), m, n, k, *[b.ptr for b in bufs], stream_ptr())
    got = [b.get() for b in bufs]
    want = oracle.compress_sparse_a(dense)
    assert np.array_equal(got[0], want[0])
    assert np.array_equal(got[1], want[1])


@pytest.mark.parametrize("rows,k", [(1, 128), (7, 384), (127, 14336), (128, 4096), (129, 256), (1000, 18944)])
@pytest.mark.parametrize("peak", [1.0, 1.90625, 3e38, 1e-30])
def test_scaled_quantisation_equals_the_torch_passes(rows, k, peak):
    """Edges of the 128-row scale bands and of the 256-group chunks; absmax values whose bf16(scale) is a power of
    two, a short significand, near overflow and clamped to 1e-9.  Bytes equal those of torch's own absmax and division
    in front of the quantisation of the scaled tensor."""
    from sharq_b200 import ops, quantize

    x = H.config0_x(rows, k, seed=rows)
    x = (x.float() * (peak / x.float().abs().max())).to(torch.bfloat16).cuda()
    scale = quantize.global_nvfp4_scale(x)
    scaled = (x / scale).to(torch.bfloat16).contiguous()
    qw, sfs, sfd, got_scale = ops.scaled_quantize_w32_shared(x)
    for got, want in zip((qw, sfs, sfd), ops.quantize_w32_shared(scaled)):
        assert torch.equal(got, want)
    assert torch.equal(got_scale, scale)
    q, sf, got_scale = ops.scaled_quantize_nvfp4(x)
    want_q, want_sf = ops.quantize_x_nvfp4(scaled)
    assert torch.equal(q, want_q) and torch.equal(got_scale, scale)
    r = torch.arange(rows, device="cuda")[:, None]
    g = torch.arange(k // 16, device="cuda")[None]
    at = (r // 128) * (k // 64) * 512 + (g // 4) * 512 + (r % 32) * 16 + ((r // 32) % 4) * 4 + g % 4  # padding is not written
    assert torch.equal(sf[at], want_sf[at])


def test_scaled_quantisation_keeps_a_nan_like_the_torch_passes():
    from sharq_b200 import ops, quantize

    x = H.config0_x(40, 256, seed=3).cuda()
    x[7, 100] = float("nan")
    scaled = (x / quantize.global_nvfp4_scale(x)).to(torch.bfloat16).contiguous()
    qw, sfs, sfd, scale = ops.scaled_quantize_w32_shared(x)
    assert bool(torch.isnan(scale))
    for got, want in zip((qw, sfs, sfd), ops.quantize_w32_shared(scaled)):
        assert torch.equal(got, want)


def test_scaled_quantisations_back_to_back_without_a_synchronisation():
    """Calls whose kernels are all dependents of one another, with the scratch of each handed to the next by the
    allocator: every call gets its own scale (absmax 1, 2, 4, ...), whatever the one before it left there."""
    from sharq_b200 import ops, quantize

    x = H.config0_x(512, 1024, seed=2).cuda()
    x = x / x.abs().max()
    inputs = [x * 2.0 ** i for i in range(24)]
    torch.cuda.synchronize()
    scales = [(ops.scaled_quantize_w32_shared if i % 2 else ops.scaled_quantize_nvfp4)(v)[-1] for i, v in enumerate(inputs)]
    for got, v in zip(scales, inputs):
        assert torch.equal(got, quantize.global_nvfp4_scale(v))
