"""Host-side quantisation helpers with the names and meaning of the reference's
model/quantize.py (lines 43-44, 141-200), running on the sm_100a ops.

Differences in mechanism only: the helpers fold the tensor-scale passes (amax, divide) into
the kernels instead of running them as separate PyTorch ops; the returned tuples are the same.
Other dtypes than bf16 and widths that the folded kernels do not take keep the PyTorch passes.
"""
from __future__ import annotations

import functools

import torch

from . import ops


def without_grad(fn):
    """torch.no_grad() around calls that come with gradients enabled.  The calls of a layer nest up to three deep, and each of them
    paid 2 us for turning off what was off; looking costs 0.1."""
    guarded = torch.no_grad()(fn)

    @functools.wraps(fn)
    def call(*args, **kwargs):
        return guarded(*args, **kwargs) if torch.is_grad_enabled() else fn(*args, **kwargs)

    return call


def global_nvfp4_scale(x: torch.Tensor) -> torch.Tensor:
    """clamp(max|x| / (448*6), 1e-9) as a 0-dim float32 tensor (model/quantize.py:43-44)."""
    return torch.clamp(x.abs().max().float() / (448.0 * 6.0), min=1e-9)


def _folds(x: torch.Tensor, k_multiple: int) -> bool:
    """Whether the scaled quantisation kernels take x as it is."""
    return (x.is_cuda and x.dtype == torch.bfloat16 and x.dim() == 2 and x.numel() > 0 and x.shape[1] % k_multiple == 0
            and x.shape[1] <= 32768)


@without_grad
def quantize_weight_shared_nvfp4(weight: torch.Tensor):
    """-> (q_weight, scale_weight_sparse, scale_weight_dense, scale) (model/quantize.py:149-153)."""
    if _folds(weight, 128):
        return ops.scaled_quantize_w32_shared(weight)
    scale = global_nvfp4_scale(weight)
    q, sfs, sfd = ops.quantize_w32_shared((weight / scale).to(torch.bfloat16).contiguous())
    return q, sfs, sfd, scale


@without_grad
def quantize_weight_nvfp4(weight: torch.Tensor):
    """-> (q_weight, scale_weight, scale) (model/quantize.py:141-145)."""
    if _folds(weight, 64):
        return ops.scaled_quantize_nvfp4(weight)
    scale = global_nvfp4_scale(weight)
    q, sf = ops.quantize_w_nvfp4((weight / scale).to(torch.bfloat16).contiguous())
    return q, sf, scale


@without_grad
def quantize_activation_nvfp4(x: torch.Tensor):
    """-> (q_x, scale_x, scale) (model/quantize.py:165-169)."""
    if _folds(x, 64):
        return ops.scaled_quantize_nvfp4(x)
    scale = global_nvfp4_scale(x)
    q, sf = ops.quantize_x_nvfp4((x / scale).to(torch.bfloat16).contiguous())
    return q, sf, scale


@without_grad
def quantize_activation_sparse_residual_nvfp4(x: torch.Tensor, out_features: int):
    """-> (a_comp, e, sfa_sparse, q_res, sf_res, scale) (model/quantize.py:179-183)."""
    return ops.scaled_sparse_residual_quantize_x(x.to(torch.bfloat16).contiguous(), out_features)


@without_grad
def quantize_activation_rmsnorm_sparse_residual_nvfp4(x: torch.Tensor, rmsnorm_weight: torch.Tensor,
                                                      rmsnorm_eps: float, out_features: int):
    """-> (a_comp, e, sfa_sparse, q_res, sf_res, scale) (model/quantize.py:187-200)."""
    return ops.fused_rmsnorm_sparse_residual_quantize_x(
        x.to(torch.bfloat16).contiguous(), rmsnorm_weight.to(torch.bfloat16).contiguous(), float(rmsnorm_eps),
        out_features)


def apply_rmsnorm(x: torch.Tensor, weight: torch.Tensor, eps: float) -> torch.Tensor:
    """Unfused RMSNorm in PyTorch, used only by the dense NVFP4 baseline mode (model/quantize.py:47-51)."""
    xf = x.float()
    inv = torch.rsqrt(xf.pow(2).mean(dim=-1, keepdim=True) + eps)
    return (xf * inv * weight.float()).to(torch.bfloat16)
