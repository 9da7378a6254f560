"""Host side of the biased, key-masked attention operator.

Mirrors what the reference does between its Python wrapper and its C++ entry
(src/af3_kernels/__init__.py:31-52 -> src/csrc/dot_product_attention.cpp:545-559): rank-lifts
the mask, checks dtypes and shapes, allocates the output, and calls the C ABI of libaf3k.so
with raw device pointers on the current CUDA stream.  For CUDA tensors all of that is native code
(``csrc/host_torch.cpp``); what is left here are the rare forms of the arguments and the pipelined
call on host tensors.  There is no CPU path.
"""
from __future__ import annotations

import math
import os
from typing import Optional

import torch

from . import _capi

_DEBUG = os.environ.get("AF3K_DEBUG", "0") == "1"


def _status_buffer(device: torch.device) -> torch.Tensor:
    index = device.index if device.index is not None else torch.cuda.current_device()
    return _capi.host().status_buffer(index)


def read_status(device: torch.device) -> list:
    """Synchronises and returns the device status words {bits, 1+barrier, block, warp}; clears them."""
    buf = _status_buffer(torch.device(device))
    vals = buf.cpu().tolist()
    buf.zero_()
    return vals


class StagedBias:
    """A bias converted once into the form the kernel reads in place (bf16, rows padded to 16
    bytes; with fp8 q/k also divided by each head's logit scale).  Made by ``stage_bias``; pass it
    to ``dot_product_attention`` instead of the bias tensor."""

    def __init__(self, data: torch.Tensor, B2: int, Sq: int, Sk: int, prescaled: bool):
        self.data, self.B2, self.Sq, self.Sk, self.prescaled = data, B2, Sq, Sk, prescaled


def stage_bias(bias: torch.Tensor, B2: int, Sq: int, Sk: int, *, q_scale=None, k_scale=None,
               softmax_scale: Optional[float] = None, head_dim: int = 32) -> StagedBias:
    """Runs the bias staging pass on its own (``af3k_stage_bias``) on the current stream, for a
    bias that is applied in many calls: those calls then launch one kernel instead of two.
    ``softmax_scale`` / ``head_dim`` matter only with fp8 scales (the copy is divided by
    ``softmax_scale * q_scale[h] * k_scale[h]``, default scale ``1/sqrt(head_dim)``)."""
    if not bias.is_cuda:
        raise RuntimeError("af3_kernels_b200 runs on CUDA tensors only (no CPU fallback)")
    if bias.numel() != B2 * Sq * Sk:
        raise ValueError(f"bias must have B2*Sq*Sk = {B2 * Sq * Sk} elements, got {bias.numel()}")
    fp8 = q_scale is not None
    if fp8:
        q_scale = q_scale.to(device=bias.device, dtype=torch.float32).contiguous()
        k_scale = k_scale.to(device=bias.device, dtype=torch.float32).contiguous()
        if q_scale.numel() != B2 or k_scale.numel() != B2:
            raise ValueError("q_scale / k_scale must have one entry per head")
    staged = _capi.host().stage_bias(bias, B2, Sq, Sk, head_dim, q_scale, k_scale if fp8 else None,
                                     float(softmax_scale) if softmax_scale is not None else 1.0 / math.sqrt(head_dim))
    return StagedBias(staged, B2, Sq, Sk, fp8)


def readable_bias(bias: torch.Tensor, B2: int, Sq: int, Sk: int) -> torch.Tensor:
    """``bias`` itself where the kernel reads it in place with bf16 q/k, else a bf16 copy ``[B2, Sq, Sk]`` made now that it
    can read: for several calls of one step on the same bias."""
    if (bias.dtype == torch.bfloat16 and bias.shape == (B2, Sq, Sk) and bias.stride(2) == 1 and bias.stride(1) % 8 == 0
            and bias.stride(0) % 8 == 0 and 0 not in bias.stride() and bias.data_ptr() % 16 == 0):
        return bias
    return bias if bias.numel() == 0 or not bias.is_cuda else stage_bias(bias, B2, Sq, Sk).data[:, :, :Sk]


def _mask_rows(mask: Optional[torch.Tensor], B1: int, Sk: int):
    """-> (uint8 tensor [rows, Sk] with unit inner stride, row stride in bytes) or (None, 0).

    1-D [Sk] broadcasts over the batch; 2-D is [B1, Sk]; higher ranks must be [B1|1, 1, 1, Sk]
    (what the reference builds at src/af3_kernels/__init__.py:41-44).  True / non-zero = attend.
    """
    if mask is None:
        return None, 0
    if mask.dim() == 0:
        raise ValueError("mask must have at least one dimension")
    if mask.dim() >= 3:
        if mask.shape[-1] != Sk or mask.numel() not in (Sk, B1 * Sk):
            raise ValueError(f"mask of shape {tuple(mask.shape)} is not [B1|1, 1, 1, Sk]")
        mask = mask.reshape(-1, Sk)
    if mask.dim() == 1:
        mask = mask[None, :]
    if mask.shape[-1] != Sk or mask.shape[0] not in (1, B1):
        raise ValueError(f"mask of shape {tuple(mask.shape)} does not match B1={B1}, Sk={Sk}")
    if mask.dtype != torch.bool:
        mask = mask != 0
    mask = mask.contiguous().view(torch.uint8)
    stride = 0 if (mask.shape[0] == 1 and B1 != 1) else Sk
    return mask, stride


def bool_mask(mask: Optional[torch.Tensor], B1: int, Sk: int) -> Optional[torch.Tensor]:
    """The mask as the native path takes it: None, or bool ``[Sk]`` or ``[1 | B1, Sk]``."""
    if mask is None or (mask.dtype is torch.bool and mask.dim() in (1, 2)):
        return mask
    return _mask_rows(mask, B1, Sk)[0].view(torch.bool)


def dot_product_attention(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    mask: Optional[torch.Tensor],
    bias: torch.Tensor,
    *,
    q_scale: Optional[torch.Tensor] = None,
    k_scale: Optional[torch.Tensor] = None,
    softmax_scale: Optional[float] = None,
    rows_per_item: int = 0,
    out: Optional[torch.Tensor] = None,
    check_status: Optional[bool] = None,
    use_workspace: bool = True,
    cache_bias: bool = True,
    max_ctas: int = 0,
) -> torch.Tensor:
    """softmax(scale * q k^T + bias, key-masked) v on the current CUDA stream.

    q, k, v: [B1, B2, S, D] on one CUDA device.  q/k bf16, or float8_e4m3fn with per-head fp32
    ``q_scale`` / ``k_scale`` [B2].  v bf16.  bias: B2*Sq*Sk elements, bf16 or fp32, shared by
    every b1.  mask: see ``_mask_rows``.  Returns a new bf16 tensor; inputs are not modified.
    ``use_workspace=False`` hands the library no scratch: a bias that needs a staging copy (fp32, or
    rows that are not 16-byte aligned) is then refused, and fp8 q/k run on the kernel variant whose
    softmax threads add the bias themselves.  ``bias`` may be a ``StagedBias``; a plain tensor
    that needs the staging pass is staged once and the copy is reused while the same, unmodified
    tensor object keeps being passed (``cache_bias=False`` stages inside every call instead).
    Unmodified means by its version counter: after a write that bumps none (``bias.data``, a
    collective, a graph replay or a kernel on the raw pointer) pass ``cache_bias=False`` or call
    ``torch.autograd.graph.increment_version(bias)``.  Under stream capture it is always staged
    inside the graph.
    ``max_ctas`` > 0 caps the kernel's grid, leaving the other SMs to a kernel that runs beside it.
    """
    if mask is not None and q.dim() == 4 and k.dim() == 4:
        mask = bool_mask(mask, q.shape[0], k.shape[2])
    form = 0
    if isinstance(bias, StagedBias):
        fp8 = q.dtype == torch.float8_e4m3fn
        if q.dim() != 4 or (bias.B2, bias.Sq, bias.Sk) != (q.shape[1], q.shape[2], k.shape[2]) or bias.prescaled != fp8:
            raise ValueError("staged bias was made for another shape or another q/k type")
        form = 2 if bias.prescaled else 1
        bias = bias.data[:, :, :bias.Sk]
    out = _capi.host().attention(q, k, v, mask, bias, q_scale, k_scale, softmax_scale, rows_per_item, out,
                                 use_workspace, cache_bias, max_ctas, form)
    if check_status if check_status is not None else _DEBUG:
        st = read_status(q.device)
        if st[0] != 0:
            raise RuntimeError(
                f"af3k kernel reported status {st[0]} (wait timeout: barrier slot {st[1] - 1}, "
                f"block {st[2]}, warp {st[3]})"
            )
    return out


def dot_product_attention_host(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    mask: Optional[torch.Tensor],
    bias: torch.Tensor,
    *,
    q_scale: Optional[torch.Tensor] = None,
    k_scale: Optional[torch.Tensor] = None,
    softmax_scale: Optional[float] = None,
    out: Optional[torch.Tensor] = None,
    device: Optional[torch.device] = None,
    chunks: int = 8,
) -> torch.Tensor:
    """The same operator for HOST tensors (what a caller of the reference, a CPU library, holds):
    q, k, v ``[B1, B2, S, D]`` in host memory, result in host memory.

    The batch rows are independent problems, so the call is a three-stage pipeline over up to
    ``chunks`` row blocks (fewer when the blocks would get small) on three CUDA streams:
    host-to-device copies of block *i + 1*, the kernel on block *i* and the device-to-host copy of
    block *i - 1* run at the same time (PCIe is full duplex), so the call costs about the time of
    the larger transfer instead of the sum of all three.  Bias and
    mask go over once.  Pinned host tensors (``tensor.pin_memory()``) are what makes the copies
    asynchronous; pageable ones work but serialise.  ``out`` may be a preallocated (pinned) host
    tensor.  The call returns after the result has arrived in host memory.
    """
    if q.is_cuda or k.is_cuda or v.is_cuda:
        raise ValueError("dot_product_attention_host takes host tensors; use dot_product_attention for CUDA ones")
    if not torch.cuda.is_available():
        raise RuntimeError("af3_kernels_b200 needs a CUDA device (there is no CPU fallback)")
    dev = torch.device(device) if device is not None else torch.device("cuda", torch.cuda.current_device())
    if dev.index is None:
        dev = torch.device("cuda", torch.cuda.current_device())
    if q.dim() != 4:
        raise ValueError("q, k, v must be 4-D [B1, B2, S, D]")
    B1, B2, Sq, D = q.shape
    if out is None:
        out = torch.empty((B1, B2, Sq, D), dtype=torch.bfloat16, pin_memory=True)
    elif out.is_cuda or out.shape != (B1, B2, Sq, D) or out.dtype != torch.bfloat16 or not out.is_contiguous():
        raise ValueError("out must be a contiguous bf16 host tensor [B1, B2, Sq, D]")
    if B1 == 0 or out.numel() == 0:
        return out
    mask = bool_mask(mask, B1, k.shape[2])
    _capi.host().host_attention(q, k, v, mask, bias, q_scale, k_scale, softmax_scale, out, dev.index, max(1, int(chunks)))
    return out
