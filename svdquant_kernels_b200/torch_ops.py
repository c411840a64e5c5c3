"""torch.library registration of the two operators, for callers that want dispatcher-visible ops
(`torch.ops.svdq_b200.*`): tracing / torch.compile graphs, CUDA-graph capture through the dispatcher,
serving stacks that resolve kernels by qualified name.

The reference registers nothing on CUDA and keeps its pod-side registration as a pattern only
(csrc/python/svdquant_w4a4_op.cpp:127-136, docs/architecture.md:18-22); the schemas below follow its
Python signatures (triton_kernels/quantize_w4a4_act_fuse_lora/kernel.py:289-400,
cute_kernels/gemm_w4a4/kernel_v2_fa4.py:113-225).

The ops are defined and implemented in the native host path (csrc/host_ops.cpp), so a call goes from
the dispatcher to the launch without entering Python; calls that need more than a launch (first use of
a weight, strided inputs, broken contracts) come back to the operators of `ops`.  The layout twins `ops`
makes next to its outputs (tensor-core scale order, 16-bit lora_act) are recorded on the outputs' storage
objects, which the dispatcher hands through unchanged, so a `torch.ops.svdq_b200.gemm_w4a4` call on the
quantizer op's outputs finds them and runs the same kernels as the plain Python path; both ops can be
captured in a CUDA graph.
"""
from __future__ import annotations

import torch

from . import _lib

__all__ = ["quantize_w4a4_act_fuse_lora", "gemm_w4a4"]

_lib.host()                                  # loading the extension defines the ops
quantize_w4a4_act_fuse_lora = torch.ops.svdq_b200.quantize_w4a4_act_fuse_lora
gemm_w4a4 = torch.ops.svdq_b200.gemm_w4a4


@torch.library.register_fake("svdq_b200::quantize_w4a4_act_fuse_lora")
def _(input, lora_down, smooth=None, pad_size=256):
    M, K = input.shape
    R = lora_down.shape[1]
    torch._check(K % 16 == 0, lambda: "NVFP4 group size is 16; K must be divisible by 16")
    M_pad = (M + pad_size - 1) // pad_size * pad_size
    return (input.new_empty((M_pad, K // 2), dtype=torch.uint8),
            input.new_empty((K // 16, M_pad), dtype=torch.float8_e4m3fn),
            input.new_empty((M_pad, R), dtype=torch.float32))


@torch.library.register_fake("svdq_b200::gemm_w4a4")
def _(act, wgt, ascales, wscales, lora_act_in=None, lora_up=None, wcscales=None, bias=None, out_dtype=None):
    if out_dtype is None:
        out_dtype = lora_up.dtype if lora_up is not None else torch.float16
    return act.new_empty((act.shape[0], wgt.shape[0]), dtype=out_dtype)
