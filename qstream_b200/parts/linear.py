"""The matrix product y = act(x W^T + b) + residuals, and the choice of its kernel.

bfloat16 activations with a bfloat16 matrix run on the tensor cores (tcgen05, fed by
TMA, 32-bit accumulation).  float32 activations with a float32 matrix run there too, every
number as three bfloat16 terms and the sums rounded in 32 bits outside the unit, where more than a
few rows meet enough products; everything else (few rows, mixed types) runs on the CUDA cores in
true 32-bit.  Each kernel sums a row's products in an order that does not depend on
the other rows' contents.
"""
from __future__ import annotations

import torch

from ..csrc import ops

TENSOR_CORE_ACTIVATIONS = (None, "none", "gelu_new", "gelu")
# float32: from how many rows and products per result on the tensor cores serve.  Microseconds, CUDA cores | tensor cores (caches
# flushed, launches included): 16 rows, 6144 x 2048: 32 | 34; 17 rows, 2048 x 8192: 54 | 40; 32, 2048 x 2048: 28 | 21; 64, 6144 x 2048: 60 | 36; 700,
# 64 x 1024: 24 | 24; 700, 2048 x 64: 49 | 18, but 64 x 64: 12 | 12; 128, 256 x 256: 20 | 15; 700, 6144 x 2048: 412 | 99; 2048, 16384 x 4096: 5159 | 1138.
SPLIT_ROWS, SPLIT_PRODUCTS = 17, 256
OWN_KERNEL_ACTIVATIONS = ("relu2",)         # in no product's epilogue: applied by a kernel of their own behind the product


def linear(x, weight, bias=None, activation=None, residuals=(), out_dtype=None, out=None) -> torch.Tensor:
    """`out`: an optional view [M, N] with contiguous rows (any row stride) to write into."""
    residuals = tuple(r for r in residuals if r is not None)
    if x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16:
        from ..csrc import gemm_tc
        if gemm_tc.takes(x, weight):
            if activation in TENSOR_CORE_ACTIVATIONS:
                return gemm_tc.linear(x, weight, bias, activation, residuals, out_dtype, out)
            if not residuals:       # an activation that the tensor-core epilogue does not offer: a kernel of its own behind it
                return ops.activate(gemm_tc.linear(x, weight, bias, None, (), out_dtype, out), activation)
    if x.dtype == torch.float32 and out_dtype in (None, torch.float32) and x.dim() == 2 and x.shape[0] >= SPLIT_ROWS \
            and x.shape[1] >= SPLIT_PRODUCTS and ops.split_takes(x, weight, out):
        own = activation in OWN_KERNEL_ACTIVATIONS and not residuals
        y = ops.linear_split(x, weight, bias, None if own else activation, residuals, out)
        return ops.activate(y, activation) if own else y
    if activation in OWN_KERNEL_ACTIVATIONS and not residuals:
        return ops.activate(ops.linear_simt(x, weight, bias, None, (), out_dtype, out), activation)
    return ops.linear_simt(x, weight, bias, activation, residuals, out_dtype, out)


def shared_sms():
    """A context in which the tensor-core products of few tokens leave half of each SM to another product."""
    from ..csrc import gemm_tc
    return gemm_tc.shared_sms()


class beside_main_stream:
    """Enter a second CUDA stream that has waited for everything the current stream holds so far; products
    inside use a scratch of their own.  `join()` afterwards makes the current stream wait for the second."""

    def __init__(self, side: "torch.cuda.Stream", device):
        self.side, self.device = side, device

    def __enter__(self):
        from ..csrc import gemm_tc
        self.main = torch.cuda.current_stream(self.device)
        forked = torch.cuda.Event()
        forked.record(self.main)
        self.ctx = torch.cuda.stream(self.side)
        self.ctx.__enter__()
        self.side.wait_event(forked)
        self.scratch = gemm_tc.second_scratch()
        self.scratch.__enter__()
        return self

    def __exit__(self, *exc):
        self.scratch.__exit__(*exc)
        self.done = torch.cuda.Event()
        self.done.record(self.side)
        self.ctx.__exit__(*exc)

    def join(self):
        self.main.wait_event(self.done)
