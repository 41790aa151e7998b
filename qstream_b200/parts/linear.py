"""The matrix product y = act(x W^T + b) + residuals, and the choice of its kernel.

bfloat16 activations with a bfloat16 matrix run on the tensor cores (tcgen05, fed by
TMA, 32-bit accumulation).  float32 activations with a float32 matrix run there too, every
number as three bfloat16 terms and the sums rounded in 32 bits outside the unit, where a result is the
sum of 256 products or more and rows come in 16-byte pieces; everything else (short sums, mixed types)
runs on the CUDA cores in true 32-bit.

A row's result does not depend on the contents of the other rows.  Neither does it depend on their number in
the float32 engine, where the matrix alone decides the kernel and the order of the sums; the bfloat16
products change their order between up to 128 rows and more (and with the number beyond), by rounding.
"""
from __future__ import annotations

import torch

from ..csrc import ops

TENSOR_CORE_ACTIVATIONS = (None, "none", "gelu_new", "gelu")
# float32: from how many products per result on the tensor cores serve, whatever the number of rows, so that a row's result is the same bits in any
# batch.  Microseconds, CUDA cores | tensor cores (caches flushed, launches included): 1, 16, 17, 64 and 700 rows, 6144 x 2048: 29 | 31, 31 | 33,
# 49 | 33, 57 | 35, 410 | 115; 2048 x 2048: 23 | 23, 23 | 25, 25 | 25, 33 | 31, 187 | 51; 2048 x 8192: 35 | 37, 37 | 39, 53 | 39, 70 | 41, 551 | 143;
# 32000 x 2048: 94 | 102, 100 | 109, 176 | 111, 244 | 111, 2211 | 520; 64 x 2048: 18 | 15, 18 | 16, 18 | 16, 18 | 16, 27 | 29; 128 x 256: 20 | 14, 21 | 14,
# 20 | 14, 23 | 14, 22 | 16.
SPLIT_PRODUCTS = 256
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
    if x.dtype == torch.float32 and out_dtype in (None, torch.float32) and x.dim() == 2 and x.shape[1] >= SPLIT_PRODUCTS \
            and ops.split_takes(x, weight, out):
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
