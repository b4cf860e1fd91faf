"""x . W^T for the parts, by storage dtype.

float32: the package's own kernels, true 32-bit: up to F32_CORE_ROWS rows and narrow products on the float32 cores, the others
on the tensor cores with every operand as three bfloat16.  Each of the two gives a row the same bits whatever else is in the
batch, but not each other's: a row's last bits change between 32 and 33 rows and wherever else the kernel does.
bfloat16: the tensor-core kernels of this package where they take the shape,
else cuBLAS through ``torch.nn.functional.linear``, which is what the
reference's engine calls for every projection (tinyvllm/layers.py:84-85).
"""

from __future__ import annotations

import functools
import os

import torch

from . import kernels


def linear(x: torch.Tensor, weight: torch.Tensor, *, out_dtype: torch.dtype | None = None,
           out: torch.Tensor | None = None, weight_constant: bool = False) -> torch.Tensor:
    """x [m, k] times weight [n, k] transposed; the result has ``out_dtype``
    (default: the dtype of x).  ``weight_constant``: nothing in flight on the stream writes the weight (a model's, loaded
    long ago), so that float32 products may read it while the kernel before them still runs.  (bfloat16 products of few
    rows always do.)"""
    if not x.is_cuda:
        raise kernels.KernelError("linear runs on CUDA tensors only; there is no CPU path")
    out_dtype = out_dtype or x.dtype
    if x.dtype == torch.float32:
        if out_dtype != torch.float32:
            raise kernels.KernelError("a float32 product has a float32 result")
        return _linear_f32(x, weight, out, weight_constant)
    from . import gemm

    return gemm.linear_bf16(x, weight, out_dtype=out_dtype, out=out)


# Rows up to which a float32 product stays on the float32 cores: the tensor-core kernel takes 25 to 28 us for a layer's
# products at any number of rows up to 128 (a CTA walks 1,024 k in 16 steps of 1.2 us), the float32 cores 16 to 24 us
# for 32 rows, 29 to 42 us for 48.
F32_CORE_ROWS = 32
# Smallest k of the tensor cores.  Their error against 64 bits is larger below (operands of either sign, k = 4 / 8 / 16: 4.9e-8,
# 4.9e-8, 5.0e-8; float32 cores 4.1e-8, 4.8e-8, 6.0e-8).
F32_TENSOR_K = 16


@functools.lru_cache(maxsize=4096)
def _tensor_cores_are_quicker(rows: int, columns: int, k: int) -> bool:
    """Whether the tensor cores take a float32 product of more than F32_CORE_ROWS rows, by the two kernels' estimates.  The
    float32 cores are quicker where one round of their tiles holds all of a narrow or short product: splitting x, a launch
    more, and columns up to 128 are then not paid back.  Measured (us, float32 cores / tensor cores): 301 x 512 x 64 5.3 /
    6.3, 8,192 x 128 x 64 7.6 / 15.2, 2,048 x 64 x 2,048 29 / 34, 8,192 x 64 x 4,096 127 / 176; but 301 x 64 x 512 27 /
    15, 677 x 128 x 1,024 28.7 / 27.0, 2,048 x 256 x 2,048 76 / 35."""
    return k >= F32_TENSOR_K and kernels.gemm_f32_tc_us(rows, columns, k) < kernels.gemm_f32_us(rows, columns, k)


def _linear_f32(x: torch.Tensor, weight: torch.Tensor, out: torch.Tensor | None, weight_constant: bool) -> torch.Tensor:
    # (an ``out`` that is larger than the result, or of another type, is written by the float32 cores' kernels alone)
    if (x.dim() == 2 and x.shape[0] > F32_CORE_ROWS and kernels.gemm_f32_tc_takes(x, weight)
            and (out is None or (out.dtype == torch.float32 and out.shape == (x.shape[0], weight.shape[0])))
            and _tensor_cores_are_quicker(x.shape[0], weight.shape[0], x.shape[1])):
        return kernels.gemm_f32_tc(x, weight, out=out, weight_constant=weight_constant)
    return kernels.gemm_nt_simt(x, weight, out=out, weight_constant=weight_constant)


def linear_silu(x: torch.Tensor, gate_up_weight: torch.Tensor, *, weight_constant: bool = False) -> torch.Tensor:
    """round(round(silu(x . gate^T)) * (x . up^T)) for a packed [gate | up] weight, [m, inter].  ``weight_constant``: as in
    :func:`linear`."""
    if not x.is_cuda:
        raise kernels.KernelError("linear_silu runs on CUDA tensors only; there is no CPU path")
    if x.dtype == torch.float32:
        return kernels.silu_mul(_linear_f32(x, gate_up_weight, None, weight_constant))
    from . import gemm

    return gemm.linear_silu_bf16(x, gate_up_weight)


# Every CTA of the fused kernel reads all rows of the input to normalise them for itself; beyond
# a few rows those reads cost more (in L2 bandwidth) than the separate norm kernel they replace.
FUSED_NORM_MAX_ROWS = int(os.environ.get("TINYVLLM_B200_FUSED_NORM_ROWS", "2"))


# TINYVLLM_B200_STREAM_ADD=0: output projections never add to the stream themselves (the norm kernel
# runs between every two products), for comparison
STREAM_ADD = os.environ.get("TINYVLLM_B200_STREAM_ADD", "1") != "0"


def linear_into_stream(x: torch.Tensor, weight: torch.Tensor, stream: torch.Tensor, *, weight_constant: bool = False):
    """A part's output projection, added to the residual stream where that saves a kernel.  ``weight_constant``: as in
    :func:`linear`.

    Returns (None, stream + linear(x, weight)) when the product's kernel does the addition on its
    way out (small bfloat16 batches): the new stream then carries ``row_squares``, the sums of
    squares of its rows tile by tile, with which :func:`linear_norm` applies the next pre-norm
    inside the next product, so that no norm kernel runs between the two (there the norm weight
    multiplies the stream before the product and the inverse RMS the sums after it: one rounding
    where the norm kernel has two).  Otherwise
    (linear(x, weight), stream), and the next norm adds the two as usual."""
    from . import gemm

    if (STREAM_ADD and x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and stream is not None
            and stream.dtype == torch.bfloat16 and stream.is_contiguous() and gemm.small(x, weight)
            and stream.shape == (x.shape[0], weight.shape[0])):
        summed, squares = kernels.gemm_small_m(x, weight, kernels.GEMM_BF16, add_stream=stream,
                                               prefetch=gemm.next_weight(weight))
        summed.row_squares = squares
        return None, summed
    return linear(x, weight, weight_constant=weight_constant), stream


def linear_norm(hidden: torch.Tensor | None, residual: torch.Tensor | None, norm, weight: torch.Tensor, *,
                silu: bool = False, weight_constant: bool = False):
    """(linear(norm(hidden + residual), weight), hidden + residual): a pre-norm and the
    projection behind it as one operation.  ``norm`` is a norm part (``weight``, ``eps``,
    ``forward``, ``add``).  Without a residual the stream is ``hidden`` itself; without
    ``hidden`` (None) the residual holds the sum already (:func:`linear_into_stream`).  ``silu``
    applies SiLU(gate) * up to a packed [gate | up] weight.  Small bfloat16 batches run as
    one kernel; everything else as the norm kernel and the product.  ``weight_constant``: as in
    :func:`linear`."""
    from . import gemm

    if hidden is None:
        squares = getattr(residual, "row_squares", None)
        if (squares is not None and weight.dtype == torch.bfloat16 and getattr(norm, "folds_into_product", False)
                and gemm.small(residual, weight) and residual.is_contiguous()
                and norm.weight.data_ptr() % 16 == 0):
            mode = kernels.GEMM_SILU if silu else kernels.GEMM_BF16
            out = kernels.gemm_small_m(residual, weight, mode, norm_weight=norm.weight, eps=norm.eps,
                                       row_squares=squares, prefetch=gemm.next_weight(weight))
            return out, residual
        x = norm.forward(residual)
        return (linear_silu if silu else linear)(x, weight, weight_constant=weight_constant), residual
    if (hidden.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and hidden.is_contiguous()
            and getattr(norm, "folds_into_product", False) and gemm.small(hidden, weight)
            and hidden.shape[0] <= FUSED_NORM_MAX_ROWS
            and kernels.gemm_small_m_takes_norm(hidden.shape[0], hidden.shape[1])):
        mode = kernels.GEMM_SILU if silu else kernels.GEMM_BF16
        out, stream = kernels.gemm_small_m(hidden, weight, mode, norm_weight=norm.weight,
                                           residual=residual, eps=norm.eps,
                                           prefetch=gemm.next_weight(weight))
        return out, (hidden if residual is None else stream)
    if residual is None:
        x, stream = norm.forward(hidden), hidden
    else:
        x, stream = norm.add(hidden, residual)
    return (linear_silu if silu else linear)(x, weight, weight_constant=weight_constant), stream
