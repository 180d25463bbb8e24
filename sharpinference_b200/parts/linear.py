"""Matrix products of the parts: ``y = a . W^T`` with the weight stored ``[out, in]``.

Which routine runs is decided by the weight's dtype and the number of rows, not by a global mode:

* float32 weight: the CUDA-core kernel with float32 accumulation (``gemm_generic.cu``), the
  product of the true 32-bit path; no tensor cores and no reduced-precision mode are involved.
* bfloat16 weight: a tensor-core product with float32 accumulation and float32 output.  The dense ones go to
  the vendor library through ``torch.mm``, which is where the reference uses a library too (cublasGemmEx for
  batched projections, src/SharpInference.Cuda/CudaBackend.cs:2083-2117).  With few rows (decode), where the
  reference runs matvec kernels of its own (llm_matvec_*, src/SharpInference.Cuda/CudaTextKernels.cs:1325),
  they can run the engine's weight-streaming kernel instead (``stream_rows``; ``dense_rows.cu``: the weight is
  read once, rows dealt evenly over the SMs, bias, add-in or SwiGLU in its epilogue).  In an engine's steps small products
  run there by default (:func:`engine_step`); for large ones it is the faster kernel alone (see DEFAULT_STREAM_ROWS) but
  not inside a decode step, so they stay with the library.
* sizes neither takes (an inner size that is no multiple of 8) use the CUDA-core kernel.

The grouped (per-expert) product has no library counterpart and always runs our own kernels.
"""
from __future__ import annotations

import contextlib
import threading
from typing import Optional

import torch

from ..kernels import ops


# Rows up to which a bfloat16 product runs on the weight-streaming kernel by default: none.  Measured on B200
# at Scout sizes, microseconds at 1 to 8 rows, own kernel / library, alone and between two other kernels of a
# captured graph: qkv 7168 x 5120 12.8 / 14.4, o 5120 x 5120 9.9 / 11.8, shared down 5120 x 8192 14.8 / 17.5,
# shared gate|up with SwiGLU 27.0 / 29.9 (library product plus the SwiGLU kernel).  In a decode step of 8 layers
# the own kernel on every product gives 593 against 614 tokens a second at batch 1 and 2198 against 2221 at
# batch 8: it deals its rows over exactly as many CTAs as fit the SMs at once, with all their registers, so a
# kernel of another stream (the router beside the shared expert) or a block of a neighbour that is still or
# already there delays one of its CTAs by up to the whole product.
DEFAULT_STREAM_ROWS = 0
# Small products (:func:`engine_step`): up to this many rows against a weight of up to this many elements, the weight-streaming kernel,
# which may start while the kernel before it ends (the library's kernels take 8 to 13 us where reading the weight takes 1 to 3).
# Library / own kernel between two other kernels of a captured graph, us, weights from memory, at 1, 8 and 16 rows: 1024 x 1024
# 5.7 / 3.9, 6.1 / 4.5, 6.1 / 4.5; 2048 x 2048 9.3 / 5.3, 8.2 / 5.7, 7.1 / 6.3; 2048 x 4096 13.3 / 6.7, 12.1 / 7.4, 9.8 / 9.0; 4096 x
# 4096 14.5 / 10.0, 13.2 / 10.2, 10.9 / 10.8; 8192 x 2048 10.0 / 9.2, 9.5 / 9.6, 9.9 / 10.1; 16384 x 2048 15.0 / 15.0, 14.7 / 15.3,
# 14.9 / 17.1; 5120 x 5120 13.5 / 12.6, 13.5 / 12.8, 14.8 / 14.2.
SMALL_PRODUCTS = ((8, 1 << 24), (16, 1 << 23))


class _Step(threading.local):
    small_products = False


_step = _Step()


@contextlib.contextmanager
def engine_step(small_products: bool):
    """While an engine launches a step in this thread: whether small products run on the weight-streaming kernel, which may
    read a weight before the kernels in front of it have ended.  A step begins behind a copy, which waits for all that the
    stream was given before, so whatever a program wrote into its weights by then is there; outside of a step nothing is known
    of what wrote them last, and the same :class:`Linear` goes to the library."""
    before, _step.small_products = _step.small_products, small_products
    try:
        yield
    finally:
        _step.small_products = before


class Linear:
    """A weight ``[out, in]``, an optional bias ``[out]`` (float32) and the product with them.  Output is
    float32 ``[M, out]``.  The reference adds a projection's bias where a model stores one
    (src/SharpInference.Core/ModelGraph.cs:269-270 probes for it)."""

    def __init__(self, weight: torch.Tensor, name: str = "", stream_rows: int = DEFAULT_STREAM_ROWS,
                 bias: Optional[torch.Tensor] = None, split_add_rows: int = 0):
        if weight.dim() != 2:
            raise ValueError(f"linear weight '{name}' must be 2-D, found shape {tuple(weight.shape)}")
        if bias is not None and tuple(bias.shape) != (weight.shape[0],):
            raise ValueError(f"bias of '{name}' has shape {tuple(bias.shape)}, expected ({weight.shape[0]},)")
        self.weight = weight
        self.bias = bias
        self.name = name
        self.out_features, self.in_features = weight.shape
        self._use_library = (weight.dtype == torch.bfloat16 and self.in_features % 8 == 0)
        self._wt = weight.t() if self._use_library else None
        # Up to this many rows (at most ops.DENSE_ROWS_MAX) the product runs on the weight-streaming kernel
        # instead of the library; 0: the library at every size.
        self.stream_rows = stream_rows
        # Whether small products (SMALL_PRODUCTS) run there outside of an engine's steps too: for a program whose stream has waited
        # for what wrote the weight since (see engine_step).
        self.stream_small = False
        # Up to this many rows an add-in (``accumulate``) runs on the grouped tensor-core kernel with one group
        # and K cut over CTAs: small CTAs that add with reductions and run well beside other kernels.
        self.split_add_rows = split_add_rows

    def __call__(self, a: torch.Tensor, out: Optional[torch.Tensor] = None, accumulate: bool = False) -> torch.Tensor:
        """``a . W^T`` into ``out``, or added to it (``accumulate``).  Where :meth:`adds_with_reductions` says so
        the add-in is done with reductions, so that another kernel may add into the same ``out`` at the same
        time; otherwise it is the product followed by an addition."""
        if accumulate:
            if out is None:
                raise ValueError("accumulate needs an output to add to")
            if self.adds_with_reductions(a):
                if a.shape[0] <= self.split_add_rows:
                    return ops.tc_dense(a, self.weight, out=out, accumulate=True)
                return ops.dense_rows(a, self.weight, out=out, accumulate=True)
            return out.add_(self(a))
        w = self.weight
        if w.dtype == torch.float32:
            if a.dtype != torch.float32:
                a = a.to(torch.float32)
            return ops.gemm_nt(a, w, out=out, bias=self.bias)
        if self._use_library and a.dtype == torch.bfloat16:
            if self.streams(a) and (out is None or out.is_contiguous()):
                return ops.dense_rows(a, w, out=out, bias=self.bias, early=self.small(a.shape[0]))
            if out is not None:
                y = torch.mm(a, self._wt, out_dtype=torch.float32, out=out)
            else:
                y = torch.mm(a, self._wt, out_dtype=torch.float32)
            return ops.add_bias(y, self.bias) if self.bias is not None else y
        return ops.gemm_nt(a, w, out=out, bias=self.bias)

    def streams(self, a: torch.Tensor, fused: bool = False) -> bool:
        """Whether this product of ``a`` runs on the weight-streaming kernel.  ``fused``: it would apply SwiGLU there."""
        if not self._use_library or a.dtype != torch.bfloat16:
            return False
        return (a.shape[0] <= min(self.stream_rows, ops.DENSE_ROWS_MAX)
                or (self.small(a.shape[0], fused) and a.is_contiguous() and self.weight.is_contiguous()
                    and (a.data_ptr() | self.weight.data_ptr()) % 16 == 0))

    def small(self, rows: int, fused: bool = False) -> bool:
        """Whether a product of this many rows is a small one that runs on the weight-streaming kernel.  With SwiGLU in its epilogue,
        which saves a kernel of 2 to 3 us, weights may have twice as many elements."""
        return (self.stream_small or _step.small_products) and any(0 < rows <= most and self.weight.numel() <= size << fused for most, size in SMALL_PRODUCTS)

    def adds_with_reductions(self, a: torch.Tensor) -> bool:
        """Whether ``accumulate`` adds this product of ``a`` into the output element by element with reductions
        (one of the engine's own kernels) rather than as a product followed by an addition."""
        return (self._use_library and self.bias is None and a.dtype == torch.bfloat16
                and a.shape[0] <= max(self.split_add_rows, min(self.stream_rows, ops.DENSE_ROWS_MAX)))


class GroupedLinear:
    """Per-expert weights ``[E, out, in]``; rows arrive sorted by expert."""

    def __init__(self, weight: torch.Tensor, name: str = ""):
        if weight.dim() != 3:
            raise ValueError(f"grouped weight '{name}' must be [E, out, in], found shape {tuple(weight.shape)}")
        self.weight = weight
        self.name = name
        self.num_groups, self.out_features, self.in_features = weight.shape

    def __call__(self, a: torch.Tensor, group_offsets: torch.Tensor, *, rows: int,
                 a_rows: Optional[torch.Tensor] = None, out_rows: Optional[torch.Tensor] = None,
                 out: Optional[torch.Tensor] = None, accumulate: bool = False) -> torch.Tensor:
        if self.weight.dtype == torch.float32 and a.dtype != torch.float32:
            a = a.to(torch.float32)
        return ops.gemm_nt(a, self.weight, out=out, group_offsets=group_offsets, a_rows=a_rows, out_rows=out_rows,
                           rows=rows, accumulate=accumulate)

    def per_group_minor(self, a: torch.Tensor, rows_per_group: int, out: torch.Tensor) -> bool:
        """:meth:`per_group` in bfloat16 with the groups minor, ``out [rows_per_group, groups, ld]``, where the tensor-core product
        takes it (more than 16 rows in all: with fewer it cuts K over CTAs); False: nothing was written.  ``a`` as there, or with the
        groups minor, ``[rows_per_group, groups, ld]``, of which the first ``in`` columns are read."""
        if not (self.weight.dtype == torch.bfloat16 == a.dtype and self.in_features % 8 == 0 and self.num_groups * rows_per_group > 16
                and (a.dim() == 2 or a.shape[2] % 8 == 0)):
            return False
        ops.tc_per_head(a, self.weight, rows_per_group, out)
        return True

    def per_group(self, a: torch.Tensor, rows_per_group: int) -> torch.Tensor:
        """The product for ``a [groups * rows_per_group, in]`` that holds every group's rows one group after the
        other, the same number each (one weight a head: heads are the groups): float32 ``[groups * rows_per_group,
        out]``.  bfloat16 operands with an inner size that is a multiple of 8 run the tcgen05 grouped product,
        everything else the CUDA-core one."""
        offsets = torch.arange(0, (self.num_groups + 1) * rows_per_group, max(rows_per_group, 1), dtype=torch.int32,
                               device=a.device)
        if (self.weight.dtype == torch.bfloat16 and a.dtype == torch.bfloat16 and self.in_features % 8 == 0):
            return ops.tc_grouped_gemm(a, self.weight, offsets, mode=ops.TC_MODE_STORE)
        return self(a, offsets, rows=a.shape[0])
