"""The three operators of the reference's ``matgptq_cuda`` package, on the B200 library.

Same names, schemas and argument meaning as ``inference_lib/matgptq_cuda/__init__.py:5-63``
(Python custom ops) and ``csrc/bindings.cpp:43-191,197-207`` (checks, allocation,
stream): ``torch.ops.matgptq_cuda.{pack_matgptq_qweights, reorder_matgptq_scales,
matmul_matgptq}``.  They are registered and checked in C++ (``csrc/torch_ops.cpp``, the module
``_torch_ops``), because a call with few rows costs more on the host than on the GPU; PyTorch supplies
device memory and the current stream, and the work is done by ``libmatgptq_b200.so`` through its C ABI.
Additions sit beside them: ``slice_pack_matgptq_qweights`` (slicing fused into packing),
``matmul_matgptq_out``, ``matmul_matgptq_grouped``, ``matmul_matgptq_zeros`` and
``dequantize_matgptq`` (dense weights for checks).
"""
from __future__ import annotations

import torch

from . import _native

_lib = _native.load()
_ext = _native.load_torch_ops()  # registers torch.ops.matgptq_cuda.*

_ops = torch.ops.matgptq_cuda


def pack_matgptq_qweights(qweights: torch.Tensor, n_out_features: int, n_in_features: int, bitwidth: int, group_size: int,
                          feature_flag: int) -> torch.Tensor:
    """Pack already-sliced b-bit codes ``[N, K]`` (uint8, CPU or CUDA) into the 1-D
    uint32 CUDA tensor of ``b*N*K/32`` words that ``matmul_matgptq`` reads."""
    return _ops.pack_matgptq_qweights(qweights, n_out_features, n_in_features, bitwidth, group_size, feature_flag)


@torch.library.register_fake("matgptq_cuda::pack_matgptq_qweights")
def _pack_fake(qweights, n_out_features, n_in_features, bitwidth, group_size, feature_flag):
    return qweights.new_empty((bitwidth * n_out_features * n_in_features // 32,), dtype=torch.uint32)


def slice_pack_matgptq_qweights(qweights: torch.Tensor, n_out_features: int, n_in_features: int, master_bitwidth: int,
                                bitwidth: int, group_size: int, feature_flag: int) -> torch.Tensor:
    """``pack_matgptq_qweights(matryoshka_slice(qweights, master_bitwidth, bitwidth), ...)`` in one
    pass over the master codes (the two steps of ``vllm_matgptq.py:152-166``)."""
    return _ops.slice_pack_matgptq_qweights(qweights, n_out_features, n_in_features, master_bitwidth, bitwidth, group_size,
                                            feature_flag)


@torch.library.register_fake("matgptq_cuda::slice_pack_matgptq_qweights")
def _slice_pack_fake(qweights, n_out_features, n_in_features, master_bitwidth, bitwidth, group_size, feature_flag):
    return qweights.new_empty((bitwidth * n_out_features * n_in_features // 32,), dtype=torch.uint32)


def reorder_matgptq_scales(scales: torch.Tensor, m: int, n: int, group_size: int) -> torch.Tensor:
    """Reorder scales ``[N, G]`` for the kernels; same shape and dtype, on CUDA
    (``m`` = out features, ``n`` = in features, as in the reference)."""
    return _ops.reorder_matgptq_scales(scales, m, n, group_size)


@torch.library.register_fake("matgptq_cuda::reorder_matgptq_scales")
def _reorder_fake(scales, m, n, group_size):
    return torch.empty_like(scales)


def matmul_matgptq(input: torch.Tensor, matgptq_weights: torch.Tensor, matgptq_scales: torch.Tensor, n_out_features: int,
                   n_in_features: int, bitwidth: int, group_size: int, feature_flag: int) -> torch.Tensor:
    """``y[M, N] = x[M, K] @ Wdq.T`` for packed b-bit weights; ``M = input.size(-2)``.
    Output is float16, or bfloat16 when ``feature_flag & 2``."""
    return _ops.matmul_matgptq(input, matgptq_weights, matgptq_scales, n_out_features, n_in_features, bitwidth, group_size,
                               feature_flag)


@torch.library.register_fake("matgptq_cuda::matmul_matgptq")
def _matmul_fake(input, matgptq_weights, matgptq_scales, n_out_features, n_in_features, bitwidth, group_size,
                 feature_flag):
    # inference_lib/matgptq_cuda/__init__.py:49-63
    return input.new_empty((input.shape[-2], n_out_features),
                           dtype=torch.bfloat16 if feature_flag & 2 else torch.float16)


def matmul_matgptq_out(input: torch.Tensor, matgptq_weights: torch.Tensor, matgptq_scales: torch.Tensor, n_out_features: int,
                       n_in_features: int, bitwidth: int, group_size: int, feature_flag: int, out: torch.Tensor) -> None:
    """``matmul_matgptq`` into a tensor the caller owns (``out [M, N]``, contiguous, float16 or bfloat16 like the
    input): nothing is allocated, which is what callers that gather several layers' outputs in one buffer, or that
    capture the call in a CUDA graph with their own memory plan, want.  The reference's operator only has the
    allocating form (csrc/bindings.cpp:158-201)."""
    return _ops.matmul_matgptq_out(input, matgptq_weights, matgptq_scales, n_out_features, n_in_features, bitwidth,
                                   group_size, feature_flag, out)


@torch.library.register_fake("matgptq_cuda::matmul_matgptq_out")
def _matmul_out_fake(input, matgptq_weights, matgptq_scales, n_out_features, n_in_features, bitwidth, group_size,
                     feature_flag, out):
    return None


def matmul_matgptq_grouped_raw(x: torch.Tensor, packed, scales, n_out, n_in: int, bitwidths, group_size: int,
                               flags: int, out: torch.Tensor | None = None,
                               workspace: torch.Tensor | None = None) -> torch.Tensor:
    """The C-ABI grouped product without checks: segment ``i`` (``packed[i]``, ``scales[i]``, ``n_out[i]`` rows at
    ``bitwidths[i]`` bits) fills its column block of ``out [M, sum(n_out)]``.  One kernel launch up to 16 rows."""
    if out is None and workspace is None:
        return _ext.grouped_raw(x, list(packed), list(scales), [int(n) for n in n_out], n_in, [int(b) for b in bitwidths],
                                group_size, flags)
    batch = x.size(-2)
    total = int(sum(n_out))
    if out is None:
        out = torch.empty((batch, total), dtype=x.dtype, device=x.device)
    segs = (_native.Segment * len(packed))()
    need = 0
    for i, (w, s, n, b) in enumerate(zip(packed, scales, n_out, bitwidths)):
        segs[i] = _native.Segment(w.data_ptr(), s.data_ptr(), int(n), int(b))
        if batch >= 32 and workspace is None and flags & _native.FLAG_SCRATCH_REDUCE:
            need = max(need, _lib.matgptq_b200_matmul_workspace_bytes(int(n), n_in, batch))
    if need > 0:
        workspace = torch.empty(need, dtype=torch.uint8, device=x.device)
    st = _lib.matgptq_b200_matmul_grouped(segs, len(packed), group_size, n_in, batch, x.data_ptr(), out.data_ptr(),
                                          torch.cuda.current_stream(x.device).cuda_stream, flags,
                                          workspace.data_ptr() if workspace is not None else None,
                                          workspace.numel() if workspace is not None else 0)
    _native.check(st, "matgptq_b200_matmul_grouped")
    return out


def matmul_matgptq_grouped(input: torch.Tensor, matgptq_weights: list[torch.Tensor], matgptq_scales: list[torch.Tensor],
                           n_out_features: list[int], n_in_features: int, bitwidths: list[int], group_size: int,
                           feature_flag: int) -> torch.Tensor:
    """Addition: ``matmul_matgptq`` for a fused layer whose output partitions have their own bitwidths
    (``vllm_matgptq.py:113-121`` fuses q/k/v and gate/up; ``evo_quant_search.py:659-671`` gives each checkpoint
    layer its own bitwidth).  ``y[M, sum N_i] = x[M, K] @ cat(Wdq_i).T`` in one launch up to 16 rows;
    the reference's operator takes a single bitwidth per call."""
    return _ops.matmul_matgptq_grouped(input, matgptq_weights, matgptq_scales, n_out_features, n_in_features, bitwidths,
                                       group_size, feature_flag)


@torch.library.register_fake("matgptq_cuda::matmul_matgptq_grouped")
def _matmul_grouped_fake(input, matgptq_weights, matgptq_scales, n_out_features, n_in_features, bitwidths, group_size,
                         feature_flag):
    return input.new_empty((input.shape[-2], sum(n_out_features)),
                           dtype=torch.bfloat16 if feature_flag & 2 else torch.float16)


def matmul_matgptq_zeros(input: torch.Tensor, matgptq_weights: torch.Tensor, matgptq_scales: torch.Tensor,
                         matgptq_zeros: torch.Tensor, n_out_features: int, n_in_features: int, bitwidth: int, group_size: int,
                         feature_flag: int) -> torch.Tensor:
    """Extension: ``matmul_matgptq`` with per-group zero points, ``Wdq = s * (code * 2^(8-b) - zero)`` as in the
    reference's ``dequantize`` (``src/quant_utils_matgpqt.py:19-22``).  ``matgptq_zeros`` are the zero points in
    master (8-bit) units, in the dtype of the scales, passed through ``reorder_matgptq_scales`` like the scales.
    The reference's operator has no such argument (its zero point is the implicit ``2^(b-1)``)."""
    return _ops.matmul_matgptq_zeros(input, matgptq_weights, matgptq_scales, matgptq_zeros, n_out_features, n_in_features,
                                     bitwidth, group_size, feature_flag)


@torch.library.register_fake("matgptq_cuda::matmul_matgptq_zeros")
def _matmul_zeros_fake(input, matgptq_weights, matgptq_scales, matgptq_zeros, n_out_features, n_in_features, bitwidth,
                       group_size, feature_flag):
    return input.new_empty((input.shape[-2], n_out_features),
                           dtype=torch.bfloat16 if feature_flag & 2 else torch.float16)


def dequantize_matgptq(matgptq_weights: torch.Tensor, matgptq_scales: torch.Tensor, n_out_features: int, n_in_features: int,
                       bitwidth: int, group_size: int, feature_flag: int) -> torch.Tensor:
    """Dense ``W[N, K]`` (fp16/bf16) from packed weights and reordered scales, bit-exact with the
    reference's ``dequantize`` for zero point 128."""
    return _ops.dequantize_matgptq(matgptq_weights, matgptq_scales, n_out_features, n_in_features, bitwidth, group_size,
                                   feature_flag)


@torch.library.register_fake("matgptq_cuda::dequantize_matgptq")
def _dequant_fake(matgptq_weights, matgptq_scales, n_out_features, n_in_features, bitwidth, group_size, feature_flag):
    return matgptq_scales.new_empty((n_out_features, n_in_features))


def matmul_matgptq_raw(x: torch.Tensor, packed: torch.Tensor, scales: torch.Tensor, n_out: int, n_in: int,
                       bitwidth: int, group_size: int, flags: int, out: torch.Tensor | None = None,
                       warps_per_cta: int = 0, split_k: int = 0, path: int = 0,
                       workspace: torch.Tensor | None = None) -> torch.Tensor:
    """The C-ABI matmul without the dispatcher around it: no argument checks beyond the library's own,
    optional preallocated output and scratch, forced path (1 GEMV, 2 tensor cores) and launch shape.
    Used by the decode loop, the benchmarks and the tests."""
    if not (warps_per_cta or split_k or path) and workspace is None:
        return _ext.matmul_raw(x, packed, scales, n_out, n_in, bitwidth, group_size, flags, out)
    batch = x.size(-2)
    if out is None:
        out = torch.empty((batch, n_out), dtype=x.dtype, device=x.device)
    stream = torch.cuda.current_stream(x.device).cuda_stream
    if warps_per_cta:
        st = _lib.matgptq_b200_matmul_tuned(bitwidth, group_size, n_out, n_in, batch, packed.data_ptr(),
                                            scales.data_ptr(), x.data_ptr(), out.data_ptr(), stream, flags,
                                            warps_per_cta, split_k)
    else:
        if workspace is None and path != 1 and flags & _native.FLAG_SCRATCH_REDUCE:  # scratch only where it is used
            if path == 2 and split_k > 1:
                need = split_k * batch * n_out * 4
            elif path == 2:
                need = _lib.matgptq_b200_matmul_workspace_bytes(n_out, n_in, max(batch, 64))
            else:
                need = _lib.matgptq_b200_matmul_workspace_bytes(n_out, n_in, batch)
            if need > 0:
                workspace = torch.empty(need, dtype=torch.uint8, device=x.device)
        st = _lib.matgptq_b200_matmul_ws(bitwidth, group_size, n_out, n_in, batch, packed.data_ptr(),
                                         scales.data_ptr(), x.data_ptr(), out.data_ptr(), stream, flags,
                                         workspace.data_ptr() if workspace is not None else None,
                                         workspace.numel() if workspace is not None else 0, path, split_k)
    _native.check(st, "matgptq_b200_matmul")
    return out
