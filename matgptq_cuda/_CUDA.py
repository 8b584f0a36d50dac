"""Stand-in for the reference's pybind extension ``matgptq_cuda._CUDA`` (``csrc/bindings.cpp:214-218``):
the same three callables with the same positional arguments, served by the registered operators.  As with the pybind
functions, autograd does not see the call: a result never requires a gradient."""
import torch

from matgptq_b200 import ops as _ops


@torch.no_grad()
def pack_matgptq_qweights(qweights, n_out_features, n_in_features, bitwidth, group_size, feature_flag):
    """``csrc/bindings.cpp:43-84``."""
    return _ops.pack_matgptq_qweights(qweights, n_out_features, n_in_features, bitwidth, group_size, feature_flag)


@torch.no_grad()
def reorder_matgptq_scales(scales, m, n, group_size):
    """``csrc/bindings.cpp:86-142``."""
    return _ops.reorder_matgptq_scales(scales, m, n, group_size)


@torch.no_grad()
def matmul_matgptq(input, matgptq_weights, matgptq_scales, n_out_features, n_in_features, bitwidth, group_size,
                   feature_flag):
    """``csrc/bindings.cpp:146-191``."""
    return _ops.matmul_matgptq(input, matgptq_weights, matgptq_scales, n_out_features, n_in_features, bitwidth, group_size,
                               feature_flag)
