"""MatGPTQLinear's C++ host path: the same rows as the operator computes, whatever form the input comes in, and the
dispatcher still sees the call when something listens to it."""
import ctypes
import subprocess

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode


def _layer(cuda, n=64, k=256):
    from matgptq_b200 import synth
    from matgptq_b200.matgptq_linear import MatGPTQLinear
    w = synth.make_layer(n, k, 128, seed=2, device=cuda)
    return MatGPTQLinear.from_master(w.qweight, w.scales, 8, 4, 128)


def _op(layer, x2):
    return torch.ops.matgptq_cuda.matmul_matgptq(x2, layer.matgptq_qweight, layer.matgptq_scales, layer.n_out_features,
                                                 layer.n_in_features, layer.bitwidth, layer.group_size, 1)


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["rows", "batch_tokens", "four_dims", "strided", "misaligned", "empty"])
def test_forward_equals_operator(cuda, form):
    layer = _layer(cuda)
    base = torch.randn(12, 2 * layer.n_in_features + 8, dtype=torch.float16, device=cuda)
    k = layer.n_in_features
    x = {"rows": base[:, :k].contiguous(), "batch_tokens": base[:, :k].reshape(3, 4, k).contiguous(),
         "four_dims": base[:, :k].reshape(2, 3, 2, k).contiguous(), "strided": base[:, k:2 * k],
         "misaligned": base.flatten()[1:1 + 12 * k].view(12, k), "empty": base[:0, :k]}[form]
    y = layer(x)
    assert y.shape == (*x.shape[:-1], layer.n_out_features) and not y.requires_grad
    want = _op(layer, x.reshape(-1, k).clone()).view(y.shape)
    assert torch.equal(y, want)


@pytest.mark.gpu
def test_dispatch_mode_sees_the_operator(cuda):
    layer, seen = _layer(cuda), []

    class Record(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    x = torch.randn(3, layer.n_in_features, dtype=torch.float16, device=cuda)
    with Record():
        y = layer(x)
    assert any("matmul_matgptq" in s for s in seen) and torch.equal(y, layer(x))


@pytest.mark.gpu
def test_bad_inputs_raise(cuda):
    layer = _layer(cuda)
    for bad in (torch.randn(3, 128, dtype=torch.float16, device=cuda), torch.randn(3, 256, device=cuda),
                torch.randn(3, 256, dtype=torch.float16)):
        with pytest.raises(RuntimeError):
            layer(bad)


def _direct(layer, x):
    from matgptq_b200 import ops
    return ops._ext.linear_forward(x, layer.matgptq_qweight, layer.matgptq_scales, layer.n_out_features, layer.n_in_features,
                                   layer.bitwidth, layer.group_size, 1)


@pytest.mark.gpu
def test_ordinary_tensors_take_the_direct_path(cuda):
    layer = _layer(cuda)
    k = layer.n_in_features
    base = torch.randn(12, 2 * k + 8, dtype=torch.float16, device=cuda)
    grad = base[:, :k].contiguous().requires_grad_()
    with torch.inference_mode():
        inference = base[:, :k] + 0
    for x in (base[:, :k].contiguous(), base[:, k:2 * k], base.flatten()[1:1 + 12 * k].view(3, 4, k), base[:0, :k], grad,
              torch.nn.Parameter(base[:, :k].contiguous()), inference):
        y = _direct(layer, x)
        assert y is not None and torch.equal(y.view(-1, layer.n_out_features), _op(layer, x.detach().reshape(-1, k).clone()))

    class Seen(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    with Seen():
        assert _direct(layer, base[:, :k].contiguous()) is None


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["negative_bit", "conjugate_imag", "zero_tensor", "subclass"])
def test_tensors_that_are_not_their_storage_take_the_operator(cuda, form):
    layer = _layer(cuda)
    shape = (4, layer.n_in_features)
    values = torch.randn(shape, dtype=torch.float16, device=cuda)

    class Sub(torch.Tensor):
        pass

    if form == "negative_bit":
        x, same = torch._neg_view(values), -values
    elif form == "conjugate_imag":  # a plain way to the same bit
        x = torch.view_as_complex(torch.stack([values, values], -1)).conj().imag
        same = -values
    elif form == "zero_tensor":
        x = torch._efficientzerotensor(shape, dtype=torch.float16, device=cuda)
    else:
        x, same = values.as_subclass(Sub), values
    assert _direct(layer, x) is None
    if form != "zero_tensor":  # it has no memory at all; the operator says what it thinks of that
        y = layer(x)
        assert torch.equal(torch.Tensor(y) if form == "subclass" else y, _op(layer, same))


ALLOCATOR = """
#include <cuda_runtime.h>
extern "C" {
int PyGILState_Check(void);
int calls = 0, with_gil = 0;
void *take(size_t size, int, cudaStream_t) {
  ++calls;
  with_gil += PyGILState_Check() != 0;
  void *p = nullptr;
  return cudaMalloc(&p, size) == cudaSuccess ? p : nullptr;
}
void give(void *p, size_t, int, cudaStream_t) { cudaFree(p); }
}
"""


@pytest.mark.gpu
def test_memory_is_allocated_without_the_gil(cuda, tmp_path):
    # an allocation may wait for the device, and the device for a Python callback
    from matgptq_b200 import ops
    from matgptq_b200.build import _nvcc
    (tmp_path / "allocator.cpp").write_text(ALLOCATOR)
    path = str(tmp_path / "allocator.so")
    subprocess.run([_nvcc(), "-shared", "-Xcompiler", "-fPIC", "-o", path, str(tmp_path / "allocator.cpp")], check=True)
    counts = ctypes.CDLL(path)
    calls, with_gil = ctypes.c_int.in_dll(counts, "calls"), ctypes.c_int.in_dll(counts, "with_gil")
    allocator = torch.cuda.memory.CUDAPluggableAllocator(path, "take", "give")
    layer = _layer(cuda)
    args = (layer.matgptq_qweight, layer.matgptq_scales, layer.n_out_features, layer.n_in_features, layer.bitwidth, layer.group_size, 1)
    base = torch.randn(12, 2 * layer.n_in_features, dtype=torch.float16, device=cuda)
    x = base[:, :layer.n_in_features].contiguous()
    for call in (lambda: layer(x), lambda: layer(base[:, :layer.n_in_features]), lambda: ops.matmul_matgptq_raw(x, *args),
                 lambda: ops.matmul_matgptq_grouped_raw(x, *([a] for a in args[:3]), args[3], [args[4]], *args[5:]),
                 lambda: torch.ops.matgptq_cuda.matmul_matgptq(x, *args)):
        want, seen = call(), calls.value
        pool = torch.cuda.MemPool(allocator.allocator())
        with torch.cuda.use_mem_pool(pool):
            y = call()
        assert calls.value > seen and with_gil.value == 0
        assert torch.equal(y, want)
        torch.cuda.synchronize()
        del y, pool
