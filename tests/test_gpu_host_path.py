"""MatGPTQLinear's C++ host path: the same rows as the operator computes, whatever form the input comes in, and the
dispatcher still sees the call when something listens to it."""
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
