"""What the operators refuse before anything is launched, and what autograd makes of them."""
import numpy as np
import pytest
import torch
import torch.autograd.forward_ad as forward_ad

from matgptq_b200 import ops  # noqa: F401  registers the operators

N, K, B, G = 16, 256, 4, 128


def _tensors(device):
    words = torch.zeros(B * N * K // 32, dtype=torch.int32, device=device).view(torch.uint32)
    return words, torch.ones(N, K // G, dtype=torch.float16, device=device)


def _dequantize(words, scales, group=G):
    return torch.ops.matgptq_cuda.dequantize_matgptq(words, scales, N, K, B, group, 1)


def test_dequantize_refuses_host_tensors():
    # with a GPU present it would otherwise read the host's addresses on the device
    words, scales = _tensors("cpu")
    with pytest.raises(RuntimeError, match="expected matgptq_weights to be a CUDA tensor"):
        _dequantize(words, scales)


@pytest.mark.gpu
def test_dequantize_refuses_what_it_would_read_out_of_range(cuda):
    words, scales = _tensors(cuda)
    assert _dequantize(words, scales).shape == (N, K)
    assert torch.equal(_dequantize(words.view(torch.int32), scales), _dequantize(words, scales))
    for bad_words, bad_scales in ((words.cpu(), scales), (words, scales.cpu()), (words.cpu(), scales.cpu()), (words[:-1], scales),
                                  (words.view(torch.uint8)[:words.numel()], scales), (words.view(torch.int32).repeat(2)[::2], scales),
                                  (words, scales[:-1]), (words, scales[:, :1]), (words, scales.t().contiguous().t())):
        with pytest.raises(RuntimeError):
            _dequantize(bad_words, bad_scales)
    with pytest.raises(RuntimeError):
        _dequantize(words, scales, group=32)  # more groups than there are scales


def _matmul(x, words, scales):
    return torch.ops.matgptq_cuda.matmul_matgptq(x, words, scales, N, K, B, G, 1)


def _matmul_out(x, words, scales, out):
    torch.ops.matgptq_cuda.matmul_matgptq_out(x, words, scales, N, K, B, G, 1, out)


@pytest.mark.parametrize("device", ["meta", pytest.param("cuda", marks=pytest.mark.gpu)])
def test_tangents_are_dropped_and_gradients_are_not_defined(device):
    words, scales = _tensors(device)
    x = torch.ones(2, K, dtype=torch.float16, device=device)
    with forward_ad.dual_level():
        y = _matmul(forward_ad.make_dual(x, torch.ones_like(x)), words, scales)
        assert y.shape == (2, N) and forward_ad.unpack_dual(y).tangent is None
        torch.ops.matgptq_cuda.matmul_matgptq_grouped(forward_ad.make_dual(x, torch.ones_like(x)), [words], [scales], [N], K, [B], G, 1)
        with pytest.raises(NotImplementedError):
            _matmul(forward_ad.make_dual(x.clone().requires_grad_(), torch.ones_like(x)), words, scales)
    for inputs in ((x.clone().requires_grad_(), words, scales), (x, words, scales.clone().requires_grad_())):
        y = _matmul(*inputs)
        assert y.requires_grad
        with pytest.raises(RuntimeError, match="matmul_matgptq"):
            y.sum().backward()
        with torch.no_grad():
            assert not _matmul(*inputs).requires_grad
    y = torch.ops.matgptq_cuda.matmul_matgptq_grouped(x, [words], [scales.clone().requires_grad_()], [N], K, [B], G, 1)
    assert y.requires_grad
    assert not _matmul(x, words, scales).requires_grad


@pytest.mark.parametrize("device", ["meta", pytest.param("cuda", marks=pytest.mark.gpu)])
def test_out_counts_as_written_and_may_be_a_leaf(device):
    words, scales = _tensors(device)
    x = torch.ones(2, K, dtype=torch.float16, device=device)
    out = torch.zeros(2, N, dtype=torch.float16, device=device)
    before = out._version
    _matmul_out(x, words, scales, out)
    _matmul_out(x.clone().requires_grad_(), words, scales, out)
    assert out._version == before + 2 and not out.requires_grad
    _matmul_out(x, words, scales, out.clone().requires_grad_())
    with torch.inference_mode():
        _matmul_out(x, words, scales, torch.zeros(2, N, dtype=torch.float16, device=device))


def test_a_tangent_does_not_change_where_a_call_fails():
    # no GPU is reached with a host tensor of the wrong shape, with a tangent or without
    scales = torch.ones(N, 3, dtype=torch.float16)
    with forward_ad.dual_level(), pytest.raises(RuntimeError, match="scales must have shape"):
        torch.ops.matgptq_cuda.reorder_matgptq_scales(forward_ad.make_dual(scales, torch.ones_like(scales)), N, K, G)


@pytest.mark.gpu
@pytest.mark.parametrize("number", [np.int64, np.int32, torch.tensor])
def test_raw_entries_take_any_whole_number(cuda, number):
    words, scales = _tensors(cuda)
    x = torch.randn(2, K, dtype=torch.float16, device=cuda)
    want = _matmul(x, words, scales)
    assert torch.equal(ops.matmul_matgptq_raw(x, words, scales, *(number(v) for v in (N, K, B, G, 1))), want)
    assert torch.equal(ops.matmul_matgptq_grouped_raw(x, (words,), (scales,), (number(N),), number(K), (number(B),), number(G), number(1)),
                       want)
    if number is not torch.tensor:
        assert torch.equal(ops.matmul_matgptq_grouped_raw(x, [words], [scales], np.array([N]), K, np.array([B], dtype=np.uint8), G, 1), want)
    with pytest.raises(RuntimeError):
        ops.matmul_matgptq_raw(x, words, scales, float(N), K, B, G, 1)


@pytest.mark.gpu
def test_pybind_stand_in_is_outside_autograd(cuda):
    from matgptq_cuda import _CUDA
    words, scales = _tensors(cuda)
    grad = scales.clone().requires_grad_()
    x = torch.ones(2, K, dtype=torch.float16, device=cuda, requires_grad=True)
    assert not _CUDA.reorder_matgptq_scales(grad, N, K, G).requires_grad
    y = _CUDA.matmul_matgptq(x, words, grad, N, K, B, G, 1)
    assert not y.requires_grad and torch.equal(y, _matmul(x.detach(), words, scales))
