"""What the operators refuse before anything is launched."""
import pytest
import torch

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
