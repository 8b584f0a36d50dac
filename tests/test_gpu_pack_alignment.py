"""The GPU packer against the host packer, from code buffers that start on and off an 8-byte boundary."""
import numpy as np
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("b", (2, 3, 4, 6, 8))
@pytest.mark.parametrize("master", [0, 8, 6])
@pytest.mark.parametrize("offset", [0, 8, 3])
def test_pack_matches_host(lib, cuda, b, master, offset):
    if master and master < b:
        pytest.skip("a slice cannot be wider than its master")
    n, k = 48, 384
    rng = np.random.default_rng(b)
    codes = rng.integers(0, 256, (n, k), dtype=np.uint8)
    codes[0, :256] = np.arange(256, dtype=np.uint8)
    host = np.zeros(b * n * k // 32, dtype=np.uint32)
    assert lib.matgptq_b200_pack_qweights_host(codes.ctypes.data, host.ctypes.data, n, k, b, master) == 0
    buf = torch.zeros(n * k + 16, dtype=torch.uint8, device=cuda)
    buf[offset:offset + n * k] = torch.from_numpy(codes.ravel()).to(cuda)
    src = buf[offset:offset + n * k].view(n, k)
    dst = torch.zeros(b * n * k // 32 + 4, dtype=torch.int32, device=cuda)
    for shift in (0, 1):  # a result on and off a 16-byte boundary
        out = dst[shift:shift + b * n * k // 32]
        assert lib.matgptq_b200_pack_qweights(src.data_ptr(), out.data_ptr(), n, k, b, master,
                                              torch.cuda.current_stream().cuda_stream) == 0
        assert np.array_equal(out.cpu().numpy().view(np.uint32), host)
