"""Zero points on the tensor-core path: the weights it builds, read back through the product with one-hot rows, are the
oracle's dequantised weights bit for bit (one term per output, exact accumulation, one rounding)."""
import pytest
import torch

from matgptq_b200 import synth
from oracle import matgptq_oracle as oracle


@pytest.mark.gpu
@pytest.mark.parametrize("b", (2, 3, 4, 6, 8))
@pytest.mark.parametrize("gs", [-1, 32, 128])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_dense_tile_with_zero_points_is_bit_exact(cuda, b, gs, dtype):
    from matgptq_b200 import _native, ops  # noqa: F401  registers the operators
    n_out, n_in = 144, 256  # a ragged 128-row tile
    flag = 1 | (2 if dtype == torch.bfloat16 else 0)
    layer = synth.make_layer(n_out, n_in, gs, seed=60 + b, sym=False, dtype=dtype, device=cuda)
    layer.zeros[::7] = 0.0    # the ends of the range too
    layer.zeros[3::7] = 255.0
    packed = torch.ops.matgptq_cuda.slice_pack_matgptq_qweights(layer.qweight, n_out, n_in, 8, b, gs, flag)
    s, z = (torch.ops.matgptq_cuda.reorder_matgptq_scales(t, n_out, n_in, gs) for t in (layer.scales, layer.zeros))
    w_ref = oracle.dequantize_weight(layer.qweight.cpu(), layer.scales.cpu(), layer.zeros.cpu(), 8, b)
    x = torch.eye(n_in, dtype=dtype, device=cuda)
    y = torch.ops.matgptq_cuda.matmul_matgptq_zeros(x, packed, s, z, n_out, n_in, b, gs, flag)
    assert _native.device_status() == 0
    assert torch.equal(y.cpu(), w_ref.t().contiguous())
