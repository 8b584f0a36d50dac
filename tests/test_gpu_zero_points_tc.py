"""Zero points at the batch sizes where products without them go to the tensor cores: the weights, read back through the
product with one-hot rows, are the oracle's dequantised weights bit for bit (one term per output, exact accumulation, one
rounding), and a sum of several is that of the unrounded weights."""
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


@pytest.mark.gpu
@pytest.mark.parametrize("b", (2, 3, 4, 6, 8))
@pytest.mark.parametrize("gs", [-1, 32, 128])
@pytest.mark.parametrize("m,n_out", [(17, 2064), (25, 1040), (300, 144)])
@pytest.mark.parametrize("dtype,scale", [(torch.float16, 1 + 2.0 ** -10), (torch.bfloat16, 1 + 2.0 ** -7), (torch.float16, 300.0)])
def test_weights_are_not_rounded_at_any_batch_size(cuda, b, gs, m, n_out, dtype, scale):
    # 16 terms of +-2^-6 per row: every partial sum is a whole number below 2^12 times scale * 2^-6, exact in 24 bits.
    # Weights rounded to the type would lose the scale's last bit or, at 300, leave the range of fp16.
    from matgptq_b200 import _native, ops  # noqa: F401
    n_in, flag = 256, 1 | (2 if dtype == torch.bfloat16 else 0)
    gen = torch.Generator(device=cuda).manual_seed(m)
    q = torch.randint(0, 256, (n_out, n_in), generator=gen, device=cuda, dtype=torch.uint8)
    groups = 1 if gs == -1 else n_in // gs
    scales = torch.full((n_out, groups), scale, device=cuda, dtype=dtype)
    zeros = torch.randint(0, 256, (n_out, groups), generator=gen, device=cuda).to(dtype)
    x = torch.zeros(m, n_in, device=cuda, dtype=dtype)
    cols = torch.rand(m, n_in, generator=gen, device=cuda).argsort(1)[:, :16]
    x.scatter_(1, cols, (torch.randint(0, 2, (m, 16), generator=gen, device=cuda) * 2 - 1).to(dtype) / 64)
    packed = torch.ops.matgptq_cuda.slice_pack_matgptq_qweights(q, n_out, n_in, 8, b, gs, flag)
    s, z = (torch.ops.matgptq_cuda.reorder_matgptq_scales(t, n_out, n_in, gs) for t in (scales, zeros))
    y = torch.ops.matgptq_cuda.matmul_matgptq_zeros(x, packed, s, z, n_out, n_in, b, gs, flag)
    codes = oracle.matryoshka_slice(q.cpu(), 8, b).to(cuda).double() * 2 ** (8 - b)
    w = (codes.view(n_out, groups, -1) - zeros.double().unsqueeze(-1)) * scales.double().unsqueeze(-1)
    assert _native.device_status() == 0
    assert torch.equal(y, (x.double() @ w.view(n_out, n_in).t()).to(dtype))
