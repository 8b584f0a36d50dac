"""Tensor-core path with the weights in tensor memory and fp32 scaling: edges of its row tiles, batch blocks, stages and K
splits, against the unrounded weights in 64 bits."""
import ctypes

import pytest
import torch

from matgptq_b200 import _native, ops, synth  # noqa: F401  registers the operators
from oracle import matgptq_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("b,gs,n_out,n_in,m", [
    (2, 128, 16, 128, 17),       # one tile, one block of in-features
    (3, 32, 144, 384, 33),       # a last CTA with one tile of its eight
    (4, 128, 1040, 2944, 32),    # sixteen or eight tiles a CTA, K split unevenly
    (6, -1, 2064, 1152, 48),
    (8, 32, 272, 640, 64),
    (4, 128, 4096, 4096, 65),    # two batch blocks of 48 rows
    (8, -1, 256, 4224, 129),     # three blocks
    (2, 128, 28672, 256, 20),    # more tiles than one wave of eight a CTA holds
    (3, 128, 1024, 14336, 128)])
def test_zero_points_at_the_edges(cuda, dtype, b, gs, n_out, n_in, m):
    flag = 1 | (2 if dtype == torch.bfloat16 else 0)
    layer = synth.make_layer(n_out, n_in, gs, seed=b, sym=False, dtype=dtype, device=cuda)
    x = synth.make_activations(m, n_in, seed=m, dtype=dtype, device=cuda)
    packed = torch.ops.matgptq_cuda.slice_pack_matgptq_qweights(layer.qweight, n_out, n_in, 8, b, gs, flag)
    s, z = (torch.ops.matgptq_cuda.reorder_matgptq_scales(t, n_out, n_in, gs) for t in (layer.scales, layer.zeros))
    y = torch.ops.matgptq_cuda.matmul_matgptq_zeros(x, packed, s, z, n_out, n_in, b, gs, flag)
    again = torch.ops.matgptq_cuda.matmul_matgptq_zeros(x, packed, s, z, n_out, n_in, b, gs, flag)
    assert _native.device_status() == 0
    assert torch.equal(y, again)  # sums in a fixed order
    codes = oracle.matryoshka_slice(layer.qweight, 8, b).double() * 2 ** (8 - b) - 128
    group = n_in if gs == -1 else gs
    scale, zero = (t.double().repeat_interleave(group, 1) for t in (layer.scales, layer.zeros))
    ref = x.double() @ (scale * (codes - (zero - 128))).t()
    # the result is rounded once; sums of the integers and of the activations meet in fp32, a few dozen additions of 2^-24 each
    size = x.double().abs() @ (scale.abs() * (codes.abs() + (zero - 128).abs())).t()
    half_ulp = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)  # of a value just above a power of two: 7 and 10 bits follow it
    assert ((y.double() - ref).abs() <= half_ulp * ref.abs() * 1.01 + 2.0 ** -19 * size).all()


def _zp_layer(n_out, n_in, b, gs, dtype, cuda):
    layer = synth.make_layer(n_out, n_in, gs, seed=b, sym=False, dtype=dtype, device=cuda)
    flag = 1 | (2 if dtype == torch.bfloat16 else 0)
    packed = torch.ops.matgptq_cuda.slice_pack_matgptq_qweights(layer.qweight, n_out, n_in, 8, b, gs, flag)
    s, z = (torch.ops.matgptq_cuda.reorder_matgptq_scales(t, n_out, n_in, gs) for t in (layer.scales, layer.zeros))
    return lambda x, pdl=0: torch.ops.matgptq_cuda.matmul_matgptq_zeros(x, packed, s, z, n_out, n_in, b, gs, flag | pdl)


@pytest.mark.parametrize("gs,m", [(128, 64), (-1, 40), (32, 130)])
def test_a_slow_kernel_before_it_in_the_chain(lib, cuda, gs, m):
    # the product starts while the kernel before it rests, for longer than any of its waits would last: it waits for its
    # activations all the same and reports nothing
    product = _zp_layer(2048, 4096, 4, gs, torch.float16, cuda)
    x = synth.make_activations(m, 4096, seed=m, dtype=torch.float16, device=cuda)
    want = product(x)
    late = torch.zeros_like(x)
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.matgptq_b200_selftest_late_writer(x.data_ptr(), late.data_ptr(), x.numel(), 2500, stream) == 0
    y = product(late, pdl=4)
    assert _native.device_status() == 0
    assert torch.equal(y, want)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("n,b,gs,m", [(4096, 4, 128, 48),   # K split
                                      (8192, 8, -1, 200),   # and not
                                      (2048, 3, 32, 24)])
def test_chained_products(cuda, dtype, n, b, gs, m):
    # each product's result is the next one's input, all launched with programmatic dependent launch; a result's memory comes
    # back two products later, so that one written too early shows as well
    products = [_zp_layer(n, n, b, gs, dtype, cuda) for _ in range(2)]
    x = synth.make_activations(m, n, seed=m, dtype=dtype, device=cuda)

    def chain(pdl):
        y = x
        for i in range(4):
            y = products[i & 1](y, pdl)
        return y
    want = chain(0)
    assert want.isfinite().all() and want.abs().max() > 0
    for _ in range(4):
        assert torch.equal(chain(4), want)
    assert _native.device_status() == 0


def _path(lib, b, gs, n, k, m):
    plan = (ctypes.c_int * 8)()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert lib.matgptq_b200_zp_plan(b, gs, n, k, m, sms, (ctypes.c_int * 7)(*[sms // s for s in range(2, 9)]), 8, plan) == 0
    return plan[0]


@pytest.mark.parametrize("b", (2, 3, 4, 6, 8))
@pytest.mark.parametrize("gs", [-1, 32, 128])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_weights_read_back_on_the_tensor_cores(lib, cuda, b, gs, dtype):
    # one-hot rows give the weights, rounded once, of a layer wide enough for the tensor cores
    n_out, n_in = 4112, 512
    assert _path(lib, b, gs, n_out, n_in, n_in) == 2
    layer = synth.make_layer(n_out, n_in, gs, seed=b, sym=False, dtype=dtype, device=cuda)
    flag = 1 | (2 if dtype == torch.bfloat16 else 0)
    layer.zeros[::7] = 0.0
    layer.zeros[3::7] = 255.0
    packed = torch.ops.matgptq_cuda.slice_pack_matgptq_qweights(layer.qweight, n_out, n_in, 8, b, gs, flag)
    s, z = (torch.ops.matgptq_cuda.reorder_matgptq_scales(t, n_out, n_in, gs) for t in (layer.scales, layer.zeros))
    want = oracle.dequantize_weight(layer.qweight.cpu(), layer.scales.cpu(), layer.zeros.cpu(), 8, b)
    y = torch.ops.matgptq_cuda.matmul_matgptq_zeros(torch.eye(n_in, dtype=dtype, device=cuda), packed, s, z, n_out, n_in, b, gs, flag)
    assert _native.device_status() == 0
    assert torch.equal(y.cpu(), want.t().contiguous())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("b,gs,n,k", [(4, 128, 256, 4096), (8, 32, 1024, 1024), (3, -1, 528, 2944)])
def test_both_sides_of_the_dispatch(lib, cuda, dtype, b, gs, n, k):
    # the last batch on the GEMV, in several passes with a ragged one, and the first on the tensor cores
    rows = [m for m in range(17, 600) if _path(lib, b, gs, n, k, m) == 1][-1]
    product = _zp_layer(n, k, b, gs, dtype, cuda)
    layer = synth.make_layer(n, k, gs, seed=b, sym=False, dtype=dtype, device=cuda)
    group = k if gs == -1 else gs
    codes = oracle.matryoshka_slice(layer.qweight, 8, b).double() * 2 ** (8 - b) - 128
    scale, zero = (t.double().repeat_interleave(group, 1) for t in (layer.scales, layer.zeros))
    for m in (rows - 15, rows, rows + 1):
        x = synth.make_activations(m, k, seed=m, dtype=dtype, device=cuda)
        ref = x.double() @ (scale * (codes - (zero - 128))).t()
        # the result is rounded once; sums of the integers and of the activations meet in fp32
        size = x.double().abs() @ (scale.abs() * (codes.abs() + (zero - 128).abs())).t()
        half_ulp = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
        assert ((product(x).double() - ref).abs() <= half_ulp * ref.abs() * 1.01 + 2.0 ** -19 * size).all(), m
    assert _native.device_status() == 0


@pytest.mark.parametrize("gs,n,k,m", [(128, 4096, 4096, 40), (-1, 8192, 256, 40)])  # K split, and not
def test_output_at_any_two_byte_address(lib, cuda, gs, n, k, m):
    assert _path(lib, 4, gs, n, k, m) == 2
    layer = synth.make_layer(n, k, gs, seed=1, sym=False, dtype=torch.float16, device=cuda)
    packed = torch.ops.matgptq_cuda.slice_pack_matgptq_qweights(layer.qweight, n, k, 8, 4, gs, 1)
    s, z = (torch.ops.matgptq_cuda.reorder_matgptq_scales(t, n, k, gs) for t in (layer.scales, layer.zeros))
    x = synth.make_activations(m, k, seed=1, dtype=torch.float16, device=cuda)
    want = torch.ops.matgptq_cuda.matmul_matgptq_zeros(x, packed, s, z, n, k, 4, gs, 1)
    for shift in range(1, 8):
        room = torch.full((m * n + 16,), 7.0, dtype=torch.float16, device=cuda)
        y = room[shift:shift + m * n]
        assert lib.matgptq_b200_matmul_zp(4, gs, n, k, m, packed.data_ptr(), s.data_ptr(), z.data_ptr(), x.data_ptr(), y.data_ptr(),
                                          torch.cuda.current_stream().cuda_stream, 1) == 0
        assert torch.equal(y.view(m, n), want)
        assert (room[:shift] == 7.0).all() and (room[shift + m * n:] == 7.0).all()
    assert _native.device_status() == 0


@pytest.mark.parametrize("gs", [-1, 32, 128])
def test_bf16_activations_beyond_the_range_of_fp16(lib, cuda, gs):
    n, k, m, bf16 = 4096, 1024, 64, torch.bfloat16
    assert _path(lib, 4, gs, n, k, m) == 2
    product = _zp_layer(n, k, 4, gs, bf16, cuda)
    x = synth.make_activations(m, k, seed=3, dtype=bf16, device=cuda)
    big = (x.float() * 1e6).to(bf16)
    # a power of two more in the activations is one more in the result
    assert torch.equal(product((x.float() * 2.0 ** 20).to(bf16)).float(), product(x).float() * 2.0 ** 20)
    assert (big.abs() > 65504).any() and product(big).isfinite().all()
    # what is not finite stays in its row
    odd = x.clone()
    odd[5, 100], odd[9, 7], odd[63, 1023] = float("inf"), float("nan"), float("-inf")
    y, others = product(odd), [r for r in range(m) if r not in (5, 9, 63)]
    assert not y[[5, 9, 63]].isfinite().any()
    assert torch.equal(y[others], product(x)[others])
    # the GEMV's limit: what is larger counts as 65504
    small = _zp_layer(256, k, 4, gs, bf16, cuda)
    assert _path(lib, 4, gs, 256, k, 16) == 1
    assert torch.equal(small(big[:16]), small(big[:16].clamp(-65504, 65504)))
    assert _native.device_status() == 0
