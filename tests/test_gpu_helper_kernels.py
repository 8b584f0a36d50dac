"""The harness's rotary embedding and SiLU kernels, 16-byte path and scalar path, against fp32 torch."""
import pytest
import torch

FLAG_BF16 = 2


def _shifted(shape, dtype, device, shift, seed):
    """Contiguous random tensor whose storage starts `shift` elements off a 16-byte boundary."""
    n = 1
    for s in shape:
        n *= s
    gen = torch.Generator(device=device).manual_seed(seed)
    return torch.randn(n + shift, generator=gen, device=device).to(dtype)[shift:].view(shape)


def _bound(ref, dtype):
    # one rounding of the result, and for silu one of the activation before it, each half a unit in the last place;
    # 1e-6 of fp32 arithmetic beside it
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    return ref.abs() * (2.1 * ulp + 1e-6) + 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,inter,shift", [(1, 8, 0), (3, 2056, 0), (70, 14336, 0), (3, 2052, 0), (3, 2056, 1), (40000, 8, 0)])
def test_silu_mul(lib, cuda, dtype, rows, inter, shift):
    gu = _shifted((rows, 2 * inter), dtype, cuda, shift, 1)
    out = torch.full((rows, inter), float("nan"), dtype=dtype, device=cuda)
    flag = FLAG_BF16 if dtype == torch.bfloat16 else 0
    assert lib.matgptq_b200_silu_mul(gu.data_ptr(), out.data_ptr(), rows, inter, flag, torch.cuda.current_stream().cuda_stream) == 0
    g, u = gu[:, :inter].float(), gu[:, inter:].float()
    ref = torch.nn.functional.silu(g) * u
    assert ((out.float() - ref).abs() <= _bound(ref, dtype)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("seq,keys", [(1, 256), (1, 1), (3, 13), (5, 1032), (5000, 16)])
def test_causal_mask(lib, cuda, dtype, seq, keys):
    pos = torch.randint(-1, keys + 2, (seq,), generator=torch.Generator(device=cuda).manual_seed(seq), device=cuda)
    mask = torch.full((seq + 1, keys), 7.0, dtype=dtype, device=cuda)
    flag = FLAG_BF16 if dtype == torch.bfloat16 else 0
    assert lib.matgptq_b200_causal_mask(pos.data_ptr(), mask.data_ptr(), seq, keys, flag, torch.cuda.current_stream().cuda_stream) == 0
    hidden = torch.arange(keys, device=cuda) > pos[:, None]
    assert torch.equal(mask[:seq], torch.zeros(seq, keys, dtype=dtype, device=cuda).masked_fill_(hidden, float("-inf")))
    assert (mask[seq] == 7.0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("batch,seq,heads,kv,d,shift",
                         [(1, 1, 32, 8, 128, 0), (3, 5, 4, 2, 64, 0), (2, 7, 3, 1, 24, 0), (2, 3, 4, 2, 12, 0), (2, 3, 4, 2, 64, 1)])
def test_rope_kv(lib, cuda, dtype, batch, seq, heads, kv, d, shift):
    max_seq, flag = 16, FLAG_BF16 if dtype == torch.bfloat16 else 0
    qkv = _shifted((batch, seq, heads + 2 * kv, d), dtype, cuda, shift, 2)
    pos = torch.arange(seq, device=cuda) * 2 + 1
    ang = torch.randn(max_seq, d // 2, device=cuda)
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    q = torch.zeros(batch, heads, seq, d, dtype=dtype, device=cuda)
    k, v = (torch.zeros(batch, kv, max_seq, d, dtype=dtype, device=cuda) for _ in range(2))
    assert lib.matgptq_b200_rope_kv(qkv.data_ptr(), pos.data_ptr(), cos.data_ptr(), sin.data_ptr(), q.data_ptr(), k.data_ptr(),
                                    v.data_ptr(), batch, seq, heads, kv, d, max_seq, flag,
                                    torch.cuda.current_stream().cuda_stream) == 0
    x = qkv.float().transpose(1, 2)
    a, b, c, s = x[..., 0::2], x[..., 1::2], cos[pos], sin[pos]
    rot = torch.stack([a * c - b * s, a * s + b * c], -1).flatten(-2)
    # the two products cancel at worst: the bound is relative to their sizes
    size = torch.stack([(a * c).abs() + (b * s).abs(), (a * s).abs() + (b * c).abs()], -1).flatten(-2)
    assert ((q.float() - rot[:, :heads]).abs() <= _bound(size[:, :heads], dtype)).all()
    assert ((k[:, :, pos].float() - rot[:, heads:heads + kv]).abs() <= _bound(size[:, heads:heads + kv], dtype)).all()
    assert torch.equal(v[:, :, pos], qkv.transpose(1, 2)[:, heads + kv:])
    others = [i for i in range(max_seq) if i not in pos.tolist()]
    assert not k[:, :, others].any() and not v[:, :, others].any()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_both_access_widths_give_the_same_bits(lib, cuda, dtype):
    batch, seq, heads, kv, d, max_seq = 2, 512, 32, 8, 128, 512
    flag, stream = FLAG_BF16 if dtype == torch.bfloat16 else 0, torch.cuda.current_stream().cuda_stream
    ang = torch.arange(max_seq, device=cuda)[:, None] * 1.7 ** -torch.arange(d // 2, device=cuda)
    cos, sin, pos = ang.cos().float().contiguous(), ang.sin().float().contiguous(), torch.arange(seq, device=cuda)
    outs = []
    for shift in (0, 1):
        # the same values at both alignments
        qkv = _shifted((batch, seq, heads + 2 * kv, d), dtype, cuda, 0, 5)
        if shift:
            qkv = torch.cat([qkv.new_zeros(1), qkv.flatten()])[1:].view(qkv.shape)
        q = torch.zeros(batch, heads, seq, d, dtype=dtype, device=cuda)
        k, v = (torch.zeros(batch, kv, max_seq, d, dtype=dtype, device=cuda) for _ in range(2))
        assert lib.matgptq_b200_rope_kv(qkv.data_ptr(), pos.data_ptr(), cos.data_ptr(), sin.data_ptr(), q.data_ptr(), k.data_ptr(),
                                        v.data_ptr(), batch, seq, heads, kv, d, max_seq, flag, stream) == 0
        act = torch.zeros(batch * seq, (heads + 2 * kv) * d // 2, dtype=dtype, device=cuda)
        assert lib.matgptq_b200_silu_mul(qkv.data_ptr(), act.data_ptr(), act.shape[0], act.shape[1], flag, stream) == 0
        outs.append((q, k, v, act))
    assert all(torch.equal(a, b) for a, b in zip(*outs))
