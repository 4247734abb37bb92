"""Decode attention with the number of splits left to the op: few sequences take one cluster of eight splits, down to contexts
shorter than a split."""
import pytest
import torch

from litevllm_b200 import ops
from litevllm_b200.ops import reference


@pytest.mark.parametrize("B,nkv,hd,context,want", [(1, 4, 64, 2112, 8), (4, 4, 64, 2112, 8), (5, 4, 64, 2112, 15), (2, 8, 128, 2112, 8),
                                                    (4, 8, 128, 2112, 10), (1, 8, 256, 1024, 8), (2, 8, 256, 2112, 19), (1, 4, 64, 2561, 32),
                                                    (1, 4, 64, 300, 5), (1, 4, 64, 1, 1)])
def test_rule(B, nkv, hd, context, want):
    assert ops.pick_decode_splits(B, nkv, context, cluster_head=hd) == want
    assert ops.pick_decode_splits(B, nkv, context) == min(max(1, -(-296 // (B * nkv))), -(-context // 64), 32)


@pytest.mark.gpu
@pytest.mark.parametrize("B,nh,nkv,hd", [(1, 32, 4, 64), (2, 32, 8, 128), (1, 16, 8, 256)])
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("window", [0, 1024])
def test_few_sequences(B, nh, nkv, hd, fp8, window):
    g = torch.Generator(device="cuda").manual_seed(hd)
    bs, blocks = 16, 160
    dt = torch.float8_e4m3fn if fp8 else torch.bfloat16
    k, v = (torch.randn(1 + B * blocks, nkv, bs, hd, generator=g, device="cuda").to(torch.bfloat16).to(dt) for _ in range(2))
    table = (1 + torch.randperm(B * blocks, generator=g, device="cuda")).int().view(B, blocks)
    for lens in ([1], [63], [320], [321], [2560]):
        seq = torch.tensor((lens * B)[:B], device="cuda", dtype=torch.int32)
        if B > 1:
            seq[1] = 131
        q = torch.randn(B, nh * hd, generator=g, device="cuda").to(torch.bfloat16)
        got = ops.paged_attention_decode(q, k, v, table, seq, nh, nkv, hd, hd ** -0.5, window, 0.0, max_kv_len=2560)
        cu = torch.arange(B + 1, dtype=torch.int32)
        ref = reference.paged_attention(q.cpu().float(), k.cpu().float(), v.cpu().float(), table.cpu(), seq.cpu(), cu, nh, nkv, hd,
                                        hd ** -0.5, window, 0.0)
        # probabilities and the result are rounded to 16 bits: 2^-8 of values that average around one each
        assert torch.all((got.float().cpu() - ref.float()).abs() <= 2.0 ** -6 * (ref.float().abs() + ref.float().abs().mean()))


@pytest.mark.gpu
@pytest.mark.parametrize("nkv,group,hd", [(4, 8, 64), (8, 4, 128), (8, 2, 256)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_eight_splits_are_as_accurate_as_many(nkv, group, hd, dtype):
    """Distances from 64-bit results over several inputs, eight splits against one per 64 keys.  Both round the same weights, so
    they differ by the order of 32-bit sums alone; 1 % covers results that fall on the other side of a rounding."""
    few = many = 0.0
    nh, blocks, context = nkv * group, 132, 2040
    for seed in range(8):
        g = torch.Generator(device="cuda").manual_seed(seed)
        k, v = (torch.randn(1 + blocks, nkv, 16, hd, generator=g, device="cuda").to(dtype) for _ in range(2))
        q = torch.randn(1, nh * hd, generator=g, device="cuda").to(dtype)
        table = (1 + torch.randperm(blocks, generator=g, device="cuda")).int().view(1, -1)
        seq = torch.tensor([context], device="cuda", dtype=torch.int32)
        keys, values = (c[table[0].long()].permute(1, 0, 2, 3).reshape(nkv, -1, hd)[:, :context].double() for c in (k, v))
        ref = (torch.softmax(q.double().view(nkv, group, hd) @ keys.transpose(1, 2) * hd ** -0.5, -1) @ values).reshape(1, -1)
        for splits in (8, 32):
            got = ops.paged_attention_decode(q, k, v, table, seq, nh, nkv, hd, hd ** -0.5, splits=splits, max_kv_len=2112)
            err = float((got.double() - ref).norm() / ref.norm())
            few, many = (few + err, many) if splits == 8 else (few, many + err)
    assert few <= 1.01 * many
