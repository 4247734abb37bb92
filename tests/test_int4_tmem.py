"""Routed int4 experts whose weights are expanded into tensor memory (csrc/gemm/int4_tmem.cu) against the 32-bit oracle."""
import pytest
import torch

from litevllm_b200 import ops
from litevllm_b200.ops import moe
from litevllm_b200.ops.awq import Int4Weight

DEV = "cuda"


def test_tile_follows_the_mean_number_of_rows():
    assert [moe._tmem_tile(m) for m in (0, 10, 11, 21, 22, 500)] == [16, 16, 32, 32, 64, 64]


# tokens, experts, experts per token, widths, group, zero points: one k-block and k-blocks that end inside a stage of four, the last tile of
# 128 and 256 rows partly or half empty, tiles of 16, 32 and 64 rows, fewer and more tiles than SMs, a crowded expert and empty ones
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,E,K,H,inter,group,zeros", [
    (16, 4, 2, 64, 64, 32, False), (33, 8, 2, 320, 192, 64, True), (64, 16, 4, 2816, 704, 32, False), (60, 8, 2, 256, 1408, 128, True),
    (200, 8, 2, 192, 320, 32, True), (300, 4, 2, 1024, 384, 128, False), (130, 128, 8, 128, 128, 64, False)])
def test_experts_in_tensor_memory(T, E, K, H, inter, group, zeros, dtype):
    g = torch.Generator(device=DEV).manual_seed(T + E)

    def weight(rows, cols):
        nib = torch.randint(0, 16, (rows, cols), generator=g, device=DEV, dtype=torch.uint8)
        s = (torch.rand(rows, cols // group, generator=g, device=DEV) + 0.5).mul_(0.2 * cols ** -0.5).to(dtype)
        z = torch.randint(4, 12, (rows, cols // group), generator=g, device=DEV, dtype=torch.uint8) if zeros else None
        return Int4Weight(nib, s, z, group, dtype)
    gu, dn = weight(E * 2 * inter, H), weight(E * H, inter)
    x = torch.randn(T, 2 * H, generator=g, device=DEV).to(dtype)[:, :H]          # rows further apart than they are long
    score = torch.rand(T, E, generator=g, device=DEV)
    score[:, 0] += 0.4                                   # one crowded expert
    score[:, 1] -= 2.0                                   # and an empty one
    ids = score.topk(K).indices.int()
    wts = torch.rand(T, K, generator=g, device=DEV)
    assert T * K >= moe._TMEM_MIN_ROUTES and moe._tmem_takes(gu, dn, H, inter)
    got = moe.fused_experts(x, gu, dn, ids, wts, E, 0, "gelu_tanh").float()
    ops.check_status(x.device)
    ref = moe._reference_experts(x, gu, dn, ids, wts, E, 0, E, "gelu_tanh").float()
    # both round the expanded weights, the gated activations, the experts' rows and the sum to 16 bits (half an ulp each): four
    # roundings of relative size 2^-9 or 2^-12, the first of which the oracle does not make
    eps = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert (got - ref).norm() <= 2 * eps * ref.norm()
    assert (got - ref).abs().max() <= 8 * eps * ref.abs().max()
