"""Which int4 products of many tokens go through a 16-bit copy of their weights (ops/awq.py)."""
from types import SimpleNamespace

import pytest
import torch

from litevllm_b200 import ops
from litevllm_b200.ops import awq


def _expands(T, N, K, gated=False, group=128):
    x, out = torch.empty(T, K, dtype=torch.bfloat16), torch.empty(T, N // 2 if gated else N, dtype=torch.bfloat16)
    return awq._expands(T, SimpleNamespace(N=N, K=K, group=group, copy_fits=True), x, out, None, gated)


@pytest.mark.parametrize("switch,value,plain,gated", [
    ("_PERSISTENT_GEMM", True, True, True), ("_PERSISTENT_PLAIN", False, False, True), ("_PERSISTENT_MIN_T", 4096, False, False),
    ("_PERSISTENT_MIN_T", 2, True, True)])
def test_the_switches_of_the_persistent_kernel_hold(monkeypatch, switch, value, plain, gated):
    monkeypatch.setattr(ops, switch, value)
    assert _expands(1024, 6144, 4096) == plain
    assert _expands(1024, 6144, 4096, gated=True) == gated
    assert not _expands(128, 6144, 4096) and not _expands(128, 6144, 4096, gated=True)


def test_everything_off(monkeypatch):
    monkeypatch.setattr(ops, "_PERSISTENT_GEMM", False)      # as FI_PERSISTENT_GEMM=0 sets both
    monkeypatch.setattr(ops, "_PERSISTENT_PLAIN", False)
    assert not _expands(1024, 6144, 4096) and not _expands(1024, 6144, 4096, gated=True)


# (tokens, outputs, K, group, gated, us fused, us expanded), both timed on one B200
@pytest.mark.parametrize("T,N,K,group,gated,fused,expanded", [
    (129, 64, 4096, 128, False, 10.8, 15.3), (512, 64, 8192, 32, False, 15.0, 23.5), (129, 256, 8192, 128, False, 18.2, 24.1),
    (200, 512, 12288, 128, False, 24.9, 35.1), (1024, 4096, 512, 128, False, 13.7, 18.5), (512, 8192, 512, 32, False, 13.7, 18.9),
    (768, 6144, 256, 128, False, 11.0, 16.7), (300, 12288, 8192, 128, False, 101.6, 119.6), (200, 8192, 12288, 32, True, 180.4, 227.1),
    (192, 6144, 4096, 128, False, 42.0, 28.0), (351, 8192, 2816, 32, False, 43.8, 32.5), (1250, 2816, 2112, 32, False, 38.9, 27.5), (2048, 6144, 4096, 128, False, 157.0, 97.0), (2048, 4096, 12288, 128, False, 268.0, 201.0),
    (2048, 8192, 2816, 32, False, 139.0, 93.0), (1000, 256, 4096, 128, False, 23.3, 15.8), (512, 512, 2816, 32, False, 20.8, 13.6),
    (129, 64, 512, 128, True, 24.5, 12.4), (192, 12288, 4096, 128, True, 141.0, 109.0), (2048, 2112, 2816, 32, True, 109.0, 46.0)])
def test_the_faster_kernel_by_size(T, N, K, group, gated, fused, expanded):
    assert _expands(T, 2 * N if gated else N, K, gated, group) == (expanded < fused)


@pytest.mark.gpu
def test_products_run_where_the_copy_finds_no_memory():
    """The allocator of this process is told to stop a little above what it holds, below the 128 MiB of the copy."""
    g = torch.Generator(device="cuda").manual_seed(3)
    N = K = 8192
    w = awq.Int4Weight(torch.randint(0, 16, (N, K), generator=g, device="cuda", dtype=torch.uint8),
                       torch.rand(N, K // 128, generator=g, device="cuda").mul_(0.01).to(torch.bfloat16), None, 128, torch.bfloat16)
    x = torch.randn(256, K, generator=g, device="cuda").to(torch.bfloat16)
    want = awq.int4_linear(x, w, bn=128)                 # the fused kernel
    out = torch.empty_like(want)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (32 << 20)) / total)
    try:
        for _ in range(2):
            assert torch.equal(awq.int4_linear(x, w, out=out.zero_()), want)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
