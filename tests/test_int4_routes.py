"""Which int4 products of many tokens go through a 16-bit copy of their weights (ops/awq.py)."""
from types import SimpleNamespace

import pytest
import torch

from litevllm_b200 import ops
from litevllm_b200.ops import awq


def _expands(T, N, K, gated=False, **kw):
    x, out = torch.empty(T, K, dtype=torch.bfloat16), torch.empty(T, N // 2 if gated else N, dtype=torch.bfloat16)
    return awq._expands(T, SimpleNamespace(N=N, K=K, copy_fits=True), x, out, None, gated, **kw)


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
