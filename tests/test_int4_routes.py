"""Which int4 products of many tokens go through a 16-bit copy of their weights (ops/awq.py)."""
from types import SimpleNamespace

import pytest
import torch

from litevllm_b200 import ops
from litevllm_b200.ops import awq


def _expands(T, N, K, gated=False, **kw):
    x, out = torch.empty(T, K, dtype=torch.bfloat16), torch.empty(T, N // 2 if gated else N, dtype=torch.bfloat16)
    return awq._expands(T, SimpleNamespace(N=N, K=K), x, out, None, gated, **kw)


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
