"""Decode attention with the number of splits left to the op: few sequences take one cluster of eight splits, down to contexts
shorter than a split."""
import pytest

from litevllm_b200 import ops


@pytest.mark.parametrize("B,nkv,hd,context,want", [(1, 4, 64, 2112, 8), (4, 4, 64, 2112, 8), (5, 4, 64, 2112, 15), (2, 8, 128, 2112, 8),
                                                    (4, 8, 128, 2112, 10), (1, 8, 256, 1024, 8), (2, 8, 256, 2112, 19), (1, 4, 64, 2561, 32),
                                                    (1, 4, 64, 300, 5), (1, 4, 64, 1, 1)])
def test_rule(B, nkv, hd, context, want):
    assert ops.pick_decode_splits(B, nkv, context, cluster_head=hd) == want
    assert ops.pick_decode_splits(B, nkv, context) == min(max(1, -(-296 // (B * nkv))), -(-context // 64), 32)
