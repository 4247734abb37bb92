"""The A-stage hand-over of the int4 GEMM's row-per-thread dequantisers.

Two halves of the dequantising warps write k-blocks into a ring of AST stages; the tensor core reads the blocks in order.
A writer waits for the parity of its stage's "empty" barrier.  A parity tells only neighbouring rounds apart, so the split of
the k-blocks over the halves has to keep a writer from coming back to a stage two rounds early.  The CPU test walks every
interleaving of a model of the barriers with the split that the kernel's source states; the GPU test repeats products with few
k-blocks, where a half can run furthest ahead, and wants the same bits every time.
"""
import re
from pathlib import Path

import pytest
import torch

SOURCE = Path(__file__).resolve().parents[1] / "csrc" / "gemm" / "awq_gemm.cu"


def _early_write(stages: int, mine: list[list[int]], blocks: int) -> tuple | None:
    """First state in which a half's parity wait passes although the block AST before has not been read."""
    todo, seen = [(0, 0, 0, frozenset())], set()
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        p0, p1, read, written = state
        for half, at in enumerate((p0, p1)):
            if at == len(mine[half]):
                continue
            block = mine[half][at]
            rounds = sum(1 for b in range(read) if b % stages == block % stages)     # completed phases of the barrier
            if (rounds & 1) == ((block // stages) & 1):                              # the wait passes
                if rounds != block // stages:
                    return block, read
                todo.append((p0 + (half == 0), p1 + (half == 1), read, written | {block}))
        if read in written:
            todo.append((p0, p1, read + 1, written - {read}))
    assert any(s[2] == blocks for s in seen), "the hand-over never ends"
    return None


@pytest.mark.parametrize("stages", [2, 3])
def test_no_half_takes_an_unread_stage(stages):
    rule = re.search(r"const int sub = ([uhalf0-9 +*]+);", SOURCE.read_text()).group(1)
    blocks = 24
    mine = [[4 * rs + eval(rule, {"u": u, "half": half}) for rs in range(blocks // 4) for u in (0, 1)] for half in (0, 1)]
    assert sorted(mine[0] + mine[1]) == list(range(blocks))
    assert _early_write(stages, mine, blocks) is None


@pytest.mark.gpu
@pytest.mark.parametrize("K,group", [(704, 32), (2816, 32), (4096, 128)])
@pytest.mark.parametrize("gated", [False, True])
def test_repeated_int4_products_are_the_same(K, group, gated):
    from litevllm_b200.ops.awq import Int4Weight, int4_linear
    g = torch.Generator(device="cuda").manual_seed(1)
    N = 1408
    nib = torch.randint(0, 16, (N, K), generator=g, device="cuda", dtype=torch.uint8)
    scales = torch.rand(N, K // group, generator=g, device="cuda").mul_(0.01).to(torch.bfloat16)
    w = Int4Weight(nib, scales, None, group, torch.bfloat16)
    x = torch.randn(5, K, generator=g, device="cuda").to(torch.bfloat16)
    first = int4_linear(x, w, gated_act="gelu_tanh" if gated else None)
    for _ in range(300):
        assert torch.equal(int4_linear(x, w, gated_act="gelu_tanh" if gated else None), first)
