"""The norms around a stream in one kernel (csrc/misc/stream_norms.cu) against the separate kernels.  Both round at the same
places and differ in the order of their 32-bit sums, which can move a value across one rounding boundary per stage: at most four
units in the last place of the largest term."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _near(a, b, dtype):
    ulp = {torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -10}[dtype]
    assert torch.all((a.float() - b.float()).abs() <= 4 * ulp * torch.maximum(b.float().abs(), b.float().abs().mean()))


@pytest.mark.parametrize("T,H", [(1, 8), (3, 264), (5, 2816), (33, 8192), (2, 16384)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("outs", [0, 1, 3])
@pytest.mark.parametrize("branches", [False, True])
def test_against_separate_kernels(T, H, dtype, outs, branches):
    from litevllm_b200 import ops
    from litevllm_b200.ops import stream_norms as sn
    from litevllm_b200.ops.moe import RoutedRows
    g = torch.Generator(device="cuda").manual_seed(T + H + outs)

    def rnd(*shape, base=0.0):
        return (torch.randn(*shape, generator=g, device="cuda") + base).to(dtype)
    h, post, eps = rnd(T, H), rnd(H, base=1.0), 1e-6
    want = [(rnd(H, base=1.0), 1.0 if i != 1 else H ** -0.5) for i in range(outs)]
    if branches:
        K = 3
        rows = rnd(T * K, H)
        slot = torch.randperm(T * K, generator=g, device="cuda").int().view(T, K)
        slot[0, 1] = -1
        w = torch.rand(T, K, generator=g, device="cuda")
        w_s, w_d, d = rnd(H, base=1.0), rnd(H, base=1.0), rnd(T, H + 8)[:, :H]
        routed = RoutedRows(rows, w, slot)
        s = routed.combined().to(dtype)
        y = ops.rmsnorm(s, w_s, eps, addend=ops.rmsnorm(d.contiguous(), w_d, eps))
        got, normed = sn.stream_norms(h, eps, post, want, branches=(routed, w_s, d, w_d))
    else:
        y = rnd(T, H)
        got, normed = sn.stream_norms(h, eps, post, want, y=y)
    ref = ops.rmsnorm(y, post, eps, addend=h)
    _near(got, ref, dtype)
    assert len(normed) == outs
    for n, (wt, scale) in zip(normed, want):
        _near(n, ops.rmsnorm(got, wt, eps, out_scale=scale), dtype)
