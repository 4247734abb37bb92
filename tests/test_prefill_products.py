"""Products of many tokens: every tile of the persistent kernel, and int4 weights through their expanded copy, at sizes that
end inside a tile.  Bound as in test_skinny_gemm.py: roundings of the result, relative to its spread."""
import pytest
import torch

from test_skinny_gemm import _close

pytestmark = pytest.mark.gpu
DEV = "cuda"


# on 148 SMs tiles of 256, 192, 160, 128, 96 and 64 tokens (all of them end inside a tile), the last with several groups of weight tiles
@pytest.mark.parametrize("T,N", [(2041, 2048), (1130, 2560), (2045, 2560), (1135, 2048), (599, 2048), (1999, 136), (257, 264), (1100, 6152)])
@pytest.mark.parametrize("extra", [False, True])
def test_persistent_tiles(T, N, extra):
    from litevllm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(T + N)
    K = 200
    x = torch.randn(T, K, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)
    ref = x.float() @ w.float().t()
    if extra:
        b = torch.randn(N, generator=g, device=DEV).to(torch.bfloat16)
        r = torch.randn(T, N, generator=g, device=DEV).to(torch.bfloat16)
        _close(ops.linear(x, w, bias=b, residual=r), ref + b.float() + r.float(), torch.bfloat16)
    else:
        _close(ops.linear(x, w), ref, torch.bfloat16)
        _close(ops.linear(x, w, out_dtype=torch.float32), ref, torch.float32)


@pytest.mark.parametrize("T,inter", [(1135, 2112), (1025, 136), (2048, 200)])
def test_persistent_gated_tiles(T, inter):
    from litevllm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randn(T, 320, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(2 * inter, 320, generator=g, device=DEV) * 320 ** -0.5).to(torch.bfloat16)
    y = x.float() @ w.float().t()
    _close(ops.gated_linear(x, w, "silu"), torch.nn.functional.silu(y[:, :inter]) * y[:, inter:], torch.bfloat16, 4.0)


@pytest.mark.parametrize("T", [129, 512, 777])
@pytest.mark.parametrize("N,K,group,zero", [(48, 192, 64, True), (2832, 704, 32, False), (4096, 1152, 128, True), (64, 1024, 256, False)])
@pytest.mark.parametrize("gated", [False, True])
def test_int4_of_many_tokens(T, N, K, group, zero, gated):
    from litevllm_b200.ops.awq import Int4Weight, dequantize, int4_linear
    g = torch.Generator(device=DEV).manual_seed(N + K + T)
    dtype = torch.float16 if zero else torch.bfloat16
    nib = torch.randint(0, 16, (N, K), generator=g, device=DEV, dtype=torch.uint8)
    scales = (torch.rand(N, K // group, generator=g, device=DEV) + 0.5).mul_(0.2 * K ** -0.5).to(dtype)
    zeros = torch.randint(5, 11, (N, K // group), generator=g, device=DEV, dtype=torch.uint8) if zero else None
    x = torch.randn(T, K, generator=g, device=DEV).to(dtype)
    y = x.float() @ dequantize(nib, scales, zeros, group).t()
    w = Int4Weight(nib, scales, zeros, group, dtype)
    if gated:
        ref = torch.nn.functional.gelu(y[:, :N // 2], approximate="tanh") * y[:, N // 2:]
        _close(int4_linear(x, w, gated_act="gelu_tanh"), ref, dtype, 4.0)
    else:
        r = torch.randn(T, N, generator=g, device=DEV).to(dtype)
        _close(int4_linear(x, w, residual=r), y + r.float(), dtype, 4.0)
