"""Products of few tokens from registers (csrc/gemm/skinny_gemm.cu) against fp32 sums of the same operands, at the edges of
its tiles (16 rows, 64 or 128 k per warp, 8 tokens), for every epilogue.  Bounds: one rounding of the result to 16 bits (2^-8
relative in bf16, 2^-11 in fp16) and, where int4 weights are rounded to 16 bits first, as much again relative to the sum of
magnitudes' root, which a factor of 2 of the result's spread covers for random signs."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _close(y, ref, dtype, roundings=2.0):
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -17}[dtype]
    spread = ref.abs().mean()
    assert torch.all((y.float() - ref).abs() <= roundings * eps * (ref.abs() + 4 * spread))


@pytest.mark.parametrize("T", [1, 3, 8])
@pytest.mark.parametrize("N,K", [(16, 64), (24, 192), (40, 576), (2560, 2048), (4744, 256)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_16_bit_with_norm(T, N, K, dtype):
    from litevllm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(T * N + K)
    x = torch.randn(T, K, generator=g, device=DEV).to(dtype)
    w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).to(dtype)
    b = torch.randn(N, generator=g, device=DEV).to(dtype)
    r = torch.randn(T, N, generator=g, device=DEV).to(dtype)

    def normed(v):
        return v.float() * torch.rsqrt(v.float().square().mean(-1, keepdim=True) + 1e-5)
    ref = normed(x) @ w.float().t()
    _close(ops.linear(x, w, rms_eps=1e-5), ref, dtype)
    _close(ops.linear(x, w, bias=b, residual=r, rms_eps=1e-5), ref + b.float() + r.float(), dtype)
    _close(ops.linear(x, w, rms_eps=1e-5, out_dtype=torch.float32), ref, torch.float32)
    wide = torch.randn(T + 1, 3 * K, generator=g, device=DEV).to(dtype)       # rows of a wider buffer
    _close(ops.linear(wide[1:, K:2 * K], w, rms_eps=1e-5), normed(wide[1:, K:2 * K]) @ w.float().t(), dtype)
    if N % 16 == 0:
        y = torch.nn.functional.silu(ref[:, :N // 2]) * ref[:, N // 2:]
        _close(ops.gated_linear(x, w, "silu", rms_eps=1e-5), y, dtype, 4.0)


@pytest.mark.parametrize("T", [1, 5, 8, 9, 16, 33, 64])
@pytest.mark.parametrize("N,K,group,zero", [(16, 64, 32, False), (48, 192, 64, True), (5136, 704, 32, False), (4096, 4096, 128, True),
                                            (64, 384, 128, True), (32, 576, 192, True), (48, 12288, 256, False)])
@pytest.mark.parametrize("gated", [False, True])
def test_int4(T, N, K, group, zero, gated):
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


@pytest.mark.parametrize("T,N,gated", [(8, 9616, False), (8, 4808, True), (9, 4912, False), (9, 4808, True), (12, 9616, False),
                                       (12, 6152, True), (16, 7200, False), (16, 6152, True)])
@pytest.mark.parametrize("group", [32, 128])
def test_int4_tokens_in_pieces_over_several_rounds(T, N, gated, group):
    """Tokens that do not fit shared memory in one piece and more tiles than CTAs: every round stages the pieces again, while
    the ring of weights runs on."""
    from litevllm_b200.ops import _lib
    from litevllm_b200.ops.awq import Int4Weight, dequantize, int4_linear
    g = torch.Generator(device=DEV).manual_seed(N + T)
    dtype, K, rows = torch.float16 if group == 128 else torch.bfloat16, 12288, 2 * N if gated else N
    assert _lib.kernels().fi_skinny_takes(1, 0, T, N, K, gated)
    nib = torch.randint(0, 16, (rows, K), generator=g, device=DEV, dtype=torch.uint8)
    scales = (torch.rand(rows, K // group, generator=g, device=DEV) + 0.5).mul_(0.2 * K ** -0.5).to(dtype)
    zeros = torch.randint(5, 11, (rows, K // group), generator=g, device=DEV, dtype=torch.uint8) if group == 128 else None
    x = torch.randn(T, K, generator=g, device=DEV).to(dtype)
    y = x.float() @ dequantize(nib, scales, zeros, group).t()
    w = Int4Weight(nib, scales, zeros, group, dtype)
    if gated:
        ref = torch.nn.functional.gelu(y[:, :N], approximate="tanh") * y[:, N:]
        _close(int4_linear(x, w, gated_act="gelu_tanh"), ref, dtype, 4.0)
    else:
        _close(int4_linear(x, w), y, dtype, 4.0)


@pytest.mark.parametrize("T,E,K,H,inter", [(1, 8, 2, 128, 64), (3, 16, 4, 2816, 704), (40, 8, 2, 256, 96 * 2), (33, 128, 8, 192, 64), (11, 2, 2, 4096, 4096)])
def test_experts_of_few_rows(T, E, K, H, inter):
    """Tables of 8- and 16-row tiles, experts with more rows than a tile and with none, K that ends inside a chunk."""
    from litevllm_b200.ops import moe
    from litevllm_b200.ops.awq import Int4Weight
    g = torch.Generator(device=DEV).manual_seed(T + E)

    def weight(rows, cols):
        nib = torch.randint(0, 16, (rows, cols), generator=g, device=DEV, dtype=torch.uint8)
        s = (torch.rand(rows, cols // 32, generator=g, device=DEV) + 0.5).mul_(0.2 * cols ** -0.5).to(torch.bfloat16)
        return Int4Weight(nib, s, None, 32, torch.bfloat16)
    gu, dn = weight(E * 2 * inter, H), weight(E * H, inter)
    x = torch.randn(T, H, generator=g, device=DEV).to(torch.bfloat16)
    score = torch.rand(T, E, generator=g, device=DEV)
    score[:, 0] += 0.4                                   # one crowded expert
    ids = score.topk(K).indices.int()
    wts = torch.rand(T, K, generator=g, device=DEV)
    got = moe.fused_experts(x, gu, dn, ids, wts, E, 0, "gelu_tanh")
    ref = moe._reference_experts(x, gu, dn, ids, wts, E, 0, E, "gelu_tanh").float()
    _close(got, ref, torch.bfloat16, 6.0)


# experts of few rows: eight, four, two warps and one per tile of their up products, one for two tiles; groups of a chunk and shorter ones
@pytest.mark.gpu
@pytest.mark.parametrize("group", [32, 128])
@pytest.mark.parametrize("T,E,K", [(1, 4, 2), (1, 8, 8), (2, 32, 8), (3, 32, 8), (5, 64, 8)])
def test_warps_of_an_experts_tile(T, E, K, group):
    from litevllm_b200 import ops
    from litevllm_b200.ops import moe
    from litevllm_b200.ops.awq import Int4Weight
    H, inter, dtype = 256, 768, torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(T + E)

    def weight(rows, cols):
        nib = torch.randint(0, 16, (rows, cols), generator=g, device="cuda", dtype=torch.uint8)
        s = (torch.rand(rows, cols // group, generator=g, device="cuda") + 0.5).mul_(0.2 * cols ** -0.5).to(dtype)
        z = torch.randint(4, 12, (rows, cols // group), generator=g, device="cuda", dtype=torch.uint8)
        return Int4Weight(nib, s, z, group, dtype)
    gu, dn = weight(E * 2 * inter, H), weight(E * H, inter)
    x = torch.randn(T, H, generator=g, device="cuda").to(dtype)
    ids = torch.rand(T, E, generator=g, device="cuda").topk(K).indices.int()
    wts = torch.rand(T, K, generator=g, device="cuda")
    assert not moe._tmem_pays(T * K, E)
    got = moe.fused_experts(x, gu, dn, ids, wts, E, 0, "gelu_tanh").float()
    ops.check_status(x.device)
    ref = moe._reference_experts(x, gu, dn, ids, wts, E, 0, E, "gelu_tanh").float()
    # weights, gated activations, rows and the sum are rounded to 16 bits, half an ulp each
    assert (got - ref).norm() <= 2 * 2.0 ** -8 * ref.norm()
    assert (got - ref).abs().max() <= 8 * 2.0 ** -8 * ref.abs().max()
