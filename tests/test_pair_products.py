"""Products of many tokens by CTA pairs (csrc/gemm/dense_gemm_pair.cu): every tile at sizes that end inside a tile, a half of a pair and a k-block."""
import pytest
import torch

from test_skinny_gemm import _close

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _pair(x, w, out, tokens, bias=None, residual=None, act=None, limit=0.0, gated=False):
    from litevllm_b200 import ops
    rc = ops._lib.kernels().fi_dense_gemm_pair(
        ops._p(x), ops._p(w), ops._p(out), ops._p(bias), ops._p(residual), x.shape[0], out.shape[1], x.shape[1], x.stride(0), w.stride(0),
        out.stride(0), ops._ACT[act], limit, out.shape[1] if gated else 0, 1 if out.dtype == torch.float32 else 0, ops._DT[x.dtype], tokens,
        ops._p(ops.status_word(x.device)), ops._stream())
    assert rc == 0
    ops.check_status(x.device)
    return out


# one tile and many per pair of SMs; tokens that end in either half of a tile, rows that end in either CTA of a pair
@pytest.mark.parametrize("tokens", [256, 192, 128])
@pytest.mark.parametrize("T,N,K,dtype", [(1, 8, 8, torch.bfloat16), (130, 264, 200, torch.float16), (257, 136, 72, torch.bfloat16),
                                         (385, 2056, 64, torch.float16), (2047, 2568, 136, torch.bfloat16)])
def test_pair_tiles(T, N, K, dtype, tokens):
    g = torch.Generator(device=DEV).manual_seed(T + N)
    x = torch.randn(T, K + 8, generator=g, device=DEV).to(dtype)[:, :K]
    w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).to(dtype)
    b, r = (torch.randn(*s, generator=g, device=DEV).to(dtype) for s in ((N,), (T, N)))
    ref = x.float() @ w.float().t()
    _close(_pair(x, w, torch.empty(T, N, dtype=dtype, device=DEV), tokens, b, r), ref + b.float() + r.float(), dtype)
    _close(_pair(x, w, torch.empty(T, N, dtype=torch.float32, device=DEV), tokens, b), ref + b.float(), torch.float32)
    inplace = r.clone()
    _close(_pair(x, w, inplace, tokens, None, inplace), ref + r.float(), dtype)


@pytest.mark.parametrize("tokens", [256, 192, 128])
@pytest.mark.parametrize("T,inter,K", [(1, 8, 64), (131, 72, 200), (300, 264, 64), (1100, 1416, 136)])
def test_pair_gated_tiles(T, inter, K, tokens):
    g = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randn(T, K, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(2 * inter, K, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)
    b = torch.randn(2 * inter, generator=g, device=DEV).to(torch.bfloat16)
    y = x.float() @ w.float().t() + b.float()
    gate, up = y[:, :inter], y[:, inter:]
    def empty():
        return torch.empty(T, inter, dtype=torch.bfloat16, device=DEV)
    _close(_pair(x, w, empty(), tokens, b, act="silu", gated=True), torch.nn.functional.silu(gate) * up, torch.bfloat16, 4.0)
    low, held = gate.clamp(max=1.5), up.clamp(-1.5, 1.5)
    _close(_pair(x, w, empty(), tokens, b, act="clipped_swiglu", limit=1.5, gated=True), low * torch.sigmoid(1.702 * low) * (held + 1),
           torch.bfloat16, 4.0)
