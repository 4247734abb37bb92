"""Prefill attention of heads of 256 channels on an e4m3 cache (csrc/attn/prefill_fp8.cu) against a 64-bit oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# new tokens and cached ones per sequence: query tiles that end inside, of one row, full; one key tile, an edge of one, many
MIXED = [(130, 0), (129, 500), (1, 700), (128, 0), (64, 333), (63, 1)]


@pytest.mark.parametrize("lens,nh,nkv,bs,window,softcap,dtype", [
    (MIXED, 16, 8, 16, 0, 50.0, torch.bfloat16), (MIXED, 4, 1, 32, 70, 50.0, torch.float16), (MIXED, 6, 2, 64, 200, 0.0, torch.bfloat16),
    (MIXED, 2, 2, 128, 0, 0.0, torch.float16), (MIXED, 8, 4, 24, 0, 30.0, torch.bfloat16),       # pages of 24: the general kernel
    ([(1, 0)], 2, 1, 16, 0, 0.0, torch.bfloat16), ([(32, 32)] * 9, 16, 8, 16, 0, 0.0, torch.bfloat16),
    ([(32, 32)] * 10, 16, 8, 16, 0, 0.0, torch.bfloat16), ([(33, 31)] * 10, 16, 8, 16, 40, 0.0, torch.bfloat16)])   # both sides of the rule
def test_prefill_of_wide_heads_on_e4m3_caches(lens, nh, nkv, bs, window, softcap, dtype):
    from litevllm_b200 import ops
    hd, ks, vs = 256, 0.75, 1.25
    g = torch.Generator(device=DEV).manual_seed(nh + bs)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    totals = [n + past for n, past in lens]
    B, per = len(lens), (max(totals) + bs - 1) // bs
    raw = [rnd(B * per + 1, nkv, bs, hd).to(torch.float8_e4m3fn).view(torch.uint8) for _ in range(2)]
    bt = (torch.randperm(B * per, generator=g, device=DEV) + 1).view(B, per).int()
    for c in raw:                           # NaN in the null page and behind the last key of every sequence
        c[0] = 0x7f
        for b, n in enumerate(totals):
            for pos in range(n, per * bs):
                c[bt[b, pos // bs].long(), :, pos % bs] = 0x7f
    kc, vc = (c.view(torch.float8_e4m3fn) for c in raw)
    cu = torch.tensor([0] + [n for n, _ in lens], device=DEV).cumsum(0).int()
    sl = torch.tensor(totals, device=DEV, dtype=torch.int32)
    T, scale = int(cu[-1]), hd ** -0.5
    q = rnd(T, (nh + 2 * nkv) * hd).to(dtype)
    got = ops.paged_attention_prefill(q, kc, vc, bt, sl, cu, max(n for n, _ in lens), nh, nkv, hd, scale, window, softcap, ks, vs)
    ops.check_status(torch.device(DEV, 0))
    got = got.double().view(T, nh, hd)
    worst = 0.0
    for b, (n, past) in enumerate(lens):
        lo = int(cu[b])
        k, v = (c[bt[b].long()].double().permute(1, 0, 2, 3).reshape(nkv, per * bs, hd)[:, :n + past] * f for c, f in ((kc, ks), (vc, vs)))
        s = torch.einsum("tkgd,ksd->kgts", q[lo:lo + n, :nh * hd].view(n, nkv, nh // nkv, hd).double(), k) * scale
        if softcap:
            s = torch.tanh(s / softcap) * softcap
        pos, keys = torch.arange(past, past + n, device=DEV)[:, None], torch.arange(n + past, device=DEV)
        hidden = keys > pos
        if window:
            hidden |= keys <= pos - window
        w = s.masked_fill(hidden, float("-inf")).softmax(-1)
        ref = torch.einsum("kgts,ksd->tkgd", w, v).reshape(n, nh, hd)
        size = torch.einsum("kgts,ksd->tkgd", w, v.abs()).reshape(n, nh, hd)     # what the roundings of the weights act on
        # half an ulp for each weight, for their sum (of rounded weights) and for the result; scores of 32 bits: 2^-14 of a weight
        eps = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
        bound = eps * (size + 2 * ref.abs()) + 2.0 ** -14 * size + 1e-6
        worst = max(worst, float(((got[lo:lo + n] - ref).abs() / bound).max()))
    assert worst <= 1.0, worst
