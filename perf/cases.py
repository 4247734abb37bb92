"""What is timed on the engine: single steps of three decoder configurations, prompts and decoding apart.

A case is one step of the engine as ``LiteEngine.step`` takes it for a set of running requests: the prefill executor over
whole prompts or a later portion of one, or the decode executor over one token per request.  Both return the logits of
every request's last token.  The executors leave a request's length to their caller, so a step may be repeated.

The configurations are this repository's presets at full width:

* ``tinyllama-1.1b``, all 22 layers, 16-bit weights and cache;
* ``dense-9b-awq``, 12 of its 36 equal layers, int4 weights with zero points in groups of 128;
* ``gemma4-26b-a4b``, 6 of its 30 layers (one period of five window layers and a global one), symmetric int4 weights in
  groups of 32, 128 experts of which 8 run for a token, fp8 cache.

Weights are random.  Three of their properties are set rather than left to chance.  What a layer adds to the stream is small
beside it (the writing projections or the norms behind them are scaled down, and the embedding is not small): trained layers
refine a stream and do not replace it, and the rounding of one layer does not grow through the next.  Codes and zero points of the int4 weights
follow a normal distribution around the zero point, as quantised trained weights do.  The router of the mixture reads
channels that the layers do not write, in which every token names its experts by clear margins: a trained router's choices
do not hang on the last bit of a 16-bit stream either, and any two correct implementations run the same experts.
"""
from __future__ import annotations

import gc
import math

import torch

from litevllm_b200.config.config_builder import build_vllm_config
from litevllm_b200.engine.lite_engine import LiteEngine
from litevllm_b200.engine.step_plan import PrefillItem
from litevllm_b200.models.presets import get_preset
from litevllm_b200.models.registry import ModelRegistry

LLAMA, DENSE, MIXTURE = "tinyllama-1.1b", "dense-9b-awq", "gemma4-26b-a4b"
_SEATS = {LLAMA: 32, DENSE: 16, MIXTURE: 32}          # requests an engine of the model is set up for
_LAYERS = {LLAMA: 22, DENSE: 12, MIXTURE: 6}
_PROMPT_TOKENS = {LLAMA: 4096, DENSE: 2048, MIXTURE: 2048}      # tokens of the largest prefill step
_CONTEXT = {LLAMA: 2047, DENSE: 2047, MIXTURE: 1535}            # longest context of a drawn decode step


def _case(name: str, model: str, step: str, lens, past: int = 0, dtype: str = "bfloat16") -> dict:
    case = {"model": model, "layers": _LAYERS[model], "dtype": dtype, "step": step,
            "lens": ",".join(str(n) for n in lens), "past": past}
    return {"name": name, **case} if name else case


def _lens(case: dict) -> list[int]:
    return [int(n) for n in str(case["lens"]).split(",")]


def listed() -> list[dict]:
    return [
        # a chat turn of a few words reaches an idle server: what the user waits for is this one step
        _case("llama-prompt-37", LLAMA, "prefill", [37]),
        # requests of ordinary length that arrived together
        _case("llama-prompts-ragged", LLAMA, "prefill", [113, 257, 64, 511, 190]),
        # the headline benchmark's prompts, two to a step
        _case("llama-prompts-2x1024", LLAMA, "prefill", [1024, 1024]),
        # the second portion of a long document
        _case("llama-document-portion", LLAMA, "prefill", [2048], past=2000),
        # one user, short context: the smallest step there is
        _case("llama-decode-1", LLAMA, "decode", [131]),
        # the headline benchmark: 32 requests between 1024 and 2048 tokens
        _case("llama-decode-32", LLAMA, "decode", [1024 + (i * 613) % 1009 for i in range(32)]),
        # a prompt of the int4 benchmark
        _case("dense-prompt-2048", DENSE, "prefill", [2048]),
        # three users of the int4 model, in fp16 as such checkpoints ship
        _case("dense-decode-3", DENSE, "decode", [517, 70, 1291], dtype="float16"),
        # the int4 benchmark: 16 requests around 2048 tokens
        _case("dense-decode-16", DENSE, "decode", [1800 + (i * 101) % 248 for i in range(16)]),
        # prompts of the mixture's benchmark, two to a step
        _case("mixture-prompts-2x384", MIXTURE, "prefill", [384, 384]),
        # the mixture's benchmark with one request and with 32
        _case("mixture-decode-1", MIXTURE, "decode", [391]),
        _case("mixture-decode-32", MIXTURE, "decode", [384 + (i * 7) % 24 for i in range(32)]),
    ]


def _log_uniform(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng) -> dict:
    """Steps of the same models: any mix of prompt lengths up to the largest listed step, any number of decoding requests
    up to the seats of the engine at contexts up to the listed ones."""
    model = rng.choice([LLAMA, DENSE, MIXTURE])
    dtype = rng.choice(["bfloat16", "float16"]) if model != MIXTURE else "bfloat16"
    if rng.random() < 0.5:
        tokens = _log_uniform(rng, 16, _PROMPT_TOKENS[model] // 2)
        n = min(rng.choice([1, 1, 2, 3, 5, 8]), tokens // 8)
        weights = [rng.uniform(0.3, 1.0) for _ in range(n)]
        lens = [max(1, int(tokens * w / sum(weights))) for w in weights]
        past = rng.randint(16, 1000) if n == 1 and rng.random() < 0.3 else 0
        return _case("", model, "prefill", lens, past, dtype)
    n = _log_uniform(rng, 1, _SEATS[model])
    longest = _log_uniform(rng, 24, _CONTEXT[model])
    if n * longest > 32 * 1500:
        longest = 32 * 1500 // n
    return _case("", model, "decode", [rng.randint(longest // 2, longest) for _ in range(n)], 0, dtype)


# ---------------------------------------------------------------------------------------------------- weights
class _Weights:
    """The random checkpoint of a case: tensors by name, each from the seed and its own place in the order."""

    def __init__(self, case: dict, seed: int):
        cfg = get_preset(case["model"])
        self.cfg = cfg.get("text_config", cfg)
        self.model, self.layers, self.seed = case["model"], int(case["layers"]), seed
        self.dtype = getattr(torch, case["dtype"])
        self.hidden, self.vocab = self.cfg["hidden_size"], self.cfg["vocab_size"]
        self.heads, self.kv = self.cfg["num_attention_heads"], self.cfg["num_key_value_heads"]
        self.hd = self.cfg.get("head_dim") or self.hidden // self.heads
        self.inter = self.cfg["intermediate_size"]
        self.eps = self.cfg["rms_norm_eps"]
        self.group = {LLAMA: 0, DENSE: 128, MIXTURE: 32}[self.model]
        self.mixture = self.model == MIXTURE
        self.experts, self.top = self.cfg.get("num_experts", 0), self.cfg.get("top_k_experts", 0)
        self.expert_inter = self.cfg.get("moe_intermediate_size", 0)
        self.quiet = 1.0 if self.mixture else (2 * self.layers) ** -0.5     # projections that write the stream

    def _gen(self, place: int) -> torch.Generator:
        g = torch.Generator(device="cuda")
        g.manual_seed(self.seed * 100003 + place)
        return g

    def normal(self, place: int, *shape, std: float = 0.02, base: float = 0.0) -> torch.Tensor:
        x = torch.empty(*shape, dtype=torch.float32, device="cuda").normal_(base, std, generator=self._gen(place))
        return x.to(self.dtype)

    def int4(self, place: int, rows: int, cols: int, size: float = 1.0) -> dict:
        """Packed codes (nibble j of a word is column 8w + j), scales, and zero points where the format has them."""
        g = self._gen(place)
        code = torch.empty(rows, cols, dtype=torch.float16, device="cuda").normal_(0.0, 2.2, generator=g).round_()
        zero = None
        if self.model == DENSE:
            zero = torch.randint(6, 10, (rows, cols // self.group), generator=g, device="cuda", dtype=torch.int32)
            code = code.view(rows, -1, self.group) + zero[:, :, None].to(torch.float16)
        else:
            code = code + 8
        code = code.clamp_(0, 15).to(torch.int32).view(rows, cols // 8, 8)
        scale = torch.rand(rows, cols // self.group, generator=g, device="cuda").mul_(0.006 * size).add_(0.006 * size).to(self.dtype)
        out = {"weight_packed": _pack(code), "weight_scale": scale}
        if zero is not None:
            out["qzeros"] = _pack(torch.nn.functional.pad(zero, (0, -zero.shape[1] % 8)).view(rows, -1, 8))
            out["qweight"], out["scales"] = out.pop("weight_packed"), out.pop("weight_scale")
        return out

    def linear(self, place: int, name: str, rows: int, cols: int, size: float = 1.0):
        if not self.group:
            yield name + ".weight", self.normal(place, rows, cols, std=0.02 * size)
        else:
            for suffix, t in self.int4(place, rows, cols, size).items():
                yield f"{name}.{suffix}", t

    def embedding(self) -> torch.Tensor:
        e = self.normal(1, self.vocab, self.hidden, std=0.02 if self.mixture else 1.0)
        if self.mixture:      # channel i of the first ones: how much the token asks for expert i
            want = torch.empty(self.vocab, self.experts, device="cuda").normal_(0.0, 0.001, generator=self._gen(2))
            who = torch.rand(self.vocab, self.experts, generator=self._gen(3), device="cuda").topk(self.top).indices
            want.scatter_(1, who, torch.linspace(0.02, 0.04, self.top, device="cuda").expand(self.vocab, -1))
            e[:, :self.experts] = want.to(self.dtype)
        return e

    def norm(self, place: int, writes_stream: bool = False) -> torch.Tensor:
        if not (writes_stream and self.mixture):
            return self.normal(place, self.hidden, std=0.1, base=1.0)
        w = self.normal(place, self.hidden, std=0.01, base=0.1)
        w[:self.experts] = 0
        return w

    def layer(self, i: int):
        """(name, tensor) of layer i."""
        p, at = f"model.layers.{i}.", 100 * (i + 1)
        q, k, H = self.heads * self.hd, self.kv * self.hd, self.hidden
        yield from self.linear(at, p + "self_attn.q_proj", q, H)
        yield from self.linear(at + 1, p + "self_attn.k_proj", k, H)
        yield from self.linear(at + 2, p + "self_attn.v_proj", k, H)
        yield from self.linear(at + 3, p + "self_attn.o_proj", H, q, self.quiet)
        mlp = p + ("mlp.shared_mlp." if self.mixture else "mlp.")
        yield from self.linear(at + 4, mlp + "gate_proj", self.inter, H)
        yield from self.linear(at + 5, mlp + "up_proj", self.inter, H)
        yield from self.linear(at + 6, mlp + "down_proj", H, self.inter, self.quiet)
        yield p + "input_layernorm.weight", self.norm(at + 7)
        yield p + "post_attention_layernorm.weight", self.norm(at + 8, writes_stream=True)      # the mixture's stands behind o
        if not self.mixture:
            return
        for j, n in enumerate(("pre_feedforward_layernorm", "pre_feedforward_layernorm_2", "post_feedforward_layernorm_1",
                               "post_feedforward_layernorm_2", "post_feedforward_layernorm")):
            yield p + n + ".weight", self.norm(at + 9 + j, writes_stream=n == "post_feedforward_layernorm")
        yield p + "self_attn.q_norm.weight", self.normal(at + 14, self.hd, std=0.01, base=0.1)
        yield p + "self_attn.k_norm.weight", self.normal(at + 15, self.hd, std=0.1, base=1.0)
        E, I = self.experts, self.expert_inter
        proj = self.normal(at + 16, E, H)
        proj[:, :E] = 0
        proj[torch.arange(E, device="cuda"), torch.randperm(E, generator=self._gen(at + 17), device="cuda")] = 1
        scale = torch.zeros(H, dtype=self.dtype, device="cuda")
        scale[:E] = 3 * H ** 0.5
        yield p + "mlp.router.proj.weight", proj
        yield p + "mlp.router.scale", scale
        for j, (which, rows, cols) in enumerate((("gate_up_proj", 2 * I, H), ("down_proj", H, I))):
            for suffix, t in self.int4(at + 18 + j, E * rows, cols).items():
                yield f"{p}mlp.experts.{which}.{suffix}", t.view(E, rows, -1)

    def checkpoint(self):
        yield "model.embed_tokens.weight", self.embedding()
        for i in range(self.layers):
            yield from self.layer(i)
        yield "model.norm.weight", self.norm(4)
        if not self.mixture:
            yield "lm_head.weight", self.normal(5, self.vocab, self.hidden)

    def tokens(self, case: dict) -> list[list[int]]:
        """Per request the tokens of its context and this step; a decode step's own token is the last one."""
        g = torch.Generator().manual_seed(self.seed * 7 + 1)
        more = int(case["past"]) if case["step"] == "prefill" else 1
        return [torch.randint(0, self.vocab, (n + more,), generator=g).tolist() for n in _lens(case)]


def _pack(code: torch.Tensor) -> torch.Tensor:
    word = code[..., 0].clone()
    for j in range(1, 8):
        word |= code[..., j] << (4 * j)
    return word


# ---------------------------------------------------------------------------------------------------- the step
def _engine(case: dict, w: _Weights) -> LiteEngine:
    longest = max(_lens(case)) + int(case["past"]) + 1
    cut = {"num_hidden_layers": w.layers}
    cfg = build_vllm_config("synthetic:" + case["model"], dtype=case["dtype"], device="cuda:0",
                            max_model_len=2112 if longest <= 2112 else 4160, max_num_seqs=_SEATS[case["model"]],
                            max_num_batched_tokens=4096, hf_overrides={"text_config": cut} if w.mixture else cut)
    arch = cfg.model_config.arch
    with torch.device("cuda:0"):
        model = ModelRegistry.resolve_model_cls(arch.architecture, arch.family)(cfg)
    model.load_weights(w.checkpoint())
    model.eval()
    engine = LiteEngine(cfg, model=model)
    gc.unfreeze()         # engines come and go here: one that is dropped has to give its memory back
    return engine


def prepare(case: dict, seed: int) -> dict:
    """An engine with its weights laid out, whose requests have everything before this step in the cache."""
    w = _Weights(case, seed)
    engine = _engine(case, w)
    texts = w.tokens(case)
    ids = [f"r{i}" for i in range(len(texts))]
    prefill = case["step"] == "prefill"
    done = [int(case["past"]) if prefill else len(t) - 1 for t in texts]
    group, held = [], 0
    for rid, text, n in zip(ids, texts, done):
        if held + n > 4096 and group:
            engine.replay_step(group)
            group, held = [], 0
        group.append((rid, text[:n], []))
        held += n
    engine.replay_step(group)
    requests = engine.scheduler.requests
    state = {"engine": engine, "n": len(ids), "requests": [requests[r] for r in ids]}
    if prefill:
        engine.replay_step([(rid, text[n:], []) for rid, text, n in zip(ids, texts, done)])
        state["items"] = [PrefillItem(rid, n, len(text) - n) for rid, text, n in zip(ids, texts, done)]
    else:
        for st, text in zip(state["requests"], texts):
            st.generated_ids.append(text[-1])
            engine.kv_manager.ensure_blocks(st.request_id, len(text))
    run(state)            # the engine has served such a step before: its graph and scratch exist
    return state


def run(state: dict) -> torch.Tensor:
    engine = state["engine"]
    if "items" in state:
        return engine.prefill_executor.execute(state["items"], engine.scheduler.requests).logits
    return engine.decode_executor.execute_batch(state["requests"], engine.scheduler.requests).logits[:state["n"]]


# ---------------------------------------------------------------------------------------------------- what it needs
def work(case: dict) -> dict:
    """Weights of the matrices that are used, cached keys and values, token ids in and logits out; two operations per weight
    and token, attention over the positions each token sees."""
    w = _Weights(case, 0)
    lens, past = _lens(case), int(case["past"])
    prefill = case["step"] == "prefill"
    tokens = sum(lens) if prefill else len(lens)
    seen = [(past + (n + 1) / 2) * n if prefill else n + 1.0 for n in lens]
    if w.mixture:
        window = w.cfg["sliding_window"]
        near = [s if (past + n if prefill else n + 1) <= window else s * window / (past + n if prefill else n + 1)
                for s, n in zip(seen, lens)]
    else:
        near = seen
    q, k, H = w.heads * w.hd, w.kv * w.hd, w.hidden
    matrix = H * (2 * q + 2 * k) + 3 * H * w.inter
    bits = 16.0 if not w.group else 4 + 16.0 / w.group + (4.0 / w.group if w.model == DENSE else 0.0)
    used, active = float(matrix), float(matrix)
    if w.mixture:
        expert = 3 * H * w.expert_inter
        used += expert * w.experts * (1 - (1 - w.top / w.experts) ** tokens)
        active += expert * w.top
    router = H * w.experts
    kv_elem = 1 if w.mixture else 2
    size, flops = 0.0, 0.0
    for i in range(w.layers):
        pos = near if w.mixture and (i + 1) % w.cfg["sliding_window_pattern"] else seen
        rows = [(past + n) + n if prefill else p + 1 for n, p in zip(lens, pos)]       # read once, new ones written
        size += used * bits / 8 + 2 * router + 2 * k * kv_elem * sum(rows)
        flops += 2 * tokens * (active + router) + 4 * q * sum(pos)
    size += 2 * w.vocab * H + 2 * tokens * H + 8 * tokens + 4 * w.vocab * len(lens)
    flops += 2 * w.vocab * H * len(lens)
    return {"bytes": size, "flops": flops}


def tolerance(case: dict) -> dict:
    """16-bit activations between the kernels of up to 22 layers, e4m3 keys and values in the mixture: 1.1 to 1.3 % off the
    64-bit results in bf16 with every size tried, 0.15 to 0.18 % in fp16."""
    if case["dtype"] == "float16":
        return {"rel": 0.006, "max": 0.06}
    return {"rel": 0.03, "max": 0.3}


# ---------------------------------------------------------------------------------------------------- in 64 bits
def _norm(x, weight, eps):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight.double()


def _rotate(x, theta):
    """x [T, heads, d] of one request from position 0: pairs (j, j + d/2) turn by position * theta^(-2j/d)."""
    half = x.shape[-1] // 2
    inv = theta ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half)
    ang = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None] * inv
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _dense(t: dict, name: str, w: _Weights) -> torch.Tensor:
    if name + ".weight" in t:
        return t[name + ".weight"].double()
    packed, scale = (t[f"{name}.qweight"], t[f"{name}.scales"]) if w.model == DENSE else \
        (t[f"{name}.weight_packed"], t[f"{name}.weight_scale"])
    zero = _unpack(t[name + ".qzeros"])[..., :scale.shape[-1], None] if w.model == DENSE else 8
    code = _unpack(packed).view(*scale.shape, w.group)
    return ((code - zero).double() * scale.double()[..., None]).flatten(-2)


def _unpack(words: torch.Tensor) -> torch.Tensor:
    return torch.stack([(words >> (4 * j)) & 15 for j in range(8)], -1).flatten(-2)


def _attend(q, k, v, scale, window, softcap, first):
    """One request: q, k, v [T, heads, d]; rows of the positions from ``first`` on."""
    T, group = q.shape[0], q.shape[1] // k.shape[1]
    out = torch.empty(T - first, q.shape[1], v.shape[2], dtype=q.dtype, device=q.device)
    keys = torch.arange(T, device=q.device)
    for lo in range(first, T, 1024):
        hi = min(T, lo + 1024)
        rows = keys[lo:hi, None]
        hidden = (keys > rows) | (keys <= rows - window) if window else keys > rows
        for h in range(k.shape[1]):
            s = torch.einsum("thd,sd->hts", q[lo:hi, h * group:(h + 1) * group], k[:, h]) * scale
            if softcap:
                s = torch.tanh(s / softcap) * softcap
            s = s.masked_fill(hidden, float("-inf")).softmax(-1)
            out[lo - first:hi - first, h * group:(h + 1) * group] = torch.einsum("hts,sd->thd", s, v[:, h])
    return out


def _gated(x, gate, up, down, act):
    return (act(x @ gate.T) * (x @ up.T)) @ down.T


@torch.inference_mode()
def exact(case: dict, seed: int) -> torch.Tensor:
    """The whole contexts in one pass without a cache."""
    w = _Weights(case, seed)
    texts = w.tokens(case)
    sizes = [len(t) for t in texts]
    ends = torch.tensor(sizes, device="cuda").cumsum(0) - 1
    ids = torch.tensor([t for text in texts for t in text], device="cuda")
    embedding = w.embedding()
    h = embedding[ids].double()
    cap_attn = float(w.cfg.get("attn_logit_softcapping") or 0.0)
    act = (lambda x: torch.nn.functional.gelu(x, approximate="tanh")) if w.mixture else torch.nn.functional.silu
    if w.mixture:
        h *= w.hidden ** 0.5
    for i in range(w.layers):
        p = f"model.layers.{i}."
        t = dict(w.layer(i))
        local = w.mixture and (i + 1) % w.cfg["sliding_window_pattern"] != 0
        theta = float(w.cfg["rope_theta"]) if not w.mixture else \
            float(w.cfg["rope_local_base_freq" if local else "rope_global_base_freq"])
        x = _norm(h, t[p + "input_layernorm.weight"], w.eps)
        q, k, v = ((x @ _dense(t, f"{p}self_attn.{n}_proj", w).T).view(len(ids), -1, w.hd) for n in "qkv")
        if w.mixture:
            q = _norm(q, t[p + "self_attn.q_norm.weight"], w.eps)
            k = _norm(k, t[p + "self_attn.k_norm.weight"], w.eps)
            v = _norm(v, None, w.eps)
        a, lo = [], 0
        for n in sizes:
            ks, vs = _rotate(k[lo:lo + n], theta), v[lo:lo + n]
            if w.mixture:         # the cache holds e4m3
                ks, vs = ks.float().to(torch.float8_e4m3fn).double(), vs.float().to(torch.float8_e4m3fn).double()
            a.append(_attend(_rotate(q[lo:lo + n], theta), ks, vs, 1.0 if w.mixture else w.hd ** -0.5,
                             w.cfg["sliding_window"] if local else 0, cap_attn, 0).flatten(1))
            lo += n
        del q, k, v
        y = torch.cat(a) @ _dense(t, p + "self_attn.o_proj", w).T
        if not w.mixture:
            h = h + y
            x = _norm(h, t[p + "post_attention_layernorm.weight"], w.eps)
            h = h + _gated(x, *(_dense(t, f"{p}mlp.{n}_proj", w) for n in ("gate", "up", "down")), act)
            continue
        h = h + _norm(y, t[p + "post_attention_layernorm.weight"], w.eps)
        x = _norm(h, t[p + "pre_feedforward_layernorm.weight"], w.eps)
        y = _gated(x, *(_dense(t, f"{p}mlp.shared_mlp.{n}_proj", w) for n in ("gate", "up", "down")), act)
        y = _norm(y, t[p + "post_feedforward_layernorm_1.weight"], w.eps)
        score = (_norm(h, t[p + "mlp.router.scale"], w.eps) * w.hidden ** -0.5) @ t[p + "mlp.router.proj.weight"].double().T
        part, who = score.softmax(-1).topk(w.top)
        part = part / part.sum(-1, keepdim=True)
        x = _norm(h, t[p + "pre_feedforward_layernorm_2.weight"], w.eps)
        sparse = torch.zeros_like(h)
        for e in range(w.experts):
            row, slot = torch.nonzero(who == e, as_tuple=True)
            gate_up = _dense({n: s[e] for n, s in t.items() if ".experts.gate_up" in n}, p + "mlp.experts.gate_up_proj", w)
            down = _dense({n: s[e] for n, s in t.items() if ".experts.down" in n}, p + "mlp.experts.down_proj", w)
            sparse[row] += part[row, slot, None] * _gated(x[row], *gate_up.chunk(2), down, act)
        y = y + _norm(sparse, t[p + "post_feedforward_layernorm_2.weight"], w.eps)
        h = h + _norm(y, t[p + "post_feedforward_layernorm.weight"], w.eps)
    x = _norm(h[ends], w.norm(4), w.eps)
    logits = x @ (embedding if w.mixture else w.normal(5, w.vocab, w.hidden)).double().T
    cap = float(w.cfg.get("final_logit_softcapping") or 0.0)
    return torch.tanh(logits / cap) * cap if cap else logits
