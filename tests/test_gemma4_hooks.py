"""Hooks on the layers of a Gemma4 model whose norms run in fused form: they see what they saw before, each once per step, and a
stream that one of them replaces or changes in place is the stream that the next layer reads.  On the CPU the fused kernel is
restated with the separate norms, in 32 bits, so both forms agree to rounding; on the GPU both run in bf16 and differ by a few
roundings of a stream that six norms of a layer go through (2^-8 each)."""
import pytest
import torch

from litevllm_b200 import LLM, ops
from litevllm_b200.models.gemma4 import Gemma4Experts
from litevllm_b200.ops import stream_norms as sn
from litevllm_b200.ops.moe import RoutedRows


def _restated(h, eps, post, outs, y=None, branches=None):
    if branches is not None:
        routed, w_s, d, w_d = branches
        y = ops.rmsnorm(routed.combined().to(h.dtype), w_s, eps, addend=ops.rmsnorm(d, w_d, eps))
    new = ops.rmsnorm(y, post, eps, addend=h)
    return new, [ops.rmsnorm(new, w, eps, out_scale=s) for w, s in outs]


def _rows(self, x, ids, weights):
    T = x.shape[0]
    return RoutedRows(self(x, ids, weights), torch.ones(T, 1), torch.arange(T, dtype=torch.int32).view(T, 1))


@pytest.fixture(scope="module", params=["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
def llm(request):
    if request.param == "cpu":
        return LLM("synthetic:tiny-gemma4-moe-test", dtype="float32", device="cpu", max_num_seqs=2, max_model_len=64)
    return LLM("synthetic:tiny-gemma4-moe-test", dtype="bfloat16", device="cuda:0", max_num_seqs=2, max_model_len=64)


def _logits(llm, fused):
    with pytest.MonkeyPatch.context() as mp:
        if not fused:
            mp.setattr(sn, "takes", lambda h, *w: False)
        elif llm.engine.device.type == "cpu":
            mp.setattr(sn, "takes", lambda h, *w: True)
            mp.setattr(sn, "stream_norms", _restated)
            mp.setattr(Gemma4Experts, "rows", _rows)
        return llm.engine.replay_step([("r", list(range(3, 22)), [0, 7, 18])], ["r"]).float().cpu()


def _add_one(h):
    return h + 1.0


def _in_place(h):
    h.add_(1.0)


def _places(model):
    first, second = model.layers[0], model.layers[1]

    def after(change):
        return lambda m, args, out: change(out)

    def before(change):
        def hook(m, args):
            y = change(args[0])
            return None if y is None else (y, *args[1:])
        return hook
    return {
        "none": lambda: [],
        "after a layer": lambda: [first.register_forward_hook(after(_add_one))],
        "after a layer, in place": lambda: [first.register_forward_hook(after(_in_place))],
        "before a layer": lambda: [second.register_forward_pre_hook(before(_add_one))],
        "before a layer, in place": lambda: [second.register_forward_pre_hook(before(_in_place))],
        "after the first norm": lambda: [second.input_layernorm.register_forward_hook(after(_add_one))],
        "before the first norm": lambda: [second.input_layernorm.register_forward_pre_hook(before(_add_one))],
        "after an inner norm": lambda: [second.pre_feedforward_layernorm.register_forward_hook(after(_add_one))],
        "after the experts": lambda: [m.experts.register_forward_hook(after(_add_one)) for m in (first, second)],
        "after the shared branch": lambda: [second.shared_mlp.register_forward_hook(after(_add_one))],
    }


@pytest.mark.parametrize("place", ["none", "after a layer", "after a layer, in place", "before a layer", "before a layer, in place",
                                   "after the first norm", "before the first norm", "after an inner norm", "after the experts",
                                   "after the shared branch"])
def test_a_changed_stream_reaches_the_next_layer(llm, place):
    handles = _places(llm.engine.model)[place]()
    try:
        fused, plain = _logits(llm, True), _logits(llm, False)
    finally:
        for h in handles:
            h.remove()
    bound = 1e-5 if llm.engine.device.type == "cpu" else 2e-2
    assert (fused - plain).norm() <= bound * plain.norm()


def test_every_hook_is_called_once(llm):
    model = llm.engine.model
    calls = {}
    for i, layer in enumerate(model.layers):         # one layer at a time: its neighbours keep the fused form
        names = [n for n, m in layer.named_modules() if n]
        for fused in (True, False):
            handles = [layer.get_submodule(n).register_forward_hook(
                lambda m, args, out, key=(i, n, fused): calls.__setitem__(key, calls.get(key, 0) + 1)) for n in names]
            _logits(llm, fused)
            for h in handles:
                h.remove()
    assert {k[:2]: v for k, v in calls.items() if k[2]} == {k[:2]: v for k, v in calls.items() if not k[2]}
    assert all((i, "input_layernorm", True) in calls for i in range(len(model.layers)))


def test_hooks_on_all_modules(llm):
    def count(fused):
        seen = []
        handle = torch.nn.modules.module.register_module_forward_hook(lambda m, args, out: seen.append(type(m).__name__))
        try:
            _logits(llm, fused)
        finally:
            handle.remove()
        return sorted(seen)
    assert count(True) == count(False)


def test_a_replaced_forward_is_called(llm):
    norm, seen = llm.engine.model.layers[1].input_layernorm, []
    norm.forward = lambda x, out=None: seen.append(1) or type(norm).forward(norm, x, out)
    try:
        _logits(llm, True)
    finally:
        del norm.forward
    assert seen == [1]
