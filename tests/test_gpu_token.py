"""The projections of a cached token at the edges of their tiles, and the native token stack against the module path."""
import copy
import ctypes

import pytest
import torch
import torch.nn.functional as F
from torch.utils._python_dispatch import TorchDispatchMode

from solvedelta_b200 import SolveDeltaConfig, SolveDeltaForCausalLM, _lib
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,norm,delta,swiglu", [
    (1, 24, 8, False, False, False), (7, 2376, 264, True, True, False), (8, 2368, 2048, True, False, False),
    (9, 40, 2816, False, False, False), (16, 2384, 1000, False, False, False), (17, 8, 72, False, False, True),
    (32, 112, 1024, False, False, True), (3, 48, 1024, True, True, True),
    (9, 2376, 1024, True, True, False), (16, 48, 2048, True, False, True)])
def test_token_linear(M, N, K, norm, delta, swiglu):
    gen = torch.Generator().manual_seed(M * N + K)
    bf = lambda *s: torch.randn(*s, generator=gen).to(torch.bfloat16).cuda()
    x, d, w, b = bf(M, K), bf(M, K), bf(N, K) / K ** 0.5, bf(N)
    nw = (1 + 0.2 * torch.randn(K, generator=gen)).cuda()
    y = torch.full((M, N // 2 if swiglu else N), float("nan"), dtype=torch.bfloat16, device="cuda")
    total = torch.empty_like(x)
    a = _lib.TokenLinearArgs(M, N, K, int(swiglu), x.data_ptr(), K, w.data_ptr(), b.data_ptr(), y.data_ptr(), y.shape[1],
                             d.data_ptr() if delta else None, nw.data_ptr() if norm else None, 1e-6, 1, total.data_ptr())
    _lib.check(_lib.load().sd_token_linear(ctypes.byref(a),
                                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    rows = x
    if delta:
        rows = x + d
        assert torch.equal(total, rows)
    rows = rows.float()
    if norm:
        rows = (rows * torch.rsqrt(rows.pow(2).mean(-1, keepdim=True) + 1e-6) * nw).to(torch.bfloat16).float()
    want = rows @ w.float().t() + b.float()
    if swiglu:
        gate, value = want.to(torch.bfloat16).float().chunk(2, -1)
        want = F.silu(gate) * value
    assert rel_l2(y.float().cpu().numpy(), want.cpu().numpy()) <= 4e-3


@pytest.mark.parametrize("B", [1, 8, 9, 20])
def test_token_stack_equals_the_module_path(B):
    torch.manual_seed(5)
    model = SolveDeltaForCausalLM(SolveDeltaConfig(hidden_size=256, num_heads=4, head_k_dim=64, head_v_dim=64,
                                                   num_hidden_layers=2, vocab_size=320)).prepare("cuda").eval()
    ids = torch.randint(0, 320, (B, 70), device="cuda")
    seen = []
    for hooked in (False, True):
        handle = model.model.layers[1].mlp.register_forward_hook(lambda *a: None) if hooked else None
        with torch.no_grad():
            cache = model(input_ids=ids[:, :66], use_cache=True).past_key_values
            logits = [model(input_ids=ids[:, t:t + 1], past_key_values=cache, use_cache=True).logits for t in range(66, 70)]
        assert cache.get_seq_length() == 70
        seen.append((torch.cat(logits, 1), cache[1]["recurrent_state"][1].clone(), cache[1]["conv_state"].clone()))
        if handle is not None:
            handle.remove()
    for got, want in zip(*seen):
        assert rel_l2(got.float().cpu().numpy(), want.float().cpu().numpy()) <= 1e-2


@pytest.mark.parametrize("B,T", [(1, 33), (3, 70), (2, 129)])
def test_prompt_through_the_stack_equals_the_module_path(B, T):
    torch.manual_seed(6)
    model = SolveDeltaForCausalLM(SolveDeltaConfig(hidden_size=256, num_heads=4, head_k_dim=64, head_v_dim=64,
                                                   num_hidden_layers=2, vocab_size=320)).prepare("cuda").eval()
    ids = torch.randint(0, 320, (B, T), device="cuda")
    seen = []
    for hooked in (False, True):
        handle = model.model.layers[1].mlp.register_forward_hook(lambda *a: None) if hooked else None
        with torch.no_grad():
            bare = model(input_ids=ids, use_cache=False).logits
            out = model(input_ids=ids, use_cache=True)
        assert torch.equal(out.logits, bare)
        cache = out.past_key_values
        assert cache.get_seq_length() == T and len(cache) == 2
        seen.append((out.logits, *cache[1]["recurrent_state"], cache[1]["conv_state"]))
        if handle is not None:
            handle.remove()
    for got, want in zip(*seen):
        assert rel_l2(got.float().cpu().numpy(), want.float().cpu().numpy()) <= 1e-2


class _Dispatched(TorchDispatchMode):
    """The torch calls made below the Python layer, in order: name and result type."""

    def __init__(self):
        super().__init__()
        self.calls = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        out = func(*args, **(kwargs or {}))
        self.calls.append((func.overloadpacket.__name__, getattr(out, "dtype", None)))
        return out


@pytest.mark.parametrize("B", [1, 20])
def test_parameter_copies_precede_the_launches(B):
    """A chained launch reads its FP32 parameters while the kernel before it runs, so the copies that a parameter update
    has put out of date are all made ahead of the first launch (and with it of the workspace); the step then sees the
    new values."""
    torch.manual_seed(6)
    model = SolveDeltaForCausalLM(SolveDeltaConfig(hidden_size=256, num_heads=4, head_k_dim=64, head_v_dim=64,
                                                   num_hidden_layers=2, vocab_size=320)).prepare("cuda").eval()
    ids = torch.randint(0, 320, (B, 41), device="cuda")
    with torch.no_grad():
        cache = model(input_ids=ids[:, :40], use_cache=True).past_key_values
        same = copy.deepcopy(cache)
        for name, p in model.named_parameters():
            if "norm" in name or "conv_weight" in name:
                p.add_(0.25 * torch.randn_like(p))
        with _Dispatched() as log:
            got = model(input_ids=ids[:, 40:], past_key_values=cache, use_cache=True).logits
        model.model.layers[1].mlp.register_forward_hook(lambda *a: None)   # the module path
        want = model(input_ids=ids[:, 40:], past_key_values=same, use_cache=True).logits
    copies = [i for i, call in enumerate(log.calls) if call == ("_to_copy", torch.float32)]
    workspace = [i for i, call in enumerate(log.calls) if call == ("empty", torch.uint8)]
    assert len(copies) == 4 * 2 + 1 and len(workspace) == 1 and max(copies) < workspace[0]
    assert rel_l2(got.float().cpu().numpy(), want.float().cpu().numpy()) <= 1e-2


def test_parameter_copies_made_on_another_stream():
    """The copies that one stream is still making (behind a long kernel) are waited for on the other."""
    torch.manual_seed(7)
    model = SolveDeltaForCausalLM(SolveDeltaConfig(hidden_size=256, num_heads=4, head_k_dim=64, head_v_dim=64,
                                                   num_hidden_layers=2, vocab_size=320)).prepare("cuda").eval()
    ids = torch.randint(0, 320, (2, 41), device="cuda")
    step = lambda cache: model(input_ids=ids[:, 40:], past_key_values=cache, use_cache=True).logits
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.no_grad():
        cache = model(input_ids=ids[:, :40], use_cache=True).past_key_values
        caches = [copy.deepcopy(cache) for _ in range(3)]
        for name, p in model.named_parameters():
            if "norm" in name or "conv_weight" in name:
                p.add_(0.25 * torch.randn_like(p))
        torch.cuda.synchronize()
        with torch.cuda.stream(one):
            torch.cuda._sleep(200_000_000)
            first = step(caches[0])
        with torch.cuda.stream(two):
            second = step(caches[1])
        torch.cuda.synchronize()
        want = step(caches[2])
    assert torch.equal(first, want) and torch.equal(second, want)


def test_copies_missing_during_a_capture_belong_to_the_graph():
    """A step captured with its parameter copies out of date converts them inside the graph, and leaves nothing behind that
    only a replay would fill."""
    torch.manual_seed(8)
    model = SolveDeltaForCausalLM(SolveDeltaConfig(hidden_size=256, num_heads=4, head_k_dim=64, head_v_dim=64,
                                                   num_hidden_layers=2, vocab_size=320)).prepare("cuda").eval()
    ids = torch.randint(0, 320, (2, 41), device="cuda")
    token = ids[:, 40:].contiguous()
    step = lambda cache: model(input_ids=token, past_key_values=cache, use_cache=True).logits
    with torch.no_grad():
        cache = model(input_ids=ids[:, :40], use_cache=True).past_key_values
        caches = [copy.deepcopy(cache) for _ in range(3)]
        step(copy.deepcopy(cache))   # lazy initialisation
        for name, p in model.named_parameters():
            if "norm" in name or "conv_weight" in name:
                p.add_(0.25 * torch.randn_like(p))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured = step(caches[0])
        want = step(caches[1])
        graph.replay()
        assert torch.equal(captured, want)
        del graph
        assert torch.equal(step(caches[2]), want)
