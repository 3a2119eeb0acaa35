"""The gated MLP calls its two projections as modules unless they are bare ``nn.Linear`` layers: hooks run, and adapters
that show the base layer's ``weight`` keep their own part."""
import pytest
import torch
import torch.nn.functional as F
from torch import nn

from solvedelta_b200 import SolveDeltaConfig, SolveDeltaForCausalLM
from solvedelta_b200.modeling import SolveDeltaMLP, _bare_linear


class Adapter(nn.Module):
    """A low-rank update on a frozen layer, with the base layer's weight in sight as adapter libraries show it."""

    def __init__(self, base):
        super().__init__()
        self.base = base
        self.down = nn.Linear(base.in_features, 4, bias=False)
        self.up = nn.Linear(4, base.out_features, bias=False)

    weight = property(lambda self: self.base.weight)
    bias = property(lambda self: self.base.bias)

    def forward(self, x):
        return self.base(x) + self.up(self.down(x))


def _mlp(device, change):
    torch.manual_seed(8)
    mlp = SolveDeltaMLP(64, intermediate_size=128)
    calls = []
    if change == "adapter":
        mlp.gate_up_proj, mlp.down_proj = Adapter(mlp.gate_up_proj), Adapter(mlp.down_proj)
    elif change == "replaced forward":
        real = mlp.down_proj.forward
        mlp.down_proj.forward = lambda x: 2 * real(x)
    elif change == "hooks":
        mlp.gate_up_proj.register_forward_hook(lambda m, a, out: 2 * out)
        mlp.down_proj.register_forward_pre_hook(lambda m, a: calls.append("pre"))
    elif change == "backward hook":
        mlp.gate_up_proj.register_full_backward_hook(lambda m, gi, go: calls.append("backward"))
    return mlp.to(device=device, dtype=torch.bfloat16), calls


def _by_modules(mlp, x):
    gate, value = mlp.gate_up_proj(x).chunk(2, -1)
    return mlp.down_proj(F.silu(gate) * value)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,grad", [(2, False), (40, False), (40, True), (2, True)])
@pytest.mark.parametrize("change", ["none", "adapter", "replaced forward", "hooks", "backward hook"])
def test_projections_are_called_unless_bare(change, rows, grad):
    mlp, calls = _mlp("cuda", change)
    x = torch.randn(1, rows, 64, device="cuda").to(torch.bfloat16).requires_grad_(grad)
    with torch.set_grad_enabled(grad):
        want = _by_modules(mlp, x)
        expected = {"hooks": ["pre"]}.get(change, [])
        assert calls == expected
        calls.clear()
        got = mlp(x)
    # BF16 rounding of the activation's two factors on one side, of their product on the other
    assert (got.float() - want.float()).norm() <= 1e-2 * want.float().norm()
    assert calls == expected
    if grad:
        got.float().sum().backward()
        assert calls == {"backward hook": ["backward"]}.get(change, expected)
        assert all(p.grad is not None for p in mlp.parameters())


@pytest.mark.gpu
def test_hook_on_a_projection_runs_for_cached_tokens():
    torch.manual_seed(9)
    model = SolveDeltaForCausalLM(SolveDeltaConfig(hidden_size=256, num_heads=4, head_k_dim=64, head_v_dim=64,
                                                   num_hidden_layers=2, vocab_size=320)).prepare("cuda").eval()
    ids = torch.randint(0, 320, (2, 41), device="cuda")
    with torch.no_grad():
        cache = model(input_ids=ids[:, :40], use_cache=True).past_key_values
        calls = []
        model.model.layers[1].mlp.down_proj.register_forward_hook(lambda *a: calls.append(1))
        model(input_ids=ids[:, 40:], past_key_values=cache, use_cache=True)
    assert calls == [1]


def test_what_counts_as_bare():
    layer = lambda: nn.Linear(8, 8)
    assert _bare_linear(layer())
    for register in ("register_forward_hook", "register_forward_pre_hook", "register_full_backward_hook",
                     "register_full_backward_pre_hook"):
        hooked = layer()
        handle = getattr(hooked, register)(lambda *a: None)
        assert not _bare_linear(hooked)
        handle.remove()
        assert _bare_linear(hooked)
    replaced = layer()
    replaced.forward = lambda x: x
    parametrised = nn.utils.parametrizations.weight_norm(layer())
    for changed in (replaced, parametrised, Adapter(layer()), type("Sub", (nn.Linear,), {})(8, 8)):
        assert not _bare_linear(changed)
    handle = nn.modules.module.register_module_forward_hook(lambda *a: None)
    try:
        assert not _bare_linear(layer())
    finally:
        handle.remove()
