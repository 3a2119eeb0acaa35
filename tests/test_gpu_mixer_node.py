"""The layer as one autograd node against its separate nodes: ragged lengths, unequal widths, biases, masks."""
import pytest
import torch

from solvedelta_b200 import SolveDelta, SolveDeltaConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,hidden,heads,r,V,bias,masked", [
    (1, 1, 128, 2, 64, 64, False, False), (2, 65, 128, 3, 24, 40, True, False),   # five-column tail behind the row
    (1, 130, 256, 2, 128, 128, False, False), (3, 70, 128, 2, 64, 32, True, True)])
def test_one_node_equals_the_separate_nodes(B, T, hidden, heads, r, V, bias, masked, monkeypatch):
    torch.manual_seed(3)
    layer = SolveDelta(SolveDeltaConfig(hidden_size=hidden, num_heads=heads, head_k_dim=r, head_v_dim=V, bias=bias)).cuda()
    for name, p in layer.named_parameters():
        if name not in ("geometry_write_bias", "associative_log_rate", "associative_decay_bias"):
            p.data = p.data.to(torch.bfloat16)
    x = torch.randn(B, T, hidden, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    dy = torch.randn(B, T, hidden, device="cuda", dtype=torch.bfloat16)
    masks = {}
    if masked:
        masks = dict(valid_mask=torch.rand(B, T, device="cuda") < 0.9, reset_mask=torch.rand(B, T, device="cuda") < 0.05)
    named = dict(layer.named_parameters())
    seen = []
    for one in (True, False):
        if not one:
            monkeypatch.setattr(SolveDelta, "_one_node_applies", lambda *a: False)
        out = layer(x, **masks)
        assert (out.grad_fn.name().find("MixerFunction") >= 0) == one
        seen.append([out.detach(), *torch.autograd.grad(out, [x, *named.values()], dy)])
    for name, got, want in zip(["out", "x", *named], *seen):
        assert got.dtype == want.dtype and got.shape == want.shape, name
        scale = want.float().abs().max().item()
        assert (got.float() - want.float()).abs().max().item() <= 1e-2 * scale, name


@pytest.mark.parametrize("one", [True, False])
def test_first_order_gradients_with_create_graph(one, monkeypatch):
    """``create_graph=True`` records gradients during the reverse pass; the layer's kernels have no second derivative, and
    the first-order gradients are the same."""
    torch.manual_seed(4)
    layer = SolveDelta(SolveDeltaConfig(hidden_size=128, num_heads=2, head_k_dim=32, head_v_dim=32, bias=True)).cuda()
    for name, p in layer.named_parameters():
        if name not in ("geometry_write_bias", "associative_log_rate", "associative_decay_bias"):
            p.data = p.data.to(torch.bfloat16)
    x = torch.randn(2, 70, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    dy = torch.randn(2, 70, 128, device="cuda", dtype=torch.bfloat16)
    if not one:
        monkeypatch.setattr(SolveDelta, "_one_node_applies", lambda *a: False)
    leaves = [x, *layer.parameters()]
    plain = torch.autograd.grad(layer(x), leaves, dy)
    recorded = torch.autograd.grad(layer(x), leaves, dy, create_graph=True)
    for got, want in zip(recorded, plain):
        assert torch.equal(got.detach(), want)
