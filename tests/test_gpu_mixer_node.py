"""The layer as one autograd node against its separate nodes and the checker: ragged lengths, unequal widths, biases, masks."""
import numpy as np
import pytest
import torch

from oracle import mixer_oracle as mo
from solvedelta_b200 import SolveDelta, SolveDeltaConfig
from tests.helpers import max_rel, rel_l2

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


@pytest.mark.parametrize("B,T,hidden,heads,r,V,bias,masked", [
    (2, 128, 256, 4, 64, 64, False, False), (2, 150, 128, 3, 24, 40, True, True)])
def test_one_node_matches_checker(B, T, hidden, heads, r, V, bias, masked):
    """What a training step runs (BF16 weights, one autograd node) against the FP64 checker, output and every gradient
    end to end."""
    torch.manual_seed(6)
    layer = SolveDelta(SolveDeltaConfig(hidden_size=hidden, num_heads=heads, head_k_dim=r, head_v_dim=V, bias=bias)).cuda()
    for name, p in layer.named_parameters():
        if name not in ("geometry_write_bias", "associative_log_rate", "associative_decay_bias"):
            p.data = p.data.to(torch.bfloat16)
    gen = torch.Generator().manual_seed(7)
    x = torch.randn(B, T, hidden, generator=gen).to(torch.bfloat16)
    dy = torch.randn(B, T, hidden, generator=gen).to(torch.bfloat16)
    masks = {}
    if masked:
        valid = torch.rand(B, T, generator=gen) < 0.9
        masks = dict(valid_mask=valid, reset_mask=(torch.rand(B, T, generator=gen) < 0.05) & valid)
    named = dict(layer.named_parameters())
    xg = x.cuda().requires_grad_()
    out = layer(xg, **{k: m.cuda() for k, m in masks.items()})
    assert "MixerFunction" in out.grad_fn.name()
    grads = dict(zip(["x", *named], torch.autograd.grad(out, [xg, *named.values()], dy.cuda())))
    f = lambda t: t.detach().double().cpu().numpy()
    checker = mo.MixerOracle({n: f(p) for n, p in named.items()}, hidden_size=hidden, num_heads=heads, head_k_dim=r,
                             head_v_dim=V, use_short_conv=True, norm_eps=layer.output_norm.eps,
                             activation_rounding=lambda z: torch.as_tensor(z).to(torch.bfloat16).double().numpy())
    want_out, _, _ = checker.forward(f(x), **{k: m.numpy() for k, m in masks.items()})
    assert max_rel(f(out), want_out) <= 2e-2
    dx, want, _, _ = checker.backward(f(dy))
    want["x"] = dx
    # The operator's gradients are good to 2e-2 of their largest value at each token.  The three gate families are sums
    # of them over the tokens, times a factor each, that may cancel: 2e-2 of the largest times the factors' sum.
    c, og = checker.cache, checker.operator_grads
    rate = np.exp(f(named["associative_log_rate"]))[None, None, :, None]
    bound = {"geometry_write_bias": np.abs(og["geometry_write"]).max() * (c["gamma"] * (1 - c["gamma"])).sum((0, 1)),
             "associative_log_rate": np.abs(og["log_decay"]).max() * np.abs(c["log_decay"]).sum((0, 1, 3)),
             "associative_decay_bias": np.abs(og["log_decay"]).max() * (rate * (1 - np.exp(c["log_decay"] / rate))).sum((0, 1))}
    for name, got in grads.items():
        got = f(got).reshape(want[name].shape)
        if name in bound:
            assert (np.abs(got - want[name]) <= 2e-2 * bound[name].reshape(got.shape)).all(), name
        else:
            # the decay projection's gradient cancels over the tokens too
            assert rel_l2(got, want[name]) <= (5e-2 if name == "decay_proj.weight" else 2e-2), name
