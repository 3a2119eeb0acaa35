"""A NaN in one operand: every result that the checker finds NaN is NaN here too, whatever contraction it passes through,
and nothing before its chunk or in another stream is touched by it."""
import numpy as np
import pytest
import torch

from oracle import solvedelta_oracle as orc
from solvedelta_b200 import SolveDeltaState, solvedelta_native
from tests.gpu_harness import make_inputs, oracle_args, oracle_state, raw_gate_grads

pytestmark = pytest.mark.gpu
OPERANDS = ("u", "h", "q", "keys", "values", "log_decay", "erase_raw", "write_raw", "geometry_write")
B, T, H, AT, HEAD = 2, 150, 2, 70, 1   # the NaN: row 0, token 70 (second chunk of 64), head 1


def _run(dev, dy):
    leaves = [dev[n].detach().requires_grad_() for n in OPERANDS + ("C0", "S0")]
    y, fin = solvedelta_native(*leaves[:-2], initial_state=SolveDeltaState(*leaves[-2:]), return_final_state=True)
    grads = torch.autograd.grad([y, fin.predictor, fin.S], leaves, [dy, torch.ones_like(fin.predictor), torch.ones_like(fin.S)])
    with torch.no_grad():   # the forward pass that keeps nothing for a reverse pass
        bare, _ = solvedelta_native(*leaves[:-2], initial_state=SolveDeltaState(*leaves[-2:]), return_final_state=True)
    assert torch.equal(bare.isnan(), y.isnan())
    f = lambda t: t.detach().double().cpu().numpy()
    return f(y), f(fin.predictor), f(fin.S), [f(g) for g in grads]


QUIET, ALL_ONES, SIGNALLING = 0x7fc00000, -1, 0x7f800001   # FP32 patterns; only memory can hold the last two


@pytest.mark.parametrize("r,V", [(32, 48), (20, 12)])   # aligned rows, and the general row accesses
@pytest.mark.parametrize("name,bits", [(n, QUIET) for n in OPERANDS + ("C0", "S0")] + [
    (n, b) for n in ("log_decay", "geometry_write", "C0", "S0") for b in (ALL_ONES, SIGNALLING)])
def test_nan_reaches_what_it_reaches_in_the_checker(name, bits, r, V):
    cpu, dev = make_inputs(B, T, H, r, V, seed=11)
    dy = torch.randn(B, T, H, V, generator=torch.Generator().manual_seed(12)).to(torch.bfloat16)
    clean = _run(dev, dy.cuda())
    where = (0, HEAD, 1, 3) if name in ("C0", "S0") else (0, AT, HEAD) + ((0,) if cpu[name].ndim == 5 else ()) + (
        () if cpu[name].ndim == 3 else (3,))
    if bits == QUIET:
        cpu[name][where] = float("nan")
    else:
        cpu[name].view(torch.int32)[where] = bits
    dev[name] = cpu[name].cuda()
    y, C, S, grads = _run(dev, dy.cuda())
    with np.errstate(invalid="ignore"):
        yo, so = orc.forward(*oracle_args(cpu), initial_state=oracle_state(cpu))
        ref = orc.backward(*oracle_args(cpu), dy.double().numpy(), dC_T=np.ones((B, H, r, r)), dS_T=np.ones((B, H, r, V)),
                           initial_state=oracle_state(cpu))
        der, dwr = raw_gate_grads(cpu, ref)
    assert np.isnan(yo).any()
    for got, want in ((y, yo), (C, so.predictor), (S, so.S)):
        assert np.isnan(got[np.isnan(want)]).all()
    want = [ref["u"], ref["h"], ref["q"], ref["keys"], ref["values"], ref["log_decay"], der, dwr, ref["geometry_write"],
            ref["C0"], ref["S0"]]
    for leaf, got, expect in zip(OPERANDS + ("C0", "S0"), grads, want):
        expect = expect.reshape(got.shape)
        assert np.isnan(got[np.isnan(expect)]).all(), leaf
    # other streams, and the chunk before: the bits of the run without the NaN
    assert np.array_equal(y[1], clean[0][1]) and np.array_equal(y[0, :, 1 - HEAD], clean[0][0, :, 1 - HEAD])
    if name not in ("C0", "S0"):
        assert np.array_equal(y[0, :64, HEAD], clean[0][0, :64, HEAD])


@pytest.mark.parametrize("name", ["u", "h", "keys", "values", "log_decay", "erase_raw", "geometry_write"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_last_token_of_a_chunk_touches_nothing_before_the_chunk(name, bad):
    """Sums over a chunk may carry a NaN to the chunk's earlier tokens (token 127 to 64 and on), but not further back."""
    cpu, dev = make_inputs(B, T, H, 32, 48, seed=13)
    args = lambda: [dev[n] for n in OPERANDS]
    with torch.no_grad():
        clean, _ = solvedelta_native(*args(), initial_state=SolveDeltaState(dev["C0"], dev["S0"]), return_final_state=True)
        dev[name] = dev[name].clone()
        dev[name][(0, 127, HEAD) + (0,) * (dev[name].ndim - 3)] = bad if name != "log_decay" else -abs(bad)
        y, _ = solvedelta_native(*args(), initial_state=SolveDeltaState(dev["C0"], dev["S0"]), return_final_state=True)
    assert torch.equal(y[0, :64, HEAD], clean[0, :64, HEAD])
    assert torch.equal(y[1], clean[1]) and torch.equal(y[0, :, 1 - HEAD], clean[0, :, 1 - HEAD])
