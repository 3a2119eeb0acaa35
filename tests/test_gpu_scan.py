"""The state scans cut into segments (few streams, many chunks) against the checker, and against the uncut scans."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import solvedelta_oracle as orc
from solvedelta_b200 import SolveDeltaState, _lib, solvedelta_native
from tests.gpu_harness import make_inputs, oracle_args, oracle_state, raw_gate_grads
from tests.helpers import max_rel, rel_l2

pytestmark = pytest.mark.gpu
OPERANDS = ("u", "h", "q", "keys", "values", "log_decay", "erase_raw", "write_raw", "geometry_write")


@pytest.mark.parametrize("B,T,H,r,V", [(1, 4097, 1, 128, 128), (1, 4800, 2, 32, 48), (2, 4500, 4, 16, 16), (3, 4200, 6, 24, 8)])
def test_segmented_scans_match_checker(B, T, H, r, V):
    assert _lib.load().sd_forward_launches(ctypes.byref(_lib.Shape(B, T, H, r, V))) > 5
    cpu, dev = make_inputs(B, T, H, r, V, seed=T, gamma_max=0.3)
    leaves = [dev[n].requires_grad_() for n in OPERANDS]
    state = SolveDeltaState(dev["C0"].requires_grad_(), dev["S0"].requires_grad_())
    y, fin = solvedelta_native(*leaves, initial_state=state, return_final_state=True)
    gen = torch.Generator().manual_seed(7)
    dy, dC, dS = (torch.randn(t.shape, generator=gen) for t in (y, fin.predictor, fin.S))
    dy = dy.to(torch.bfloat16)
    grads = torch.autograd.grad([y, fin.predictor, fin.S], leaves + [state.predictor, state.S],
                                [dy.cuda(), dC.cuda(), dS.cuda()])
    yo, so = orc.forward(*oracle_args(cpu), initial_state=oracle_state(cpu))
    assert max_rel(y.detach().float().cpu().numpy(), yo) <= 2e-2
    assert max_rel(fin.predictor.detach().cpu().numpy(), so.predictor) <= 1e-3
    assert max_rel(fin.S.detach().cpu().numpy(), so.S) <= 1e-3
    ref = orc.backward(*oracle_args(cpu), dy.double().numpy(), dC_T=dC.double().numpy(), dS_T=dS.double().numpy(),
                       initial_state=oracle_state(cpu))
    der, dwr = raw_gate_grads(cpu, ref)
    want = [ref["u"], ref["h"], ref["q"], ref["keys"], ref["values"], ref["log_decay"], der, dwr, ref["geometry_write"],
            ref["C0"], ref["S0"]]
    for name, got, expect in zip(OPERANDS + ("C0", "S0"), grads, want):
        got = got.float().cpu().numpy().reshape(np.shape(expect))
        assert rel_l2(got, expect) <= 3e-2, name
