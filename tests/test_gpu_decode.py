"""The single-token step at the edges of its dispatch: four CTAs per stream against one, whole and ragged state rows,
zero / given initial states, and states left alone unless the caller hands them over."""
import numpy as np
import pytest
import torch

from oracle import solvedelta_oracle as orc
from solvedelta_b200 import SolveDelta, SolveDeltaConfig, SolveDeltaState, solvedelta_native
from tests.gpu_harness import make_inputs, oracle_args, oracle_state
from tests.helpers import max_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,r,V,with_state,inplace", [
    (32, 2, 128, 128, True, False), (13, 5, 128, 128, True, False),   # 64 and 65 streams: the two launch shapes
    (1, 1, 7, 13, True, True), (76, 1, 7, 13, True, False),           # rows that are no multiple of four
    (1, 2, 128, 36, False, False), (80, 1, 20, 128, False, False)])
def test_decode_step_launch_shapes(B, H, r, V, with_state, inplace):
    cpu, dev = make_inputs(B, 1, H, r, V, seed=29, with_state=with_state, gamma_max=0.9)
    operands = [dev[n] for n in ("u", "h", "q", "keys", "values", "log_decay", "erase_raw", "write_raw",
                                 "geometry_write")]
    state = SolveDeltaState(dev["C0"].clone(), dev["S0"].clone()) if with_state else None
    with torch.no_grad():
        y, fin = solvedelta_native(*operands, initial_state=state, return_final_state=True, _inplace_state=inplace)
    yo, so = orc.forward(*oracle_args(cpu), initial_state=oracle_state(cpu))
    assert max_rel(y.float().cpu().numpy(), yo) <= 8e-3
    assert max_rel(fin.predictor.cpu().numpy(), so.predictor) <= 1e-5
    assert max_rel(fin.S.cpu().numpy(), so.S) <= 1e-5
    if with_state:
        assert (fin.S.data_ptr() == state.S.data_ptr()) == inplace
        if not inplace:
            np.testing.assert_array_equal(state.S.cpu().numpy(), cpu["S0"].numpy())


@pytest.mark.parametrize("width", [64, 128])
def test_mixer_step_does_not_depend_on_the_number_of_streams(width):
    # 76 streams: one CTA each; 38: clusters of four
    torch.manual_seed(11)
    layer = SolveDelta(SolveDeltaConfig(hidden_size=256, num_heads=2, head_k_dim=width, head_v_dim=width))
    layer = layer.cuda().to(torch.bfloat16)
    for name in ("geometry_write_bias", "associative_log_rate", "associative_decay_bias"):
        getattr(layer, name).data = getattr(layer, name).data.float()
    x = torch.randn(38, 71, 256, device="cuda", dtype=torch.bfloat16)

    def steps(rows):
        with torch.no_grad():
            _, state = layer(rows[:, :66], return_final_state=True)
            outs = []
            for t in range(66, 71):
                y, state = layer(rows[:, t:t + 1], initial_state=state, return_final_state=True)
                outs.append(y)
            return torch.cat(outs, 1)

    whole, halves = steps(x), torch.cat([steps(x[:19]), steps(x[19:])])
    assert max_rel(whole.float().cpu().numpy(), halves.float().cpu().numpy()) <= 1.6e-2
