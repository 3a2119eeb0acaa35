"""The two kinds of chunk kernels against the checker where a call changes from one to the other: a chunk is fast while
every channel's prefix stays within 60 nats.  Decays just inside, just outside and mixed over heads and chunks; chunks of
one token, full ones and ragged ends; widths that need the padded and the unaligned accesses; masked tokens."""
import numpy as np
import pytest
import torch

from oracle import solvedelta_oracle as orc
from solvedelta_b200 import SolveDeltaState, solvedelta_masked_native, solvedelta_native
from tests.gpu_harness import RawRun, make_inputs, oracle_args, oracle_state, raw_gate_grads
from tests.test_gpu_parity import _check_forward, _check_vjp, _masked_case, _native

pytestmark = pytest.mark.gpu

NATS = 60.0
NAMES = ("u", "h", "q", "keys", "values", "log_decay", "erase_raw", "write_raw", "geometry_write")


def _with_decay(cpu, dev, per_token):
    """Channel 1 of head h and chunk c forgets per_token[h][c] nats a token, which alone decides the chunk's kind; the
    others keep about 0.02.  (Strong decays of all channels: test_strong_decay_in_all_channels.)"""
    for t in range(cpu["log_decay"].shape[1]):
        for h in range(cpu["log_decay"].shape[2]):
            cpu["log_decay"][:, t, h, 1] = -per_token[h][t // 64]
    dev["log_decay"] = cpu["log_decay"].cuda()


# the oracle's tolerances of tests/test_gpu_parity.py: 2e-2 on BF16 results, 1e-3 on the FP32 states
@pytest.mark.parametrize("T,r,V", [(64, 128, 128), (65, 64, 96), (130, 20, 12), (191, 128, 64)])
@pytest.mark.parametrize("kind", ["inside", "outside", "mixed"])
def test_chunks_at_the_limit_match_checker(T, r, V, kind):
    cpu, dev = make_inputs(1, T, 2, r, V, seed=41)
    low, high = 0.995 * NATS / 64, 1.005 * NATS / 64
    rows = {"inside": [[low] * 3, [0.02] * 3], "outside": [[high] * 3, [2.5] * 3],
            "mixed": [[0.02, high, 0.02], [high, 0.3, 4.0]]}[kind]
    _with_decay(cpu, dev, rows)
    full = [(h, c) for h in range(2) for c in range((T + 63) // 64) if rows[h][c] * min(64, T - 64 * c) > NATS]
    flags, _ = RawRun(dev).panel(0, "Flags")
    flags = flags.contiguous().flatten().numpy().view(np.uint8)[:2 * ((T + 63) // 64)].reshape(2, -1)
    assert sorted(map(tuple, np.argwhere(flags & 1))) == full
    leaves, state, y, fin = _native(dev, grad=True)
    _check_forward(cpu, y, fin)
    _check_vjp(cpu, leaves, state, y, fin)


def test_more_chunks_than_resident_ctas_with_slow_ones_between():
    """More CTAs than fit the device at once, slow chunks shared out over one CTA per SM: the bits of each stream on its own."""
    B, T, H, r, V = 5, 64 * 24 + 7, 4, 32, 32   # 500 chunks, more than two CTAs on each of 148 SMs
    cpu, dev = make_inputs(B, T, H, r, V, seed=43)
    for b in range(B):
        cpu["log_decay"][b, 64 * (3 + b):64 * (3 + b) + 90, b % H] -= 1.5
    dev["log_decay"] = cpu["log_decay"].cuda()
    dy = torch.randn(B, T, H, V, generator=torch.Generator().manual_seed(44)).to(torch.bfloat16).cuda()

    def run(cut):
        leaves = [cut(dev[n]).contiguous().requires_grad_() for n in NAMES]
        y, fin = solvedelta_native(*leaves, initial_state=SolveDeltaState(cut(dev["C0"]), cut(dev["S0"])),
                                   return_final_state=True)
        return [y, *fin, *torch.autograd.grad(y, leaves, cut(dy))]

    whole = run(lambda t: t)
    for b in (0, 4):
        for one, all_ in zip(run(lambda t: t[b:b + 1]), whole):
            assert torch.equal(one[0], all_[b])


@pytest.mark.parametrize("per_token", [0.1, 0.4, 0.88])
def test_strong_decay_in_all_channels(per_token):
    """The kinds against each other where a fast chunk uses its whole range: the same call with one channel past the limit
    takes the block-centred kernels.  Both round the same quantities to BF16, so neither may be further from the oracle: the
    norm of the roundings of n >= 1024 results scatters by 1 / sqrt(2 n) = 2.2 %, and four times that is allowed.  (The
    log-decay gradient has no fixed bound here: near a nat a token it is the difference of BF16 terms ten times its size.)"""
    T, r, V = 512, 128, 128
    errors = []
    for first in (per_token, 1.1):
        cpu, dev = make_inputs(1, T, 2, r, V, seed=67)
        gen = torch.Generator().manual_seed(68)
        cpu["log_decay"] = -per_token * (0.95 + 0.1 * torch.rand(1, T, 2, r, generator=gen))
        cpu["log_decay"][..., 0] = -first
        dev["log_decay"] = cpu["log_decay"].cuda()
        flags, _ = RawRun(dev).panel(0, "Flags")
        flags = flags.contiguous().flatten().numpy().view(np.uint8)[:2 * (T // 64)]
        assert (flags == (0 if first == per_token else 1)).all()
        leaves, state, y, fin = _native(dev, grad=True)
        dy = torch.randn(y.shape, generator=gen).to(torch.bfloat16)
        got = [y, *fin, *torch.autograd.grad(y, list(leaves) + list(state), dy.cuda())]
        yo, so = orc.forward(*oracle_args(cpu), initial_state=oracle_state(cpu))
        ref = orc.backward(*oracle_args(cpu), dy.double().numpy(), initial_state=oracle_state(cpu))
        der, dwr = raw_gate_grads(cpu, ref)
        want = [yo, so.predictor, so.S, ref["u"], ref["h"], ref["q"], ref["keys"], ref["values"], ref["log_decay"], der, dwr,
                ref["geometry_write"], ref["C0"], ref["S0"]]
        pairs = [(g.detach().double().cpu().numpy().reshape(w.shape), w) for g, w in zip(got, want)]
        pairs[8] = tuple(a[..., 1:] for a in pairs[8])   # the channel that decides the kind differs
        errors.append([np.linalg.norm(g - w) / np.linalg.norm(w) for g, w in pairs])
    for i, (fast, slow) in enumerate(zip(*errors)):
        assert fast <= 1.09 * slow, (i, fast, slow)
        assert slow <= (1e-3 if i in (1, 2) else 2e-2) or i == 8, (i, slow)


def _device_case(B, T, H, r, V, seed):
    """Operands like those of make_inputs, drawn on the device, and the forward and reverse pass over some of the rows."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    bf = lambda t: t.to(torch.bfloat16)
    unit = torch.nn.functional.normalize
    x = dict(u=bf(rn(B, T, H, r)), h=bf(rn(B, T, H, r)), q=bf(unit(rn(B, T, H, r), dim=-1)),
             keys=bf(unit(rn(B, T, H, 1, r), dim=-1)), values=bf(rn(B, T, H, 1, V)),
             log_decay=torch.nn.functional.logsigmoid(rn(B, T, H, r) + 4.0), erase_raw=bf(0.5 * rn(B, T, H, 1, r)),
             write_raw=bf(0.5 * rn(B, T, H, 1, V)), geometry_write=0.1 * torch.rand(B, T, H, generator=gen, device="cuda"))
    dy = bf(rn(B, T, H, V))

    def run(rows=slice(None)):
        leaves = [x[n][rows].detach().requires_grad_() for n in NAMES]
        y, fin = solvedelta_native(*leaves, return_final_state=True)
        return [y.detach(), *(t.detach() for t in fin), *torch.autograd.grad(y, leaves, dy[rows])]

    return x, run, gen


def test_slow_chunks_beyond_one_pass_over_the_flags():
    """8448 chunks, every third slow: the flags of a launch are ranked 8192 at a time.  The bits of one row on its own."""
    B, T, H = 4, 64 * 66, 32
    x, run, gen = _device_case(B, T, H, 16, 8, 59)
    slow = torch.rand(B, T // 64, 1, H, 1, generator=gen, device="cuda") < 1 / 3
    x["log_decay"].view(B, T // 64, 64, H, 16).sub_(1.5 * slow)
    whole = run()
    for b in (0, B - 1):
        for one, all_ in zip(run(slice(b, b + 1)), whole):
            assert torch.equal(one[0], all_[b])


def test_slow_chunks_cost_their_own_work():
    """4096 chunks, all slow, against the same number of fast ones: 1.4 times the time by the work of the two kinds of kernel.
    With every CTA stepping through all slow chunks of a launch it was 2.2 times."""
    x, run, _ = _device_case(8, 4096, 8, 128, 128, 61)

    def milliseconds():
        run()
        times = []
        for _ in range(5):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            run()
            end.record()
            end.synchronize()
            times.append(start.elapsed_time(end))
        return sorted(times)[2]

    fast = milliseconds()
    x["log_decay"] -= 1.3
    assert milliseconds() < 1.8 * fast


@pytest.mark.parametrize("B,T,H", [(11, 150, 1), (37, 200, 1), (1, 64 * 149, 1)])   # 33, 148 and 149 chunks
@pytest.mark.parametrize("masked", [False, True])
def test_calls_without_gradients_give_the_bits_of_those_with(B, T, H, masked):
    """Both kinds of chunk in one launch up to 148 chunks without gradients, up to 32 with them: the same results."""
    x, _, gen = _device_case(B, T, H, 32, 48, 71)
    x["log_decay"] -= 1.5 * (torch.rand(B, T // 50 + 1, 1, H, 1, generator=gen, device="cuda") < 0.3).expand(
        -1, -1, 50, -1, -1).reshape(B, -1, H, 1)[:, :T]
    masks = dict(valid_mask=torch.rand(B, T, generator=gen, device="cuda") < 0.9,
                 reset_mask=torch.rand(B, T, generator=gen, device="cuda") < 0.01) if masked else {}
    masks = {n: m & masks["valid_mask"] for n, m in masks.items()}
    call = solvedelta_masked_native if masked else solvedelta_native
    leaves = [x[n].detach().requires_grad_() for n in NAMES]
    y, fin = call(*leaves, **masks, return_final_state=True)
    with torch.no_grad():
        bare, end = call(*leaves, **masks, return_final_state=True)
    assert torch.equal(bare, y) and all(torch.equal(a, b) for a, b in zip(end, fin))


@pytest.mark.parametrize("r,V", [(128, 128), (20, 12)])
def test_masked_tokens_without_resets_in_fast_chunks(r, V):
    cpu, dev = make_inputs(2, 150, 2, r, V, seed=47)
    valid = torch.ones(2, 150, dtype=torch.bool)
    valid[0, :70] = False      # a whole chunk and the head of the next
    valid[1, 100:103] = False
    _masked_case(cpu, dev, valid, torch.zeros_like(valid))


@pytest.mark.parametrize("rate", [0.0, 1e-30, -0.01])
def test_vanishing_geometry_rates_between_others(rate):
    """The closure divides by the rate in fast chunks: a chunk with one below 1e-20 evaluates the residual instead."""
    cpu, dev = make_inputs(1, 200, 2, 64, 96, seed=53)
    cpu["geometry_write"][0, 70, 0] = rate    # second chunk of head 0
    cpu["geometry_write"][0, 199, 1] = rate   # the ragged end of head 1
    dev["geometry_write"] = cpu["geometry_write"].cuda()
    leaves, state, y, fin = _native(dev, grad=True)
    _check_forward(cpu, y, fin)
    _check_vjp(cpu, leaves, state, y, fin)
