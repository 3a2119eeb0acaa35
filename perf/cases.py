"""Timed cases of this package: what its users run, over the range of sizes they run it at.

Kinds of case (``kind``):

* ``op_train``    the operator, forward + full VJP: what a mixer of one's own calls in training
* ``op_forward``  the operator without gradients: prefill of a serving loop, evaluation
* ``op_decode``   one recurrent token of the operator from its states
* ``mixer_train`` the ``SolveDelta`` layer, forward + backward with every gradient
* ``lm_prefill``  ``SolveDeltaForCausalLM`` on a prompt: last-token logits and the decode cache
* ``lm_decode``   one cached token of that model, called directly or replayed by ``GraphedDecoder``

Geometries are those of the package's benchmark (8 heads of 128/128, hidden 1024, vocabulary 32000,
T = 4096 / 2048 / 32768; three of its 24 equal layers, so that roundings do not add up beyond
comparison) and of its tests (4 heads of 64/64, hidden 256, T = 128; ragged lengths; unequal
widths; token masks with resets), with the sizes in between drawn by ``draw``.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from solvedelta_b200 import (GraphedDecoder, SolveDelta, SolveDeltaConfig, SolveDeltaForCausalLM,
                             SolveDeltaState, solvedelta_masked_native, solvedelta_native)

VOCAB = 32000
OPERANDS = ("u", "h", "q", "keys", "values", "log_decay", "erase_raw", "write_raw", "geometry_write")


def _op(kind, batch, tokens, heads=8, rank=128, value=128, masked=False):
    return {"kind": kind, "batch": batch, "tokens": tokens, "heads": heads, "rank": rank, "value": value,
            "masked": masked}


def _model(kind, batch, tokens, hidden=1024, heads=8, width=128, layers=1, graphed=False):
    return {"kind": kind, "batch": batch, "tokens": tokens, "hidden": hidden, "heads": heads, "width": width,
            "layers": layers, "graphed": graphed}


def listed():
    return [
        # one token of one sequence through the bare operator: launches and host time
        dict(_op("op_decode", 1, 1), name="op_decode_b1"),
        # the same step for a full serving batch: both FP32 states of every stream move once
        dict(_op("op_decode", 96, 1), name="op_decode_b96"),
        # the small configuration of the tests (4 heads of 64): a short training call, bound by launches
        dict(_op("op_train", 2, 128, heads=4, rank=64, value=64), name="op_train_b2_t128_r64"),
        # one sequence of 1024 tokens: too few chunks to fill the device
        dict(_op("op_train", 1, 1024), name="op_train_b1_t1024"),
        # a padded batch of packed sequences of odd length with unequal widths: masks and resets in the kernels
        dict(_op("op_train", 5, 1531, rank=96, value=128, masked=True), name="op_train_b5_t1531_masked"),
        # the benchmark's training step of the operator
        dict(_op("op_train", 8, 4096), name="op_train_b8_t4096"),
        # the same batch without gradients, final states returned
        dict(_op("op_forward", 8, 4096), name="op_forward_b8_t4096"),
        # long-context prefill of one sequence: 512 chunks in a row, eight streams
        dict(_op("op_forward", 1, 32768), name="op_forward_b1_t32768"),
        # one layer in a training step of the benchmark's model
        dict(_model("mixer_train", 8, 2048), name="mixer_train_b8_t2048"),
        # prompts through three of the benchmark model's layers and its head
        dict(_model("lm_prefill", 4, 4096, layers=3), name="lm_prefill_b4_t4096"),
        # one cached token as a generation loop without graphs calls it
        dict(_model("lm_decode", 1, 1, layers=3), name="lm_decode_b1"),
        # one cached token of a small serving batch, replayed from the decoder's graph
        dict(_model("lm_decode", 4, 1, layers=3, graphed=True), name="lm_decode_b4_graphed"),
    ]


def _between(rng, low, high):
    """A whole number, spread evenly over the logarithm of the range."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(("op_train", "op_train", "op_train", "op_forward", "op_forward", "op_decode", "mixer_train",
                       "lm_prefill", "lm_decode", "lm_decode"))
    if kind == "op_decode":
        heads, width = rng.choice(((8, 128), (8, 128), (4, 64), (16, 128)))
        return _op(kind, _between(rng, 1, 96 if heads <= 8 else 48), 1, heads, width, width)
    if kind in ("op_train", "op_forward"):
        heads = rng.choice((4, 8, 8, 16))
        rank, value = rng.choice(((128, 128), (128, 128), (64, 64), (96, 128), (128, 64), (80, 112)))
        # token-heads up to those of the benchmark batch, split between batch and length
        total = _between(rng, 64, 32768 * 8 // heads)
        batch = _between(rng, 1, max(1, min(16, total // 64)))
        return _op(kind, batch, max(2, total // batch), heads, rank, value, masked=rng.random() < 0.25)
    hidden, heads, width = rng.choice(((1024, 8, 128), (1024, 8, 128), (256, 4, 64), (2048, 16, 128)))
    if kind == "lm_decode":
        return _model(kind, _between(rng, 1, 32), 1, hidden, heads, width, rng.randint(1, 3), rng.random() < 0.5)
    if kind == "mixer_train":
        # a training batch: gradients of the scalar gate parameters are sums over many tokens
        hidden, heads, width = rng.choice(((1024, 8, 128), (2048, 16, 128)))
    total = _between(rng, 1024 if kind == "mixer_train" else 128, 16384 if hidden <= 1024 else 8192)
    batch = _between(rng, 1, min(16, total // 64))
    if kind == "mixer_train":
        return _model(kind, batch, total // batch, hidden, heads, width)
    return _model(kind, batch, max(2, total // batch), hidden, heads, width, rng.randint(1, 3))


def _config(case):
    return SolveDeltaConfig(hidden_size=case["hidden"], num_heads=case["heads"], head_k_dim=case["width"],
                            head_v_dim=case["width"], num_hidden_layers=case["layers"], vocab_size=VOCAB)


def _op_inputs(case, gen):
    """The benchmark's distributions: unit q / k, decay of about 2 % per token and channel, carried states."""
    B, T, H, r, V = (case[n] for n in ("batch", "tokens", "heads", "rank", "value"))
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    bf = lambda x: x.to(torch.bfloat16)
    return dict(
        u=bf(rn(B, T, H, r)), h=bf(rn(B, T, H, r)), q=bf(F.normalize(rn(B, T, H, r), dim=-1)),
        keys=bf(F.normalize(rn(B, T, H, 1, r), dim=-1)), values=bf(rn(B, T, H, 1, V)),
        log_decay=F.logsigmoid(rn(B, T, H, r) + 4.0), erase_raw=bf(0.5 * rn(B, T, H, 1, r)),
        write_raw=bf(0.5 * rn(B, T, H, 1, V)),
        geometry_write=0.1 * torch.rand(B, T, H, generator=gen, device="cuda"),
        C0=0.02 * rn(B, H, r, r), S0=0.02 * rn(B, H, r, V))


def _masks(case, gen):
    """Left padding of up to a quarter of each row, and a new sequence every few hundred tokens."""
    B, T = case["batch"], case["tokens"]
    pad = torch.randint(0, T // 4 + 1, (B, 1), generator=gen, device="cuda")
    valid = torch.arange(T, device="cuda") >= pad
    reset = torch.rand(B, T, generator=gen, device="cuda") < 1.0 / 300.0
    return {"valid_mask": valid, "reset_mask": reset & valid}


def _bench_gates(module):
    """Geometry rates around 0.05 and decays of about 2 % per token, as in the operator's benchmark.  The initial
    rate of 0.9 belongs to projections that are trained with it: on random ones it amplifies a rounding of the first
    layer until nothing is comparable."""
    constants = {"geometry_write_bias": math.log(0.05 / 0.95), "associative_log_rate": 0.0,
                 "associative_decay_bias": math.log(math.expm1(0.018))}
    for name, p in module.named_parameters():
        if (value := constants.get(name.rsplit(".", 1)[-1])) is not None:
            p.data.fill_(value)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    kind, B, T = case["kind"], case["batch"], case["tokens"]
    state = {"kind": kind}
    if kind.startswith("op_"):
        H, r, V = case["heads"], case["rank"], case["value"]
        x = _op_inputs(case, gen)
        train = kind == "op_train"
        leaves = [x[n].requires_grad_(train) for n in OPERANDS + ("C0", "S0")]
        state.update(leaves=leaves, carried=SolveDeltaState(leaves[-2], leaves[-1]),
                     masks=_masks(case, gen) if case["masked"] else None)
        if train:
            state["cotangents"] = [rn(B, T, H, V).to(torch.bfloat16), rn(B, H, r, r), rn(B, H, r, V)]
        return state
    torch.manual_seed(seed)
    with torch.device("cuda"):
        module = SolveDelta(_config(case)) if kind == "mixer_train" else SolveDeltaForCausalLM(_config(case))
    _bench_gates(module)
    if kind == "mixer_train":
        for name, p in module.named_parameters():   # BF16 weights, the scalar gate families in FP32
            if name not in ("geometry_write_bias", "associative_log_rate", "associative_decay_bias"):
                p.data = p.data.to(torch.bfloat16)
        state.update(module=module, x=rn(B, T, case["hidden"]).to(torch.bfloat16).requires_grad_(),
                     target=(0.3 * rn(B, T, case["hidden"])).to(torch.bfloat16), params=list(module.parameters()))
        return state
    model = module.prepare("cuda").eval()
    state["model"] = model
    if kind == "lm_prefill":
        state["ids"] = torch.randint(0, VOCAB, (B, T), generator=gen, device="cuda")
        return state
    # decoding goes on from the cache of a short prompt
    ids = torch.randint(0, VOCAB, (B, 64), generator=gen, device="cuda")
    with torch.no_grad():
        cache = model(input_ids=ids, use_cache=True, logits_to_keep=1).past_key_values
    state.update(token=torch.randint(0, VOCAB, (B, 1), generator=gen, device="cuda"), cache=cache,
                 decoder=GraphedDecoder(model, cache, B) if case["graphed"] else None)
    return state


def _cache_tensors(cache):
    return [t for layer in cache for t in (*layer["recurrent_state"], layer["conv_state"])]


def run(state):
    kind = state["kind"]
    if kind.startswith("op_"):
        operands, masks = state["leaves"][:-2], state["masks"]
        with torch.set_grad_enabled(kind == "op_train"):
            if masks is None:
                y, after = solvedelta_native(*operands, initial_state=state["carried"], return_final_state=True)
            else:
                y, after = solvedelta_masked_native(*operands, **masks, initial_state=state["carried"],
                                                    return_final_state=True)
        if kind != "op_train":
            return [y, after.predictor, after.S]
        outputs = [y, after.predictor, after.S]
        return [t.detach() for t in outputs] + list(torch.autograd.grad(outputs, state["leaves"], state["cotangents"]))
    if kind == "mixer_train":
        out = state["module"](state["x"])
        loss = F.mse_loss(out, state["target"], reduction="sum")
        return [out.detach()] + list(torch.autograd.grad(loss, [state["x"]] + state["params"]))
    if kind == "lm_prefill":
        with torch.no_grad():
            out = state["model"](input_ids=state["ids"], use_cache=True, logits_to_keep=1)
        return [out.logits] + _cache_tensors(out.past_key_values)
    if state["decoder"] is not None:
        return [state["decoder"].step(state["token"])] + _cache_tensors(state["cache"])
    with torch.no_grad():
        logits = state["model"](input_ids=state["token"], past_key_values=state["cache"], use_cache=True,
                                logits_to_keep=1).logits
    return [logits] + _cache_tensors(state["cache"])


def _op_work(batch, tokens, heads, rank, value, train):
    """Operands and results once; the operations of the token recurrence (its VJP does twice those)."""
    tok, streams = batch * tokens * heads, batch * heads
    operands = 2 * (5 * rank + 2 * value) + 4 * rank + 4
    states = 4 * streams * (rank * rank + rank * value)
    if train:
        return tok * (2 * operands + 4 * value) + 4 * states, 3 * tok * (6 * rank * rank + 8 * rank * value)
    return tok * (operands + 2 * value) + 2 * states, tok * (6 * rank * rank + 8 * rank * value)


def work(case):
    kind, B, T, H = case["kind"], case["batch"], case["tokens"], case["heads"]
    if kind.startswith("op_"):
        nbytes, flops = _op_work(B, T, H, case["rank"], case["value"], kind == "op_train")
        return {"bytes": nbytes + (2 * B * T if case["masked"] else 0), "flops": flops}
    D, w, L = case["hidden"], case["width"], case["layers"]
    mixer = D * (7 * H * w + H + 2 * w) + H * w * D + 2 * w * H * w
    op_flops = _op_work(B, T, H, w, w, kind == "mixer_train")[1]
    if kind == "mixer_train":   # activations, their gradients, weights and their gradients
        return {"bytes": 2 * (4 * B * T * D + 2 * mixer), "flops": 6 * B * T * mixer + op_flops}
    inner = 256 * ((int(D * 4 * 2 / 3) + 255) // 256)
    layer = mixer + 3 * D * inner
    cache = B * H * (8 * w * w + 2 * 3 * 3 * w)
    nbytes = L * (2 * layer + cache * (2 if kind == "lm_decode" else 1)) + 2 * VOCAB * (D + B)
    return {"bytes": nbytes, "flops": L * (2 * B * T * layer + op_flops) + 2 * B * VOCAB * D}


def tolerance(case):
    # BF16 rows in and out, TF32 / BF16 contractions with FP32 sums: the operator's own parity bound is 3e-2 in the
    # 2-norm on gradients; the decode step is FP32 arithmetic on BF16 rows; stacked layers add up BF16 roundings
    if case["kind"] == "op_decode":
        return {"rel": 5e-3}
    if case["kind"] == "op_forward":
        return {"rel": 1e-2}
    return {"rel": 3e-2}
