"""Throughput benchmark of the SolveDelta chunked recurrence (forward + full VJP).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference]

One "step" is one forward + backward pass of the operator over one batch of
synthetic input of the benchmark geometry (B=8 per GPU, H=8, T=4096,
r=V=128; BF16 vectors, FP32 decay/geometry rate, non-zero initial states and
state cotangents).  Ranks are independent (batch x heads shard with no
collective inside the op): weak scaling, each rank draws its own batch from
seed+rank.  Rank 0 prints one JSON line.

`value`      tokens/s of the whole job with inputs resident in HBM (C-ABI calls
             on preallocated buffers, CUDA events, max over ranks).
`e2e`        the same metric through the public Python entry point with HOST
             (pinned) buffers: host->device copies of every operand and
             device->host copies of the output and all gradients are inside the
             timed region.
`roofline`   `frac` is the whole path: compulsory HBM bytes of one step / step
             time, against the measured HBM peak.  `kernel_frac` is the same
             ratio for the dominant kernel alone on its own inputs and
             outputs; `traffic_per_step` sums the DRAM bytes of all launches
             (from the ncu table under profiles/), `traffic_ratio` divides
             that by the compulsory bytes.
`cpu_baseline`  the FP64 CPU checker (a port of the upstream token loop) timed
             on the host cores on a bounded sample of the same workload.

`--impl reference` times that CPU port alone, with all host threads, on a
bounded sample per step, and prints the same line shape.
"""
from __future__ import annotations

import argparse
import ctypes
import json
import os
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

WORKLOAD = dict(B=8, H=8, T=4096, r=128, V=128)
REPEATS = 3   # timed repeats of the block of --steps steps
METRIC = "solvedelta_fwd_bwd_tokens_per_s"
# compulsory HBM bytes of one token of one head, forward + backward:
# fwd reads 7 BF16 vectors + FP32 decay + gamma, writes y; bwd reads the same
# plus dy, writes 7 BF16 gradients + FP32 d(decay) + d(gamma)
BYTES_PER_TOKEN_HEAD = 7436
STATE_BYTES_PER_STREAM = 10 * 128 * 128 * 4  # C0,S0,C_T,S_T in fwd; 6 state tensors in bwd


def _peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        with open(path) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


class ClockSampler:
    """Samples nvidia-smi clocks and throttle reasons while the timed region runs."""

    FIELDS = ("clocks.sm,clocks.max.sm,clocks_event_reasons.hw_slowdown,"
              "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
              "clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.lines = []

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index), "--query-gpu=" + self.FIELDS,
                 "--format=csv,noheader,nounits", "-lms", "20"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._pump, daemon=True)
            self.thread.start()
        except OSError:
            self.proc = None

    def _pump(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, mx, reasons = [], [], set()
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        for line in self.lines:
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 6:
                continue
            try:
                sm.append(float(parts[0]))
                mx.append(float(parts[1]))
            except ValueError:
                continue
            for name, val in zip(names, parts[2:6]):
                if val.lower().startswith("active"):
                    reasons.add(name)
        sm.sort()
        return {"sm_mhz": sm[len(sm) // 2] if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "samples": len(sm), "reasons": sorted(reasons)}


def make_cpu_inputs(B, T, H, r, V, seed):
    import torch

    gen = torch.Generator().manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=gen)
    bf = lambda x: x.to(torch.bfloat16)
    norm = torch.nn.functional.normalize
    beta = rn(B, T, H, 1, 1)
    return dict(
        u=bf(rn(B, T, H, r)), h=bf(rn(B, T, H, r)), q=bf(norm(rn(B, T, H, r), dim=-1)),
        keys=bf(norm(rn(B, T, H, 1, r), dim=-1)), values=bf(rn(B, T, H, 1, V)),
        log_decay=torch.nn.functional.logsigmoid(rn(B, T, H, r) + 4.0),
        erase_raw=bf(beta.expand(B, T, H, 1, r).contiguous()),
        write_raw=bf(beta.expand(B, T, H, 1, V).contiguous()),
        geometry_write=0.1 * torch.rand(B, T, H, generator=gen),
        C0=0.02 * rn(B, H, r, r), S0=0.02 * rn(B, H, r, V),
        dy=bf(rn(B, T, H, V)), dC_T=rn(B, H, r, r), dS_T=rn(B, H, r, V))


def cpu_port_throughput(cpu, batch_rows, tokens, threads, repeats=1):
    """tokens/s of the CPU port (forward + full VJP) on the first `batch_rows`
    batch entries and the first `tokens` tokens of the workload."""
    import torch

    from oracle import solvedelta_oracle as orc

    orc.set_threads(threads)
    d = lambda x: x[:batch_rows, :tokens].double().numpy()
    args = [d(cpu["u"]), d(cpu["h"]), d(cpu["q"]), d(cpu["keys"]), d(cpu["values"]), d(cpu["log_decay"]),
            d(torch.sigmoid(cpu["erase_raw"].double())), d(torch.sigmoid(cpu["write_raw"].double())),
            d(cpu["geometry_write"])]
    state = (cpu["C0"][:batch_rows].double().numpy(), cpu["S0"][:batch_rows].double().numpy())
    dy = d(cpu["dy"])
    dC, dS = cpu["dC_T"][:batch_rows].double().numpy(), cpu["dS_T"][:batch_rows].double().numpy()
    best = None
    for _ in range(repeats):
        t0 = time.perf_counter()
        orc.forward(*args, initial_state=state)
        orc.backward(*args, dy, dC_T=dC, dS_T=dS, initial_state=state)
        dt = time.perf_counter() - t0
        best = dt if best is None else min(best, dt)
    return batch_rows * tokens / best, best


def run_reference(opts, rank, world):
    """The upstream algorithm's CPU implementation (the FP64 port) on the host cores."""
    if rank != 0:
        return
    w = WORKLOAD
    threads = os.cpu_count() or 1
    H, r, V = w["H"], w["r"], w["V"]
    # calibrate on a small slice, then size one step to keep the whole run near two minutes
    # one OpenMP thread per (batch, head) stream: take enough batch rows to occupy every core
    rows = min(w["B"], max(1, -(-threads // H)))
    calib = make_cpu_inputs(rows, 64, H, r, V, seed=0)
    rate, _ = cpu_port_throughput(calib, rows, 64, threads)
    budget = 100.0 / max(opts.steps + opts.warmup, 1)
    tokens = int(min(w["T"], max(64, (rate * budget / rows) // 64 * 64)))
    cpu = make_cpu_inputs(rows, tokens, H, r, V, seed=0)
    for _ in range(opts.warmup):
        cpu_port_throughput(cpu, rows, tokens, threads)
    t0 = time.perf_counter()
    for _ in range(opts.steps):
        cpu_port_throughput(cpu, rows, tokens, threads)
    dt = (time.perf_counter() - t0) / max(opts.steps, 1)
    value = rows * tokens / dt
    sample = f"B={rows} of 8, first {tokens} of {w['T']} tokens, H={H}, r=V={r}, fwd+bwd per step"
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": "tokens/s", "n_gpus": opts.gpus,
        "steps": opts.steps, "warmup": opts.warmup, "ms_per_step": dt * 1e3, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": "operator fwd+bwd, B=8,H=8,T=4096,r=V=128 per GPU (CPU arm: bounded sample per step)",
                   "sample": sample},
        "cpu_baseline": {"value": value, "unit": "tokens/s", "cores": threads, "kind": "port", "sample": sample},
        "e2e": {"value": value, "unit": "tokens/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "gpu_launches": 0,
    }
    print(json.dumps(line), flush=True)


class DeviceStep:
    """Preallocated buffers and C-ABI argument blocks for repeated fwd+bwd steps."""

    def __init__(self, cpu, device):
        import torch

        from solvedelta_b200 import _lib
        from solvedelta_b200.ops import _fill_operands, _operand

        self.torch, self.lib_mod = torch, _lib
        self.lib = _lib.load()
        self.dev = {k: v.to(device) for k, v in cpu.items()}
        d = self.dev
        B, T, H, r = d["u"].shape
        V = d["values"].shape[-1]
        self.shape = _lib.Shape(B, T, H, r, V)
        self.tokens = B * T
        self.streams = B * H
        nb = lambda f: max(int(f(ctypes.byref(self.shape))), 16)
        u8 = dict(dtype=torch.uint8, device=device)
        self.saved = torch.empty(nb(self.lib.sd_saved_bytes), **u8)
        self.fscr = torch.empty(nb(self.lib.sd_forward_scratch_bytes), **u8)
        self.bscr = torch.empty(nb(self.lib.sd_backward_scratch_bytes), **u8)
        bf = dict(dtype=torch.bfloat16, device=device)
        f32 = dict(dtype=torch.float32, device=device)
        self.y = torch.empty(B, T, H, V, **bf)
        self.C_T, self.S_T = torch.empty(B, H, r, r, **f32), torch.empty(B, H, r, V, **f32)
        self.grads = dict(
            u=torch.empty(B, T, H, r, **bf), h=torch.empty(B, T, H, r, **bf), q=torch.empty(B, T, H, r, **bf),
            keys=torch.empty(B, T, H, r, **bf), values=torch.empty(B, T, H, V, **bf),
            erase_raw=torch.empty(B, T, H, r, **bf), write_raw=torch.empty(B, T, H, V, **bf),
            log_decay=torch.empty(B, T, H, r, **f32), geometry_write=torch.empty(B, T, H, **f32),
            C0=torch.empty(B, H, r, r, **f32), S0=torch.empty(B, H, r, V, **f32))
        sq = lambda x: x.squeeze(-2)
        tensors = (d["u"], d["h"], d["q"], sq(d["keys"]), sq(d["values"]), d["log_decay"],
                   sq(d["erase_raw"]), sq(d["write_raw"]), d["geometry_write"])
        fa = _lib.ForwardArgs()
        fa.shape = self.shape
        _fill_operands(fa, tensors)
        fa.C0, fa.S0 = d["C0"].data_ptr(), d["S0"].data_ptr()
        fa.y, fa.C_T, fa.S_T = self.y.data_ptr(), self.C_T.data_ptr(), self.S_T.data_ptr()
        fa.saved, fa.saved_bytes = self.saved.data_ptr(), self.saved.numel()
        fa.scratch, fa.scratch_bytes = self.fscr.data_ptr(), self.fscr.numel()
        ba = _lib.BackwardArgs()
        ba.shape = self.shape
        _fill_operands(ba, tensors)
        ba.dy = _operand(d["dy"])
        ba.dC_T, ba.dS_T = d["dC_T"].data_ptr(), d["dS_T"].data_ptr()
        ba.saved, ba.saved_bytes = self.saved.data_ptr(), self.saved.numel()
        ba.scratch, ba.scratch_bytes = self.bscr.data_ptr(), self.bscr.numel()
        g = self.grads
        ba.du, ba.dh, ba.dq = g["u"].data_ptr(), g["h"].data_ptr(), g["q"].data_ptr()
        ba.dkeys, ba.dvalues = g["keys"].data_ptr(), g["values"].data_ptr()
        ba.derase_raw, ba.dwrite_raw = g["erase_raw"].data_ptr(), g["write_raw"].data_ptr()
        ba.dlog_decay, ba.dgamma = g["log_decay"].data_ptr(), g["geometry_write"].data_ptr()
        ba.dC0, ba.dS0 = g["C0"].data_ptr(), g["S0"].data_ptr()
        self.fa, self.ba = fa, ba
        self.launches = (self.lib.sd_forward_launches(ctypes.byref(self.shape))
                         + self.lib.sd_backward_launches(ctypes.byref(self.shape)))

    def stream(self):
        return ctypes.c_void_p(self.torch.cuda.current_stream().cuda_stream)

    def forward_only(self):
        self.lib_mod.check(self.lib.sd_forward(ctypes.byref(self.fa), self.stream()))

    def step(self):
        st = self.stream()
        self.lib_mod.check(self.lib.sd_forward(ctypes.byref(self.fa), st))
        self.lib_mod.check(self.lib.sd_backward(ctypes.byref(self.ba), st))

    def profile(self):
        """Device time of every launch of one step, from the profiling build of the library (an event
        between launches); the timed legs above run the product build."""
        diag = self.lib_mod.load_diagnostics()
        ms = (ctypes.c_float * 40)()
        count = ctypes.c_int(0)
        self.lib_mod.check(diag.sd_profile_step(ctypes.byref(self.fa), ctypes.byref(self.ba), self.stream(),
                                                ms, 40, ctypes.byref(count)))
        return [(diag.sd_launch_name(i).decode(), float(ms[i])) for i in range(count.value)]


# Algorithmic HBM bytes one launch of each kernel must move, per chunk of 64
# token rows of one stream (panel = 64 x 128 FP32 = 32 KiB, BF16 operand chunk
# = 16 KiB, state = 64 KiB, pair matrix = 16 KiB): every input and output of
# the kernel counted once.
KIB = 1024
# f = FP32 panel 32 KiB, b = BF16 panel or BF16 operand chunk 16 KiB, s = FP32 state 64 KiB,
# t = BF16 state 32 KiB, m = BF16 pair matrix 8 KiB, p = FP32 pair matrix 16 KiB
_F, _B, _S, _T, _M, _P = 32 * KIB, 16 * KIB, 64 * KIB, 32 * KIB, 8 * KIB, 16 * KIB
KERNEL_BYTES_PER_CHUNK = {
    "k_prep_fwd": 2 * _B + _F + 4 * _F + _P,                    # u,h,g -> Upd,Qc,Ubar,G,N
    "k_state_scan[C]": 4 * _F + _S + _T,                        # P,Q,R -> X, FP32 + BF16 ckpt
    # u,k,q,er,wr,v,G,Delta,Ubar,Ct -> d, Wd,Ud,Dt, Aqd,Aed, Xg,Ag,Dcol,DtB (fast chunks, like the three below)
    "k_primal_exterior_fwd": 6 * _B + 3 * _F + _S + _F + 3 * _F + _M + _P + 4 * _B,
    "k_state_scan[S]": 3 * _F + _B + _T,                        # P,Q,R -> Z~ (BF16), BF16 ckpt
    "k_output_fwd_tc": _B + _M + _B + _T + _B,                  # Xg,Aqd,Zt,S -> y
    # dy,DtB,Aqd,Aed -> Dyf,Pp,Qp
    "k_exterior_prep_bwd": 2 * _B + _M + _P + 3 * _B,
    "k_state_scan_b[dS]": 6 * _B + _T,
    # Dyf,dR,Zt,Dcol,Xg,Ag,S,dSe + u,k,q,er,wr,v,G,Delta,d -> 5 partial panels, DG,Dd, dq,der,dv,dwr
    "k_exterior_pair_bwd": 6 * _B + 2 * _T + 6 * _B + 3 * _F + 7 * _B + 4 * _B,
    # u,k,G,Delta,DG,Ct(bf16),N,dkPart,dDelta -> Khat,Rneg,Tu,dk,Ppp,Qpp
    "k_primal_bwd": 2 * _B + 2 * _F + _B + _T + _P + 2 * _B + 6 * _B,
    "k_state_scan_b[dC]": 6 * _B + _T,
    # u,G,Delta,dRr,Ct,dCe,Rneg,duPart,Tu,dGPart,Xext -> du,dh,dlog_decay
    "k_predictor_close_bwd": _B + 2 * _F + _B + _T + _T + 5 * _B + 2 * _B + _F,
}


# DRAM bytes per chunk task of every kernel, as ncu measured them (dram__bytes_read.sum +
# dram__bytes_write.sum on the B=8, T=1024 case; traffic is proportional to the number of chunk tasks).
# The table is a text file written by `python bench.py --summarize-ncu <ncu csv>`; without it the
# traffic figures of the line are null.
DRAM_TABLE = os.path.join(ROOT, "profiles", "dram_bytes_per_chunk_task.txt")


def load_dram_table(path=DRAM_TABLE):
    table = {}
    if not os.path.exists(path):
        return table
    with open(path) as f:
        for line in f:
            parts = line.split()
            if len(parts) >= 2 and not line.startswith("#"):
                try:
                    table[parts[0]] = float(parts[1]) * KIB
                except ValueError:
                    continue
    return table


def summarize_ncu(csv_path, tasks):
    """ncu --csv log with dram__bytes_read.sum / dram__bytes_write.sum / gpu__time_duration.sum of the
    launches of ONE fwd+bwd step -> the text table load_dram_table reads (KiB per chunk task)."""
    import csv

    with open(csv_path) as f:
        rows = list(csv.DictReader(l for l in f if l.startswith('"')))
    per_launch, order = {}, []
    for row in rows:
        key = row["ID"]
        if key not in per_launch:
            per_launch[key] = {"name": row["Kernel Name"]}
            order.append(key)
        val = float(row["Metric Value"].replace(",", ""))
        unit = row.get("Metric Unit", "")
        scale = {"Kbyte": 1e3, "Mbyte": 1e6, "Gbyte": 1e9, "byte": 1.0}.get(unit, 1.0)
        per_launch[key][row["Metric Name"]] = val * scale
    def short(full):
        return full.split("(")[0].replace("void ", "").split("<")[0].replace("sd::", "")

    # the last complete step of the capture: k_prep_fwd ... k_predictor_close_bwd.  Of the kernels that come in two kinds
    # the fast chunks' one is the line's (this case has no slow chunks).
    kinds = {"k_primal_exterior_fast": "k_primal_exterior_fwd", "k_exterior_pair_fast": "k_exterior_pair_bwd",
             "k_primal_fast": "k_primal_bwd", "k_predictor_close_fast": "k_predictor_close_bwd"}
    order = [k for k in order if short(per_launch[k]["name"]) not in kinds.values()]
    names = [kinds.get(n, n) for n in (short(per_launch[k]["name"]) for k in order)]
    starts = [i for i, n in enumerate(names) if n == "k_prep_fwd" and i + 11 <= len(names)
              and names[i + 10] == "k_predictor_close_bwd"]
    if not starts:
        raise SystemExit("no complete fwd+bwd step in the capture")
    order = order[starts[-1]:starts[-1] + 11]
    scans = iter(("k_state_scan[C]", "k_state_scan[S]"))
    scans_b = iter(("k_state_scan_b[dS]", "k_state_scan_b[dC]"))
    print("# kernel  KiB-per-chunk-task (DRAM read + write, ncu)  time-us")
    for key in order:
        m = per_launch[key]
        name = kinds.get(short(m["name"]), short(m["name"]))
        if name == "k_state_scan_tc":
            name = next(scans)
        elif name == "k_state_scan_b":
            name = next(scans_b)
        total = m.get("dram__bytes_read.sum", 0.0) + m.get("dram__bytes_write.sum", 0.0)
        print(f"{name} {total / tasks / KIB:.1f} {m.get('gpu__time_duration.sum', 0.0) / 1e3:.1f}")


def time_mixer_glue(B, T, H, r, V, device, reps=20):
    """Device time of the glue kernels around the operator at the workload's shape (conv over the q|k|v slice of
    a projection row, decay gate, gated RMSNorm; residual add + RMSNorm and SwiGLU of the block at hidden 1024 /
    intermediate 2816), forward and reverse, called through the C ABI on preallocated buffers like the main leg,
    with the HBM bandwidth their one-pass algorithmic bytes amount to.  Every operand set is larger than the
    126 MB L2 except the block glue's (B*T rows of 1024), which is stated in `shape`."""
    import torch

    from solvedelta_b200 import _lib

    lib = _lib.load()
    peak, _ = _peaks()
    stream = ctypes.c_void_p(torch.cuda.current_stream(device).cuda_stream)
    gen = torch.Generator(device="cpu").manual_seed(3)

    def bf16(*shape):
        return torch.randn(*shape, generator=gen).to(torch.bfloat16).to(device)

    def scratch(nbytes):
        return torch.empty(max(int(nbytes), 16), dtype=torch.uint8, device=device)

    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)

    def timed(fn, args):
        for _ in range(3):
            _lib.check(fn(ctypes.byref(args), stream))
        torch.cuda.synchronize()
        e0.record()
        for _ in range(reps):
            _lib.check(fn(ctypes.byref(args), stream))
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / reps

    def entry(fwd_ms, bwd_ms, fwd_bytes, bwd_bytes):
        return {"fwd_ms": round(fwd_ms, 4), "bwd_ms": round(bwd_ms, 4),
                "fwd_gbs": round(fwd_bytes / fwd_ms / 1e6, 1), "bwd_gbs": round(bwd_bytes / bwd_ms / 1e6, 1),
                "fwd_frac": round(fwd_bytes / fwd_ms / 1e6 / peak, 3),
                "bwd_frac": round(bwd_bytes / bwd_ms / 1e6 / peak, 3)}

    out = {}
    rows = B * T * H
    # conv4 + SiLU on the first D columns of a wider row (the projection row's layout)
    D = 2 * H * r + H * V
    row = bf16(B, T, D + 64)
    x = row[..., :D]
    w = (0.5 * torch.randn(D, 4, generator=gen)).to(device)
    y, dy, dx = torch.empty(B, T, D, dtype=torch.bfloat16, device=device), bf16(B, T, D), torch.empty(
        B, T, D, dtype=torch.bfloat16, device=device)
    dw = torch.empty(D, 4, device=device)
    sc = scratch(lib.sd_conv4_backward_scratch_bytes(B, T, D))
    f = _lib.Conv4ForwardArgs(B, T, D, x.data_ptr(), x.stride(0), x.stride(1), w.data_ptr(), None, y.data_ptr(), None,
                              None, None)
    g = _lib.Conv4BackwardArgs(B, T, D, x.data_ptr(), x.stride(0), x.stride(1), w.data_ptr(), None, dy.data_ptr(),
                               dx.data_ptr(), dw.data_ptr(), None, sc.data_ptr(), sc.numel(), None, None)
    n = B * T * D
    out["conv4_silu"] = entry(timed(lib.sd_conv4_silu_forward, f), timed(lib.sd_conv4_silu_backward, g), 4 * n, 6 * n)
    del row, x, y, dy, dx
    # decay gate
    raw, A, bias = bf16(rows, r), torch.zeros(H, device=device), torch.zeros(H, r, device=device)
    ld, dld, draw = torch.empty(rows, r, device=device), torch.randn(rows, r, generator=gen).to(device), torch.empty(
        rows, r, dtype=torch.bfloat16, device=device)
    dA, db = torch.empty(H, device=device), torch.empty(H, r, device=device)
    sc = scratch(lib.sd_kda_gate_backward_scratch_bytes(B * T, H, r))
    f = _lib.KdaGateArgs(B * T, H, r, raw.data_ptr(), A.data_ptr(), bias.data_ptr(), ld.data_ptr())
    g = _lib.KdaGateArgs(B * T, H, r, raw.data_ptr(), A.data_ptr(), bias.data_ptr(), None, dld.data_ptr(),
                         draw.data_ptr(), dA.data_ptr(), db.data_ptr(), sc.data_ptr(), sc.numel())
    n = rows * r
    out["kda_decay_gate"] = entry(timed(lib.sd_kda_gate_forward, f), timed(lib.sd_kda_gate_backward, g), 6 * n, 8 * n)
    del raw, ld, dld, draw
    # gated RMSNorm
    o, gate, dyn = bf16(rows, V), bf16(rows, V), bf16(rows, V)
    nw, yn = torch.ones(V, device=device), torch.empty(rows, V, dtype=torch.bfloat16, device=device)
    dxn, dgn, dwn = torch.empty_like(yn), torch.empty_like(yn), torch.empty(V, device=device)
    sc = scratch(lib.sd_norm_gate_backward_scratch_bytes(rows, V))
    f = _lib.NormGateArgs(rows, V, 1e-6, o.data_ptr(), gate.data_ptr(), nw.data_ptr(), yn.data_ptr())
    g = _lib.NormGateArgs(rows, V, 1e-6, o.data_ptr(), gate.data_ptr(), nw.data_ptr(), None, dyn.data_ptr(),
                          dxn.data_ptr(), dgn.data_ptr(), dwn.data_ptr(), sc.data_ptr(), sc.numel())
    n = rows * V
    out["rms_norm_gated"] = entry(timed(lib.sd_norm_gate_forward, f), timed(lib.sd_norm_gate_backward, g), 6 * n, 10 * n)
    del o, gate, dyn, yn, dxn, dgn
    # the block's residual add + RMSNorm and SwiGLU (hidden 1024, intermediate 2816 of the 24-layer model)
    hidden, inter, tokens = 1024, 2816, B * T
    xh, dh, hw = bf16(tokens, hidden), bf16(tokens, hidden), torch.ones(hidden, device=device)
    sh, nh = torch.empty_like(xh), torch.empty_like(xh)
    dsh, dnh, dxh, dwh = bf16(tokens, hidden), bf16(tokens, hidden), torch.empty_like(xh), torch.empty(hidden, device=device)
    sc = scratch(lib.sd_add_rmsnorm_backward_scratch_bytes(tokens, hidden))
    f = _lib.AddRmsnormArgs(tokens, hidden, 1e-6, xh.data_ptr(), dh.data_ptr(), hw.data_ptr(), sh.data_ptr(), nh.data_ptr())
    g = _lib.AddRmsnormBackwardArgs(tokens, hidden, 1e-6, sh.data_ptr(), hw.data_ptr(), dsh.data_ptr(), dnh.data_ptr(),
                                    dxh.data_ptr(), dwh.data_ptr(), sc.data_ptr(), sc.numel())
    n = tokens * hidden
    out["add_rmsnorm"] = entry(timed(lib.sd_add_rmsnorm, f), timed(lib.sd_add_rmsnorm_backward, g), 8 * n, 8 * n)
    del xh, dh, sh, nh, dsh, dnh, dxh
    gv, so, dso = bf16(tokens, 2 * inter), torch.empty(tokens, inter, dtype=torch.bfloat16, device=device), bf16(tokens, inter)
    dgv = torch.empty_like(gv)
    f = _lib.SwigluArgs(tokens, inter, gv.data_ptr(), so.data_ptr(), None, None)
    g = _lib.SwigluArgs(tokens, inter, gv.data_ptr(), None, dso.data_ptr(), dgv.data_ptr())
    n = tokens * inter
    out["swiglu"] = entry(timed(lib.sd_swiglu, f), timed(lib.sd_swiglu_backward, g), 6 * n, 10 * n)
    out["shape"] = (f"B={B}, T={T}: conv channels {D}; gate/norm rows {rows} x {r}; add+norm {tokens} x {hidden} "
                    f"(0.27 GB per pass, above L2); SwiGLU {tokens} x {inter}; through the C ABI on preallocated buffers")
    return out


def time_mixer_module(B, T, H, r, V, device, reps=5):
    """Forward + backward of the SolveDelta mixer (projections through cuBLAS, glue kernels, operator)
    at the layer shape of the reference's 24-layer configuration: hidden 1024, conv on, random init."""
    import torch

    from solvedelta_b200 import SolveDelta, SolveDeltaConfig

    hidden = 1024
    torch.manual_seed(0)
    module = SolveDelta(SolveDeltaConfig(hidden_size=hidden, num_heads=H, head_k_dim=r, head_v_dim=V)).to(device)
    gen = torch.Generator(device="cpu").manual_seed(4)
    x = torch.randn(B, T, hidden, generator=gen).to(torch.bfloat16).to(device).requires_grad_()
    dout = torch.randn(B, T, hidden, generator=gen).to(torch.bfloat16).to(device)
    params = [p for p in module.parameters()]

    def step():
        out = module(x)
        torch.autograd.grad(out, [x] + params, dout)

    for _ in range(2):
        step()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(reps):
        step()
    e1.record()
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / reps
    with torch.no_grad():
        e0.record()
        for _ in range(reps):
            module(x)
        e1.record()
        torch.cuda.synchronize()
    fwd_ms = e0.elapsed_time(e1) / reps
    return {"ms_per_step": round(ms, 3), "value": round(B * T / (ms * 1e-3), 1), "unit": "tokens/s",
            "forward_ms": round(fwd_ms, 3),
            "shape": f"hidden {hidden}, {H} heads, {r}/{V}, B={B}, T={T}, in_proj {hidden}->{module.in_proj.out_features}, "
                     "fwd + bwd (input and all parameter gradients)"}


def time_causal_lm(device, train_steps=3, decode_steps=256):
    """The reference's 24-layer model (hidden 1024, 8 heads of 128/128, conv4, vocabulary 32000, random
    init) through this package's causal LM: one training step (B=8, T=2048: forward, loss, backward,
    fused AdamW on FP32 master weights, BF16 copy back) and long-context serving (prefill of 32768 random
    tokens at B=1, then one-token cached steps).  Uniform random token ids, as the reference's do."""
    import torch

    from solvedelta_b200 import SolveDeltaConfig, SolveDeltaForCausalLM

    torch.manual_seed(0)
    config = SolveDeltaConfig(hidden_size=1024, num_heads=8, head_k_dim=128, head_v_dim=128,
                              num_hidden_layers=24, vocab_size=32000)
    model = SolveDeltaForCausalLM(config).prepare(device).train()
    params = list(model.parameters())
    master = [p.detach().float().clone().requires_grad_() for p in params]
    optimizer = torch.optim.AdamW(master, lr=1e-4, fused=True)
    B, T = 8, 2048
    ids = torch.randint(0, config.vocab_size, (B, T), device=device)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)

    def train_step():
        for p in params:
            p.grad = None
        loss = model(input_ids=ids, labels=ids).loss
        loss.backward()
        for m, p in zip(master, params):
            m.grad = p.grad.float()
        optimizer.step()
        with torch.no_grad():
            for m, p in zip(master, params):
                p.copy_(m)
        return loss

    for _ in range(2):
        train_step()
    torch.cuda.synchronize()
    e0.record()
    for _ in range(train_steps):
        loss = train_step()
    e1.record()
    torch.cuda.synchronize()
    train_ms = e0.elapsed_time(e1) / train_steps
    loss_value = float(loss.detach())
    del loss    # a live autograd graph would keep this stream's gradient accumulators alive into the capture below
    peak_gb = torch.cuda.max_memory_allocated(device) / 2 ** 30
    out = {"parameters": sum(p.numel() for p in params),
           "train": {"ms_per_step": round(train_ms, 1), "value": round(B * T / (train_ms * 1e-3), 1),
                     "unit": "tokens/s", "shape": f"B={B}, T={T}, fwd + loss + bwd + AdamW (FP32 master weights)",
                     "loss": round(loss_value, 4), "peak_memory_gib": round(peak_gb, 1)}}
    del optimizer, master
    for p in params:
        p.grad = None
    torch.cuda.empty_cache()
    # the same step with forward, chunked fixed-denominator loss and backward replayed from one CUDA
    # graph, AdamW on the FP32 masters outside it
    from solvedelta_b200 import BF16ShadowWeights, SolveDeltaGraphedTrainingStep

    torch.cuda.reset_peak_memory_stats(device)
    shadows = BF16ShadowWeights(model, lambda masters: torch.optim.AdamW(masters, lr=1e-4, fused=True))
    graphed = SolveDeltaGraphedTrainingStep(model, ids, ids, num_warmup_iters=2)
    for _ in range(2):
        graphed(ids, ids)
        shadows.optimizer.step()
    torch.cuda.synchronize()
    e0.record()
    for _ in range(train_steps):
        gloss = graphed(ids, ids)
        shadows.optimizer.step()
    e1.record()
    torch.cuda.synchronize()
    graphed_ms = e0.elapsed_time(e1) / train_steps
    out["train_graphed"] = {"ms_per_step": round(graphed_ms, 1), "value": round(B * T / (graphed_ms * 1e-3), 1),
                            "unit": "tokens/s", "loss": round(float(gloss), 4),
                            "shape": "same step: CUDA-graph replay of fwd + chunked loss + bwd, AdamW outside",
                            "peak_memory_gib": round(torch.cuda.max_memory_allocated(device) / 2 ** 30, 1)}
    del graphed, shadows
    for p in params:
        p.grad = None
    model.eval()
    torch.cuda.empty_cache()
    prompt = torch.randint(0, config.vocab_size, (1, 32768), device=device)
    with torch.no_grad():
        model(input_ids=prompt[:, :4096], use_cache=True, logits_to_keep=1)   # warm-up
        torch.cuda.synchronize()
        e0.record()
        step = model(input_ids=prompt, use_cache=True, logits_to_keep=1)
        e1.record()
        torch.cuda.synchronize()
        prefill_ms = e0.elapsed_time(e1)
        cache = step.past_key_values
        token = step.logits[:, -1].argmax(-1, keepdim=True)
        for _ in range(8):
            step = model(input_ids=token, past_key_values=cache, use_cache=True, logits_to_keep=1)
        torch.cuda.synchronize()
        e0.record()
        for _ in range(decode_steps):
            step = model(input_ids=token, past_key_values=cache, use_cache=True, logits_to_keep=1)
            token = step.logits[:, -1].argmax(-1, keepdim=True)
        e1.record()
        torch.cuda.synchronize()
        decode_ms = e0.elapsed_time(e1) / decode_steps
        from solvedelta_b200 import GraphedDecoder

        decoder = GraphedDecoder(model, cache, 1)
        for _ in range(8):
            decoder.step(token)
        torch.cuda.synchronize()
        e0.record()
        for _ in range(decode_steps):
            token = decoder.step(token)[:, -1].argmax(-1, keepdim=True)
        e1.record()
        torch.cuda.synchronize()
        graphed_ms = e0.elapsed_time(e1) / decode_steps
    del cache, decoder, step
    torch.cuda.empty_cache()
    wide = torch.randint(0, config.vocab_size, (16, 32768), device=device)
    with torch.no_grad():
        e0.record()
        model(input_ids=wide, use_cache=True, logits_to_keep=1)
        e1.record()
        torch.cuda.synchronize()
    wide_ms = e0.elapsed_time(e1)
    out["prefill_b16"] = {"ms": round(wide_ms, 1), "value": round(16 * 32768 / (wide_ms * 1e-3), 1), "unit": "tokens/s",
                          "shape": "B=16, T=32768, last-token logits",
                          "peak_memory_gib": round(torch.cuda.max_memory_allocated(device) / 2 ** 30, 1)}
    out["prefill"] = {"ms": round(prefill_ms, 1), "value": round(32768 / (prefill_ms * 1e-3), 1), "unit": "tokens/s",
                      "shape": "B=1, T=32768, last-token logits"}
    out["decode"] = {"ms_per_token": round(decode_ms, 3), "value": round(1.0 / (decode_ms * 1e-3), 1),
                     "unit": "tokens/s", "shape": f"B=1, {decode_steps} cached one-token steps after the prefill",
                     "graphed_ms_per_token": round(graphed_ms, 3), "graphed_value": round(1.0 / (graphed_ms * 1e-3), 1)}
    return out


def _side_leg(fn, *args):
    """Side measurements must not cost the headline line: a failure is reported in their place."""
    try:
        return fn(*args)
    except Exception as error:  # noqa: BLE001 - reported, not swallowed
        import traceback

        traceback.print_exc(file=sys.stderr)
        return {"error": f"{type(error).__name__}: {error}"[:300]}


def run_ours(opts, rank, world, local_rank):
    import torch
    import torch.distributed as dist

    import solvedelta_b200
    from solvedelta_b200 import SolveDeltaState, solvedelta_native
    from solvedelta_b200.sharding import job_throughput, max_over_ranks, rank_seed

    if not torch.cuda.is_available():
        raise RuntimeError("bench.py needs a CUDA device; there is no CPU fallback")
    solvedelta_b200.load()
    torch.cuda.set_device(local_rank)
    device = torch.device("cuda", local_rank)
    if world > 1:
        # keep stdout to the one JSON line: library banners go to stderr
        os.environ.setdefault("NCCL_DEBUG_FILE", "/dev/stderr")
        dist.init_process_group("nccl", device_id=device)
    w = dict(WORKLOAD)
    if opts.case == "small":
        w.update(B=2, T=1024)
    elif opts.case == "medium":
        w.update(B=8, T=1024)
    B, T, H, r, V = w["B"], w["T"], w["H"], w["r"], w["V"]
    if opts.strong:
        # strong scaling: ONE workload of B x H streams dealt out over the ranks (batch rows first, then heads);
        # every rank draws the same inputs and keeps its shard, no data-path collective
        from solvedelta_b200.sharding import stream_shard

        bs, hs = stream_shard(B, H, rank, world)
        full = make_cpu_inputs(B, T, H, r, V, seed=0)
        cpu = {k: (v[bs][:, hs] if k in ("C0", "S0", "dC_T", "dS_T") else v[bs][:, :, hs]).contiguous()
               for k, v in full.items()}
        job_tokens = B * T
        B, H = cpu["u"].shape[0], cpu["u"].shape[2]
    else:
        cpu = make_cpu_inputs(B, T, H, r, V, seed=rank_seed(0, rank))
        job_tokens = world * B * T
    runner = DeviceStep(cpu, device)

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    # ---- device-resident throughput ------------------------------------
    # the clock sampler runs from the warm-up on, so that its samples are taken under load
    sampler = ClockSampler(local_rank)
    if rank == 0:
        sampler.start()
    for _ in range(max(opts.warmup, 3)):
        runner.step()
    barrier()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    # the block of `--steps` steps is timed REPEATS times, each between a barrier + synchronize on both
    # sides and taken as the max over ranks; the line reports the median block and the spread
    block_ms = []
    for _ in range(REPEATS):
        e0.record()
        for _ in range(opts.steps):
            runner.step()
        e1.record()
        barrier()
        block_ms.append(max_over_ranks(e0.elapsed_time(e1), device) / opts.steps)
    clocks = sampler.stop() if rank == 0 else None
    ms_step = sorted(block_ms)[len(block_ms) // 2]
    value = job_tokens / (ms_step * 1e-3)

    # ---- forward only (the kernel-level forward configuration), same inputs ----
    for _ in range(3):
        runner.forward_only()
    barrier()
    e0.record()
    for _ in range(opts.steps):
        runner.forward_only()
    e1.record()
    barrier()
    fwd_ms = max_over_ranks(e0.elapsed_time(e1), device) / opts.steps

    # ---- per-kernel device times (rank 0) --------------------------------
    roofline, kernels = None, None
    if rank == 0:
        acc = {}
        reps = 3
        runner.profile()   # first use of the profiling build: module load and kernel attributes stay out of the average
        for _ in range(reps):
            for name, ms in runner.profile():
                acc[name] = acc.get(name, 0.0) + ms / reps
        total = sum(acc.values())
        kernels = {k: {"ms": round(v, 4), "share": round(v / total, 4)} for k, v in acc.items()}
        top = max(acc, key=acc.get)
        chunks = runner.streams * ((T + 63) // 64)
        alg = KERNEL_BYTES_PER_CHUNK[top] * chunks
        peak, peak_kind = _peaks()
        kernel_achieved = alg / (acc[top] * 1e-3) / 1e9
        path_bytes = runner.tokens * H * BYTES_PER_TOKEN_HEAD + runner.streams * STATE_BYTES_PER_STREAM
        path_achieved = path_bytes / (ms_step * 1e-3) / 1e9
        dram = load_dram_table()
        step_traffic = sum(dram.get(k, 0.0) for k in acc) * chunks if all(k in dram for k in acc) else None
        # `frac` is the whole path (compulsory bytes of a step / step time / peak); the dominant kernel's own
        # figure, on its own inputs and outputs, sits beside it as kernel_frac
        roofline = {"bound": "hbm", "achieved": round(path_achieved, 1), "peak": peak, "unit": "GB/s",
                    "frac": round(path_achieved / peak, 4), "peak_kind": f"of {peak_kind}",
                    "algorithmic_bytes_per_step": path_bytes,
                    "traffic": int(dram[top] * chunks) if top in dram else None,
                    "traffic_per_step": int(step_traffic) if step_traffic else None,
                    "traffic_ratio": round(step_traffic / path_bytes, 2) if step_traffic else None,
                    "kernel": top, "kernel_achieved": round(kernel_achieved, 1),
                    "kernel_frac": round(kernel_achieved / peak, 4),
                    "kernel_algorithmic_bytes_per_launch": alg, "kernel_launch_ms": round(acc[top], 4)}

    # ---- end to end through the public entry point with host buffers -------
    # Every step copies all operands from pinned host memory to the device, runs
    # solvedelta_native + autograd.grad, and copies the output, both final states and all
    # eleven gradients back to pinned host memory.  Steps are pipelined over three streams
    # (upload / compute / download) with two buffer slots, as a caller feeding the operator
    # from the host would do; all of it is inside the timed region.
    names = ("u", "h", "q", "keys", "values", "log_decay", "erase_raw", "write_raw", "geometry_write")
    e2e = None
    if not opts.skip_e2e:
        pinned = {k: v.pin_memory() for k, v in cpu.items()}
        h2d = sum(v.numel() * v.element_size() for v in pinned.values())
        s_comp = torch.cuda.current_stream()
        s_in, s_out = torch.cuda.Stream(), torch.cuda.Stream()
        slots = 2
        dev_in = [{k: torch.empty_like(v, device=device) for k, v in pinned.items()} for _ in range(slots)]
        out_host = [None] * slots
        in_done = [torch.cuda.Event() for _ in range(slots)]
        comp_done = [None] * slots
        out_done = [None] * slots
        d2h_bytes = [0]

        def e2e_step(i):
            slot = i % slots
            if comp_done[slot] is not None:
                s_in.wait_event(comp_done[slot])      # the step that read this slot has finished
            with torch.cuda.stream(s_in):
                for k, v in pinned.items():
                    dev_in[slot][k].copy_(v, non_blocking=True)
                in_done[slot].record(s_in)
            s_comp.wait_event(in_done[slot])
            d = dev_in[slot]
            leaves = [d[n].detach().requires_grad_() for n in names]
            state = SolveDeltaState(d["C0"].detach().requires_grad_(), d["S0"].detach().requires_grad_())
            y, fin = solvedelta_native(*leaves, initial_state=state, return_final_state=True)
            grads = torch.autograd.grad((y, fin.predictor, fin.S), leaves + list(state),
                                        (d["dy"], d["dC_T"], d["dS_T"]))
            results = [y.detach(), fin.predictor.detach(), fin.S.detach(), *grads]
            ev = torch.cuda.Event()
            ev.record(s_comp)
            comp_done[slot] = ev
            if out_host[slot] is None:
                out_host[slot] = [torch.empty(x.shape, dtype=x.dtype).pin_memory() for x in results]
            s_out.wait_event(ev)
            with torch.cuda.stream(s_out):
                for dst, src in zip(out_host[slot], results):
                    dst.copy_(src, non_blocking=True)
                    src.record_stream(s_out)
                done = torch.cuda.Event()
                done.record(s_out)
                out_done[slot] = done
            d2h_bytes[0] = sum(x.numel() * x.element_size() for x in results)

        e2e_steps = max(4, min(opts.steps, 10))
        for i in range(slots):
            e2e_step(i)
        barrier()
        e0.record()
        for i in range(e2e_steps):
            e2e_step(i)
        for ev in out_done:
            s_comp.wait_event(ev)
        e1.record()
        barrier()
        e2e_ms = max_over_ranks(e0.elapsed_time(e1), device) / e2e_steps
        e2e = {"value": job_throughput(runner.tokens, e2e_ms * 1e-3, world), "unit": "tokens/s",
               "ms_per_step": e2e_ms, "steps": e2e_steps, "h2d_bytes_per_step": h2d,
               "d2h_bytes_per_step": d2h_bytes[0], "pipelined": "3 streams, 2 slots"}

    glue = None
    gamma_zero = None
    mixer = None
    if world == 1 and not opts.skip_glue:
        glue = _side_leg(time_mixer_glue, B, T, H, r, V, device)
        mixer = _side_leg(time_mixer_module, B, T, H, r, V, device)
        # geometry write rate 0: the operator reduces to the GDN2 edit (same launches, same traffic)
        cpu0 = dict(cpu)
        cpu0["geometry_write"] = torch.zeros_like(cpu["geometry_write"])
        runner0 = DeviceStep(cpu0, device)
        for _ in range(3):
            runner0.step()
        torch.cuda.synchronize()
        e0.record()
        for _ in range(10):
            runner0.step()
        e1.record()
        torch.cuda.synchronize()
        ms0 = e0.elapsed_time(e1) / 10
        gamma_zero = {"ms_per_step": ms0, "value": runner0.tokens / (ms0 * 1e-3), "unit": "tokens/s"}
        del runner0
    causal_lm = None
    if world == 1 and not opts.skip_glue and not opts.skip_model:
        torch.cuda.empty_cache()
        causal_lm = _side_leg(time_causal_lm, device)

    # every bounded wait inside the kernels completed (this synchronises; the timed regions are over)
    from solvedelta_b200._lib import check_device_fault
    check_device_fault()

    if rank == 0:
        cpu_baseline = None
        if world == 1 and not opts.skip_cpu:
            threads = os.cpu_count() or 1
            rows = min(B, max(1, -(-threads // H)))
            calib = make_cpu_inputs(rows, 64, H, r, V, seed=0)
            rate, _ = cpu_port_throughput(calib, rows, 64, threads)
            tokens = int(min(T, max(64, (rate * 15.0 / rows) // 64 * 64)))
            val, secs = cpu_port_throughput(cpu, rows, tokens, threads)
            cpu_baseline = {"value": val, "unit": "tokens/s", "cores": threads, "kind": "port",
                            "sample": f"B={rows} of {B}, first {tokens} of {T} tokens, H={H}, fwd+bwd once ({secs:.1f} s)"}
        line = {
            "metric": METRIC, "value": value, "unit": "tokens/s", "n_gpus": world, "steps": opts.steps,
            "warmup": max(opts.warmup, 3), "ms_per_step": ms_step, "higher_is_better": True,
            "scaling": "strong" if opts.strong else "weak",
            "vs_baseline": None, "dtype": "bf16", "data": "synthetic",
            "config": {"workload": f"operator fwd+bwd, B={B}{' x H=' + str(H) + ' streams on this rank of one B=8, H=8 job' if opts.strong else ' per GPU'}, H={H}, T={T}, r=V={r}, chunk=64, "
                                   "non-zero C0/S0 and state cotangents",
                       "l2": "inputs of one step (0.7 GB) exceed the 126 MB L2; no flush needed",
                       "arithmetic": "bf16 operands, tf32 tensor-core contractions, fp32 states",
                       "tolerance": "parity tests: norm-wise max relative error max|a-b|/max|b| per tensor, "
                                    "2e-2 outputs and gradients, 1e-3 FP32 states; relative L2 3e-2 on gradients",
                       "timing": f"median of {REPEATS} blocks of --steps steps",
                       "cpu_arm": "C/OpenMP port of the upstream FP64 token loop on a bounded sample "
                                  "(see cpu_baseline.sample); not the same config as the GPU arm"},
            "ms_per_step_min": min(block_ms), "ms_per_step_max": max(block_ms), "repeats": REPEATS,
            "clocks": clocks, "e2e": e2e, "gpu_launches": runner.launches * opts.steps,
            "roofline": roofline, "kernels": kernels, "cpu_baseline": cpu_baseline,
            "forward_only": {"ms_per_step": fwd_ms, "value": job_throughput(runner.tokens, fwd_ms * 1e-3, world),
                             "unit": "tokens/s"},
            "mixer_glue": glue, "mixer_module": mixer, "gamma_zero": gamma_zero, "causal_lm": causal_lm,
        }
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


def run_model_ddp(opts, rank, world, local_rank):
    """Side measurement, not the headline metric: the reference's 24-layer training step data-parallel
    over the ranks (B=8, T=2048 per rank; graphed forward + loss + backward, one flat gradient all-reduce
    over NCCL, AdamW on FP32 masters), tokens/s of the whole job, max over ranks."""
    import torch
    import torch.distributed as dist

    from solvedelta_b200 import BF16ShadowWeights, SolveDeltaConfig, SolveDeltaForCausalLM, SolveDeltaGraphedTrainingStep
    from solvedelta_b200.sharding import max_over_ranks

    device = torch.device("cuda", local_rank)
    torch.cuda.set_device(device)
    if world > 1:
        dist.init_process_group("nccl", device_id=device)
    torch.manual_seed(0)   # the same initial weights on every rank
    config = SolveDeltaConfig(hidden_size=1024, num_heads=8, head_k_dim=128, head_v_dim=128,
                              num_hidden_layers=24, vocab_size=32000)
    model = SolveDeltaForCausalLM(config).prepare(device).train()
    B, T = 8, 2048
    gen = torch.Generator(device="cpu").manual_seed(100 + rank)
    ids = torch.randint(0, config.vocab_size, (B, T), generator=gen).to(device)
    shadows = BF16ShadowWeights(model, lambda masters: torch.optim.AdamW(masters, lr=1e-4, fused=True))
    if opts.ddp_mode == "graphed":
        graphed = SolveDeltaGraphedTrainingStep(model, ids, ids, num_warmup_iters=2, distributed=world > 1)
        step = lambda: graphed(ids, ids)
    else:
        # eager forward / backward; gradients live in flat buckets whose all-reduces start from autograd
        # hooks while backward is still running
        from solvedelta_b200 import BucketedGradientAverager, causal_lm_loss

        averager = BucketedGradientAverager(model.parameters())

        def step():
            loss = causal_lm_loss(model, ids, ids, total=B * (T - 1))
            loss.backward()
            averager.finish()
            return loss.detach()
    for _ in range(max(opts.warmup, 3)):
        step()
        shadows.optimizer.step()
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(opts.steps):
        loss = step()
        shadows.optimizer.step()
    e1.record()
    torch.cuda.synchronize()
    ms = max_over_ranks(e0.elapsed_time(e1) / opts.steps, device) if world > 1 else e0.elapsed_time(e1) / opts.steps
    # every rank must hold the same weights after the averaged updates
    probe = model.lm_head.weight.float().sum().reshape(1)
    if world > 1:
        gathered = [torch.zeros_like(probe) for _ in range(world)]
        dist.all_gather(gathered, probe)
        same = all(torch.equal(g, gathered[0]) for g in gathered)
    else:
        same = True
    if rank == 0:
        print(json.dumps({"metric": "SolveDelta CausalLM training tokens/s (24 layers, hidden 1024, vocab 32000)",
                          "value": world * B * T / (ms * 1e-3), "unit": "tokens/s", "n_gpus": world,
                          "steps": opts.steps, "ms_per_step": ms, "scaling": "weak", "dtype": "bf16",
                          "data": "synthetic", "loss": float(loss), "weights_equal_across_ranks": same,
                          "config": {"workload": f"B={B}, T={T} per GPU; " + (
                              "graphed fwd + chunked loss + bwd, one flat NCCL gradient all-reduce after the replay"
                              if opts.ddp_mode == "graphed" else
                              "eager fwd + chunked loss + bwd, bucketed NCCL gradient all-reduces launched from "
                              "autograd hooks during backward") + ", fused AdamW on FP32 masters"}}), flush=True)
    if world > 1:
        dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--case", default="full", choices=["full", "medium", "small"],
                    help="profiler captures only: medium = B=8, T=1024 (1024 chunk tasks, larger than L2), "
                         "small = B=2, T=1024; the reported metric is defined on full")
    ap.add_argument("--skip-e2e", action="store_true", help="skip the host-buffer leg (profiler captures)")
    ap.add_argument("--skip-cpu", action="store_true", help="skip the CPU baseline leg (profiler captures)")
    ap.add_argument("--skip-glue", action="store_true", help="skip the mixer glue kernels (profiler captures)")
    ap.add_argument("--skip-model", action="store_true", help="skip the 24-layer causal LM legs")
    ap.add_argument("--summarize-ncu", metavar="CSV", default=None,
                    help="no GPU work: turn an ncu --csv log of one step's launches (medium case, 1024 chunk tasks) "
                         "into the DRAM table of profiles/ on stdout")
    ap.add_argument("--strong", action="store_true",
                    help="strong scaling: the B x H streams of ONE workload are dealt out over the ranks "
                         "(default: weak scaling, every rank its own B=8 batch)")
    ap.add_argument("--ddp-mode", default="graphed", choices=["bucketed", "graphed"],
                    help="--model-ddp only: bucketed all-reduces overlapped with an eager backward, or one flat "
                         "all-reduce after a graph-replayed step")
    ap.add_argument("--model-ddp", action="store_true",
                    help="side measurement: only the data-parallel 24-layer training step at the launched world size")
    opts = ap.parse_args()
    if opts.summarize_ncu:
        summarize_ncu(opts.summarize_ncu, tasks=8 * 8 * (1024 // 64))
        return
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if opts.impl == "reference":
        run_reference(opts, rank, world)
        return
    if opts.model_ddp:
        run_model_ddp(opts, rank, world, local_rank)
        return
    run_ours(opts, rank, world, local_rank)


if __name__ == "__main__":
    main()
