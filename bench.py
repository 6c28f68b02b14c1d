#!/usr/bin/env python3
"""KDA prefill benchmark on B200: tokens/s of the serving call (H = 64, K = V = 128, varlen) at 1/2/4/8 GPUs.

    python bench.py [--gpus N] [--steps K] [--warmup W]            # N > 1: launched by torch.distributed.run
    python bench.py --impl reference ...                            # the CPU restatement of the reference's definition

Workload (the H = 64 varlen serving configuration the metric is quoted on): a paged fp32
state pool of 256 slots, 48 requests on random distinct slots, new-token lengths lognormal(ln 1024, 0.8) clipped to
[16, 8192], bf16 checkpoints every 1024 tokens, pre-activated inputs (bf16 q/k/v, fp32 log-decay g and beta).
Synthetic seeded data.  With N GPUs the 64 heads are sharded N ways (no collective on the data path: strong scaling).

A step is one prefill call (device planner + fused chunk kernel) over the whole batch.  Inputs (several GB) are far
larger than L2, so every step streams them from HBM.  Timing: CUDA events on the launching stream, barrier +
synchronize on both sides, max over ranks.  One JSON line on stdout from rank 0.
"""
from __future__ import annotations

import argparse
import json
import math
import os
import statistics
import subprocess
import sys
import tempfile
import time
from pathlib import Path

import torch

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT / "eat-kernels_b200"))

D = 128
H_TOTAL = 64
N_REQ = 48
POOL_SLOTS = 256
CK_EVERY = 1024
FLOP_PER_TOKEN_HEAD = 6 * D * D + 4 * 64 * (D + D)          # 163 840, canonical chunk 64
BYTES_PER_TOKEN_HEAD = 3 * D * 2 + D * 4 + 4 + D * 2         # q,k,v bf16 + g fp32 + beta fp32 + out bf16 = 1540
METRIC = "KDA prefill tokens/s (H=64,K=V=128 varlen)"
# dram__bytes_read.sum + dram__bytes_write.sum of kda_chunk_umma_kernel per token-head, taken from one ncu capture of
# `bench.py --small` (DRAM traffic grows in proportion to token-heads: the kernel streams every operand once).  A
# constant from that capture, not a live measurement: counters cannot be read inside a timed run.
NCU_DRAM_BYTES_PER_TOKEN_HEAD = 1693.1


def workload_lengths(seed=2):
    gen = torch.Generator().manual_seed(seed)
    ln = torch.exp(torch.randn(N_REQ, generator=gen) * 0.8 + math.log(1024.0))
    return [int(x) for x in ln.clamp(16, 8192).round().tolist()]


def peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        j = json.loads(p.read_text())
        return {"hbm_gbs": float(j["hbm_gbs"]), "tf": float(j.get("bf16_tflops_sustained", j["bf16_tflops"])),
                "tf_burst": float(j["bf16_tflops"]), "src": "measured"}
    return {"hbm_gbs": 6650.0, "tf": 1400.0, "tf_burst": 1590.0, "src": "fallback"}


class ClockSampler:
    QUERY = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
             "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
             "clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        try:
            self.p = subprocess.Popen(["nvidia-smi", f"--id={index}", f"--query-gpu={self.QUERY}", "--format=csv,noheader,nounits",
                                       "-lms", "100"], stdout=self.f, stderr=subprocess.DEVNULL)
        except OSError:
            self.p = None

    def stop(self):
        if self.p is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.p.terminate()
        try:
            self.p.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.p.kill()
        self.f.flush()
        rows = [r.split(",") for r in Path(self.f.name).read_text().strip().splitlines() if r.count(",") >= 8]
        os.unlink(self.f.name)
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in rows:
            try:
                sm.append(float(r[1])); mx.append(float(r[2]))
            except ValueError:
                continue
            for n, val in zip(names, r[5:9]):
                if val.strip().lower().startswith("active"):
                    reasons.add(n)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "samples": len(sm), "reasons": sorted(reasons)}


def make_device_inputs(H, lens, seed, dev):
    """Pre-activated inputs of the head shard on the device: q, k normalised then bf16, v bf16, g = logsigmoid(N(0,1))
    fp32, beta = sigmoid(N(0,1)) fp32."""
    gen = torch.Generator(device=dev).manual_seed(seed)
    T = sum(lens)
    q = torch.nn.functional.normalize(torch.randn(1, T, H, D, generator=gen, device=dev), dim=-1).to(torch.bfloat16)
    k = torch.nn.functional.normalize(torch.randn(1, T, H, D, generator=gen, device=dev), dim=-1).to(torch.bfloat16)
    v = torch.randn(1, T, H, D, generator=gen, device=dev).to(torch.bfloat16)
    g = torch.nn.functional.logsigmoid(torch.randn(1, T, H, D, generator=gen, device=dev))
    beta = torch.sigmoid(torch.randn(1, T, H, generator=gen, device=dev))
    return q, k, v, g, beta


def _oracle():
    sys.path.insert(0, str(ROOT / "oracle"))
    import c_oracle
    import kda_oracle as ko
    return c_oracle, ko


def verify_serving(tensors, lens, pool0, slots, ck_every, result, heads):
    """Checks one prefill of the serving workload against the fp64 recurrence on a subset of heads (heads are independent,
    so a head slice of the inputs is a complete problem for the CPU oracle): output rows, the touched pool slots and the
    checkpoint rows.  Same acceptance test as the parity suite (every element within half the gold RMS or 5 % of its
    magnitude, relative L2 < 1e-2).  Returns the largest relative L2 seen; raises SystemExit on a mismatch."""
    c_oracle, ko = _oracle()
    q, k, v, g, beta = (t[:, :, heads].cpu() for t in tensors)
    out, pool, ck = result
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    S = pool0[slots.long()][:, heads].cpu()
    gold_o = torch.zeros(q.shape, dtype=torch.float32)
    rows = [[] for _ in lens]
    waves = -(-max(lens) // ck_every) if ck_every else 1
    for j in range(waves):          # segment j of every sequence that still has one: one oracle call per wave
        step = ck_every if ck_every else max(lens)
        segs = [(n, starts[n] + j * step, starts[n] + min(lens[n], (j + 1) * step)) for n in range(len(lens)) if j * step < lens[n]]
        ids = [n for n, _, _ in segs]
        for n in ids:
            rows[n].append(S[n].clone())
        tok = torch.cat([torch.arange(a, b) for _, a, b in segs])
        cu = [0]
        for _, a, b in segs:
            cu.append(cu[-1] + b - a)
        o, f = c_oracle.recurrence_plain(q[:, tok], k[:, tok], v[:, tok], g[:, tok], beta[:, tok], D ** -0.5, S[ids], cu)
        gold_o[:, tok] = o
        S[ids] = f
    worst = 0.0
    try:
        worst = max(worst, ko.check_close(out[:, :, heads].float().cpu(), gold_o, "bench verification: output")[1])
        worst = max(worst, ko.check_close(pool[slots.long()][:, heads].cpu(), S, "bench verification: pool slots")[1])
        if ck_every:
            gold_ck = torch.stack([r for rs in rows for r in rs])
            worst = max(worst, ko.check_close(ck[:, heads].float().cpu(), gold_ck, "bench verification: checkpoint rows")[1])
    except AssertionError as e:
        raise SystemExit(f"bench: {e}")
    return worst


def cpu_baseline(lens, H, target_s=12.0):
    """The oracle's C restatement of the reference recurrence (fp32 working precision, OpenMP over sequence-heads) on
    a bounded prefix of the same workload; returns the cpu_baseline object."""
    sys.path.insert(0, str(ROOT / "oracle"))
    import c_oracle
    import kda_oracle as ko
    # every host CPU, whatever OMP_NUM_THREADS says (torch.distributed.run exports OMP_NUM_THREADS=1 to its children)
    threads = c_oracle.set_threads(0, "f32")

    def run(n_tok):
        sample_lens, left = [], n_tok
        for L in lens:
            if left <= 0:
                break
            sample_lens.append(min(L, left)); left -= sample_lens[-1]
        q, k, v, g, beta, scale, init, cu = ko.make_inputs_plain(H, sample_lens, 5)
        t = time.perf_counter()
        c_oracle.recurrence_plain(q, k, v, g, beta, scale, init, cu, precision="f32")
        return sum(sample_lens), time.perf_counter() - t, len(sample_lens)

    run(64)                                            # touch the library
    n0, t0, _ = run(256)
    n_tok = int(min(sum(lens), max(256, 256 * target_s / max(t0, 1e-3))))
    n, t, nseq = run(n_tok)
    return {"value": n / t, "unit": "tokens/s", "cores": threads, "kind": "port",
            "sample": f"first {n} tokens ({nseq} sequences) of the workload at H={H}, fp32 C restatement of "
                      f"kda/b200/reference.py, {threads} OpenMP threads of {os.cpu_count()} host CPUs, {t:.1f} s"}, n, t


def run_reference(args, lens):
    """--impl reference: the CPU implementation of the path (oracle port: the reference's own CPU code is Python and
    its CUDA path needs a GPU build) timed per step on a bounded sample of the workload."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return 0
    base, n, t = cpu_baseline(lens, H_TOTAL, target_s=3.0)
    times = []
    sys.path.insert(0, str(ROOT / "oracle"))
    import c_oracle
    import kda_oracle as ko
    sample_lens, left = [], n
    for L in lens:
        if left <= 0:
            break
        sample_lens.append(min(L, left)); left -= sample_lens[-1]
    q, k, v, g, beta, scale, init, cu = ko.make_inputs_plain(H_TOTAL, sample_lens, 5)
    for i in range(args.warmup + args.steps):
        t0 = time.perf_counter()
        c_oracle.recurrence_plain(q, k, v, g, beta, scale, init, cu, precision="f32")
        if i >= args.warmup:
            times.append(time.perf_counter() - t0)
    sec = sum(times) / len(times)
    value = n / sec
    base["value"] = value
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": "tokens/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": sec * 1e3, "higher_is_better": True,
            "scaling": "strong", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": "configs[2] serving call H=64 K=V=128, 48 requests lognormal lengths; CPU arm runs "
                                   f"a prefix of {n} tokens per step (tokens/s is per token, so the sample is comparable)",
                       "heads": H_TOTAL, "same_config": "prefix sample of the same workload", "threads": base["cores"]},
            "cpu_baseline": base,
            "e2e": {"value": value, "unit": "tokens/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line))
    return 0


def run_layouts(args, dev, kda_b200):
    """ONE captured CUDA graph (token capacity 32768, H = 64, up to 512 sequences, pool of 1024 slots)
    replayed over four batch layouts by rewriting cu_seqlens in place; trailing sequences are empty."""
    import random
    T, H, N_CAP, SLOTS = 32768, H_TOTAL, 512, 1024
    gen = torch.Generator(device=dev).manual_seed(11)
    q = torch.nn.functional.normalize(torch.randn(1, T, H, D, generator=gen, device=dev), dim=-1).to(torch.bfloat16)
    k = torch.nn.functional.normalize(torch.randn(1, T, H, D, generator=gen, device=dev), dim=-1).to(torch.bfloat16)
    v = torch.randn(1, T, H, D, generator=gen, device=dev).to(torch.bfloat16)
    g = torch.nn.functional.logsigmoid(torch.randn(1, T, H, D, generator=gen, device=dev) + 2.0)
    beta = torch.sigmoid(torch.randn(1, T, H, generator=gen, device=dev))
    pool = torch.randn(SLOTS, H, D, D, generator=gen, device=dev) * 0.05
    slots = torch.randperm(SLOTS, generator=torch.Generator().manual_seed(3))[:N_CAP].to(torch.int32).to(dev)
    rng = random.Random(5)
    mix, left = [], T
    while left > 0:
        n = min(left, rng.randint(1, 4096))
        mix.append(n)
        left -= n
    layouts = {"1x32768": [T], "32x1024": [1024] * 32, "512x64": [64] * 512, f"mix of {len(mix)} (U[1,4096])": mix}

    def cu_of(lens):
        c = [0]
        for n in lens:
            c.append(c[-1] + n)
        c += [T] * (N_CAP + 1 - len(c))
        return torch.tensor(c, dtype=torch.int64, device=dev)

    cu = cu_of(layouts["32x1024"])
    launch = kda_b200.prepare_plain(q, k, v, g, beta, D ** -0.5, pool, False, cu, dynamic_layout=True, ssm_state_indices=slots)
    for _ in range(3):
        launch()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        launch()
    res = {}
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for name, lens in layouts.items():
        cu.copy_(cu_of(lens))
        for _ in range(max(3, args.warmup)):
            graph.replay()
        torch.cuda.synchronize()
        e0.record()
        for _ in range(args.steps):
            graph.replay()
        e1.record()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1) / args.steps
        if kda_b200.status_bits(launch) != 0 or kda_b200.kernel_error(launch) != 0:
            raise SystemExit(f"bench: layout {name} reported a table or kernel error")
        res[name] = {"ms": round(ms, 4), "tokens_per_s": T / (ms * 1e-3)}
    # ---- host latency of the public calls (no synchronisation inside; the reference states limits for its run():
    # <= 1 ms + 0.01 ms per sequence for a repeated layout, <= 2 ms + 0.025 ms per sequence for a new one,
    # kda/b200/README.md:39-41).  Nothing is planned on the host here, so "new" and "repeated" layouts cost the same.
    host = {}
    for n_seq in (1, 32, 512):
        lens_h = [T // n_seq] * n_seq
        cu_h = torch.tensor([0, *torch.tensor(lens_h).cumsum(0).tolist()], dtype=torch.int64, device=dev)
        slots_h = slots[:n_seq].contiguous()

        def t_of(fn, reps=15):
            ts = []
            for _ in range(reps):
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                r = fn()
                ts.append((time.perf_counter() - t0) * 1e6)
                del r
            return sorted(ts)[len(ts) // 2]

        mk = lambda: kda_b200.prepare_plain(q, k, v, g, beta, D ** -0.5, pool, False, cu_h, dynamic_layout=True,  # noqa: E731
                                            ssm_state_indices=slots_h)
        lh = mk()
        host[f"N={n_seq}"] = {"prepare_us": round(t_of(mk), 1), "launch_us": round(t_of(lh), 1),
                              "run_us": round(t_of(lambda: mk()()), 1)}
        limit_us = 1000.0 + 10.0 * n_seq
        if host[f"N={n_seq}"]["run_us"] > limit_us:
            raise SystemExit(f"bench: host time of run() with {n_seq} sequences is {host[f'N={n_seq}']['run_us']} us, "
                             f"over the reference's limit of {limit_us} us")
    print(json.dumps({"metric": "KDA prefill tokens/s (H=64,K=V=128, one CUDA graph over batch layouts)", "unit": "tokens/s",
                      "n_gpus": 1, "steps": args.steps, "warmup": args.warmup, "higher_is_better": True, "dtype": "bf16",
                      "data": "synthetic",
                      "config": {"workload": "configs[4]: token capacity 32768, H=64, 512 sequence slots, pool of 1024 slots, "
                                             "g=logsigmoid(N(2,1)); one captured graph, cu_seqlens rewritten in place"},
                      "layouts": res, "host_latency": host,
                      "host_latency_limit": "run() <= 1000 us + 10 us per sequence (kda/b200/README.md:39-41); asserted"}))
    return 0


def run_headline(args, dev, kda_b200):
    """The single-GPU cases the reference publishes latencies for (kda/b200/README.md:84-116), with its own front-end
    (bf16 gate and beta logits, A_log, dt_bias, L2 norm in the kernel), each call captured in a CUDA graph and timed
    with a cold L2 (a 256 MB buffer is rewritten before every replay), median of the timed replays."""
    from kda_b200 import parallel
    cases = [("H=64, 1x8192", 64, [8192], 0, 0.2394), ("H=64, 8x1024", 64, [1024] * 8, 0, 0.1767),
             ("H=96, 1x8192", 96, [8192], 0, 0.3034), ("H=96, 8x1024", 96, [1024] * 8, 0, 0.2524),
             ("H=16, 1x32768, pool + bf16 checkpoints / 64", 16, [32768], 64, 0.4510),
             ("H=12, 1x32768, pool + bf16 checkpoints / 64", 12, [32768], 64, 0.3645)]
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)
    out = {}
    for name, H, lens, every, ref_ms in cases:
        T, N = sum(lens), len(lens)
        gen = torch.Generator(device=dev).manual_seed(31 + H)
        mk = lambda *shape: torch.randn(*shape, generator=gen, device=dev).to(torch.bfloat16)
        q, k, v, g, beta = mk(1, T, H, D), mk(1, T, H, D), mk(1, T, H, D), mk(1, T, H, D), mk(1, T, H)
        A_log = torch.zeros(H, device=dev)
        dt_bias = torch.zeros(H * D, device=dev)
        cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int64, device=dev)
        init = torch.randn(N, H, D, D, generator=gen, device=dev) * 0.05
        kw = {}
        if every:
            rows = sum(-(-n // every) for n in lens)
            counts = [-(-n // every) for n in lens]
            kw = dict(dynamic_layout=True, ssm_state_indices=torch.arange(N, dtype=torch.int32, device=dev),
                      state_checkpoints=torch.zeros(rows, H, D, D, dtype=torch.bfloat16, device=dev),
                      checkpoint_cu_starts=torch.tensor([0, *torch.tensor(counts).cumsum(0).tolist()], dtype=torch.int64, device=dev),
                      checkpoint_every_n_tokens=every)
        launch = kda_b200.prepare(q, k, v, g, beta, A_log, dt_bias, D ** -0.5, init, cu, **kw)
        for _ in range(3):
            launch()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            launch()

        def timed(fn):
            ts = []
            for _ in range(max(5, args.steps)):
                flush.fill_(1)
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record()
                fn()
                e1.record()
                torch.cuda.synchronize()
                ts.append(e0.elapsed_time(e1))
            return sorted(ts)[len(ts) // 2]

        entry = {"ms": round(timed(graph.replay), 4), "reference_ms": ref_ms}
        if N == 1 and not every:
            # one long sequence without a pool: the context-parallel call on one GPU cuts it into pieces that fill the SMs
            be = parallel.CudaBackend()
            fn = lambda: parallel.context_parallel_prefill(q, k, v, g, beta, A_log, dt_bias, D ** -0.5, init, backend=be)
            fn()
            entry["ms_context_parallel_call"] = round(timed(fn), 4)
        if N == 1 and every:
            # one long sequence on few heads with checkpoint rows: the cut-sequence launch (two passes over pieces)
            pool = init.clone()
            cut = parallel.prepare_cut_sequence(q, k, v, g, beta, A_log, dt_bias, D ** -0.5, pool, 0,
                                                state_checkpoints=kw["state_checkpoints"], checkpoint_every_n_tokens=every)
            for _ in range(3):
                cut()
            torch.cuda.synchronize()
            g2 = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g2):
                cut()
            entry["ms_cut_sequence_call"] = round(timed(g2.replay), 4)
            entry["pieces"] = cut.pieces
        entry["tokens_per_s"] = T / (min(entry["ms"], entry.get("ms_context_parallel_call", 1e9), entry.get("ms_cut_sequence_call", 1e9)) * 1e-3)
        out[name] = entry
    print(json.dumps({"metric": "latency of the reference's published single-GPU cases (raw front-end, cold L2, CUDA graph)",
                      "unit": "ms", "n_gpus": 1, "higher_is_better": False, "data": "synthetic", "cases": out}))
    return 0


def measure_longctx(args, world, rank, dev, steps, warmup, verify=True):
    """one sequence of 131072 tokens, H = 96, slow decay g = logsigmoid(N(2,1)), zero initial state; the
    tokens are sharded over the ranks, per-rank affine state maps are all-gathered over NCCL, scanned and fixed up.
    Returns the measurement as a dict on rank 0 (None elsewhere).  With `verify` two heads of the whole sequence are
    checked against the fp64 recurrence on rank 0's host (every rank ships those heads' inputs and output rows)."""
    import torch.distributed as dist
    from kda_b200 import parallel
    T_total, H = args.longctx_tokens, 96
    shards = parallel.balanced_shards(T_total, world, H) if not args.equal_shards else [T_total // world] * world
    T = shards[rank]
    gen = torch.Generator(device=dev).manual_seed(200 + rank)
    q = torch.nn.functional.normalize(torch.randn(1, T, H, D, generator=gen, device=dev), dim=-1).to(torch.bfloat16)
    k = torch.nn.functional.normalize(torch.randn(1, T, H, D, generator=gen, device=dev), dim=-1).to(torch.bfloat16)
    v = torch.randn(1, T, H, D, generator=gen, device=dev).to(torch.bfloat16)
    g = torch.nn.functional.logsigmoid(torch.randn(1, T, H, D, generator=gen, device=dev) + 2.0)
    beta = torch.sigmoid(torch.randn(1, T, H, generator=gen, device=dev))
    pieces = args.pieces            # 0: the library plans the piece boundaries by simulating the segment launch
    be = parallel.CudaBackend()

    def step():
        return parallel.context_parallel_prefill(q, k, v, g, beta, None, None, D ** -0.5, None, pieces=pieces, raw=False, backend=be)

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    for _ in range(max(1, warmup)):
        out, fin = step()
    barrier()
    verification = None
    if verify:
        heads = [0, H - 1]
        mine = [t[:, :, heads].cpu() for t in (q, k, v, g, beta, out)]
        if world > 1:
            gathered = [None] * world if rank == 0 else None
            dist.gather_object(mine, gathered, dst=0)
        else:
            gathered = [mine]
        if rank == 0:
            c_oracle, ko = _oracle()
            c_oracle.set_threads(0)
            full = [torch.cat([r[i] for r in gathered], dim=1) for i in range(6)]
            gold_o, gold_s = c_oracle.recurrence_plain(*full[:5], D ** -0.5, None, None)
            try:
                r1 = ko.check_close(full[5].float(), gold_o, "bench verification (configs[3]): output of every rank")[1]
                r2 = ko.check_close(fin[:, heads].transpose(-1, -2).cpu(), gold_s, "bench verification (configs[3]): final state")[1]
            except AssertionError as e:
                raise SystemExit(f"bench: {e}")
            verification = {"verified": True, "rel_l2_max": max(r1, r2), "heads_checked": heads,
                            "what": "output rows of every rank and the final state vs the fp64 recurrence"}
        barrier()
    sampler = ClockSampler(dev.index) if rank == 0 else None
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier()
    e0.record()
    for _ in range(steps):
        out, fin = step()
    e1.record()
    barrier()
    ms = e0.elapsed_time(e1) / steps
    if world > 1:
        t = torch.tensor([ms], device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    finite = bool(torch.isfinite(out.float()).all()) and bool(torch.isfinite(fin).all())
    if not finite:
        raise SystemExit("bench: the context-parallel call produced non-finite values")
    clocks = sampler.stop() if sampler else None
    # one more step with CUDA events at the phase boundaries (this rank's view; not part of the timed region)
    ev = []
    parallel.context_parallel_prefill(q, k, v, g, beta, None, None, D ** -0.5, None, pieces=pieces, raw=False, backend=be, events=ev)
    torch.cuda.synchronize()
    phases = {b[0]: round(a[1].elapsed_time(b[1]), 4) for a, b in zip(ev[:-1], ev[1:])}
    all_phases = [phases]
    if world > 1:
        all_phases = [None] * world
        dist.all_gather_object(all_phases, phases)
    bounds = parallel.plan_bounds(T, H, rank == 0) if pieces <= 0 else parallel.split_pieces(T, pieces)
    mapped_tokens = T - (bounds[1] if rank == 0 else 0)
    fix_bytes = mapped_tokens * H * 3 * D * 2 + (len(bounds) - 1 - (1 if rank == 0 else 0)) * H * D * D * 4
    if rank != 0:
        return None
    pk = peaks()
    flops = T_total * H * FLOP_PER_TOKEN_HEAD
    algo_bytes = T_total * H * BYTES_PER_TOKEN_HEAD + H * 2 * D * D * 4
    return {
        "metric": f"KDA prefill tokens/s (H=96,K=V=128, one {T_total}-token sequence, context-parallel)", "value": T_total / (ms * 1e-3),
        "unit": "tokens/s", "n_gpus": world, "steps": steps, "warmup": warmup, "ms_per_step": ms,
        "higher_is_better": True, "scaling": "strong", "vs_baseline": None, "dtype": "bf16", "data": "synthetic",
        "config": {"workload": f"configs[3]: T={T_total}, H=96, g=logsigmoid(N(2,1)), zero initial state", "piece_bounds_rank0": bounds,
                   "tokens_per_rank": shards, "parallelism": f"cp{world}", "finite": finite},
        "verification": verification, "verified": bool(verification),
        "roofline": {"bound": "hbm", "achieved": algo_bytes / (ms * 1e-3) / 1e9, "peak": pk["hbm_gbs"], "unit": "GB/s",
                     "frac": algo_bytes / (ms * 1e-3) / 1e9 / pk["hbm_gbs"], "traffic": None, "peak_source": pk["src"]},
        "tensor": {"achieved": flops / (ms * 1e-3) / 1e12, "peak": pk["tf"], "unit": "TFLOP/s",
                   "frac": flops / (ms * 1e-3) / 1e12 / pk["tf"]},
        "phases_ms_rank0": phases, "segments_ms_per_rank": [ph.get("segments") for ph in all_phases],
        "fixup": {"bytes": fix_bytes, "GB/s": (fix_bytes / (phases["fixup"] * 1e-3) / 1e9) if phases.get("fixup", 0) > 0 else None,
                  "note": "o_loc + Qt read, out written (768 B per mapped token-head) plus the entering states"},
        "clocks": clocks}


def run_longctx(args, world, rank, dev, kda_b200):
    import torch.distributed as dist
    line = measure_longctx(args, world, rank, dev, args.steps, args.warmup, verify=not args.no_verify)
    if rank == 0:
        print(json.dumps(line))
    if world > 1:
        dist.destroy_process_group()
    return 0


def main(argv=None):
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--e2e-steps", type=int, default=3)
    ap.add_argument("--e2e-groups", type=int, default=6, help="end-to-end arm: request groups whose copies and prefills overlap")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-verify", action="store_true", help="skip the oracle verification before timing (profiler captures)")
    ap.add_argument("--no-longctx", action="store_true", help="N > 1: skip the context-parallel configs[3] measurement")
    ap.add_argument("--small", action="store_true", help="8 requests, for profiler captures (not a bench value)")
    ap.add_argument("--shard-of", type=int, default=1, help="one GPU runs the head shard that each of N GPUs would run "
                    "(tuning the few-heads case without N GPUs; not a bench value)")
    ap.add_argument("--workload", default="serving", choices=["serving", "longctx", "layouts", "headline"],
                    help="serving = configs[2] (the default, head-parallel); longctx = configs[3], one 131072-token "
                         "sequence at H=96, context-parallel over the ranks")
    ap.add_argument("--pieces", type=int, default=0, help="longctx: equal pieces per rank (0 = boundaries planned by simulating the segment launch)")
    ap.add_argument("--equal-shards", action="store_true", help="longctx: equal token shards instead of cost-balanced ones")
    ap.add_argument("--longctx-tokens", type=int, default=131072, help="longctx: sequence length (smaller values for profiler captures)")
    args = ap.parse_args(argv)
    args.warmup = max(args.warmup, 3) if args.impl == "ours" else args.warmup
    lens = workload_lengths()
    if args.small:
        lens = lens[:8]
    if args.impl == "reference":
        return run_reference(args, lens)

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world != args.gpus:
        raise SystemExit(f"--gpus {args.gpus} but WORLD_SIZE={world}: launch N > 1 with torch.distributed.run")
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl", device_id=dev)
    import kda_b200

    if args.workload == "longctx":
        return run_longctx(args, world, rank, dev, kda_b200)
    if args.workload == "headline":
        if world > 1:
            raise SystemExit("--workload headline runs on one GPU")
        return run_headline(args, dev, kda_b200)
    if args.workload == "layouts":
        if world > 1:
            raise SystemExit("--workload layouts runs on one GPU")
        return run_layouts(args, dev, kda_b200)
    assert H_TOTAL % (world * args.shard_of) == 0
    H = H_TOTAL // (world * args.shard_of)
    T, N = sum(lens), len(lens)
    q, k, v, g, beta = make_device_inputs(H, lens, 100 + rank, dev)
    gen = torch.Generator(device=dev).manual_seed(7)
    pool = torch.randn(POOL_SLOTS, H, D, D, generator=gen, device=dev) * 0.05
    slots = torch.randperm(POOL_SLOTS, generator=torch.Generator().manual_seed(3))[:N].to(torch.int32).to(dev)
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int64, device=dev)
    counts = [-(-n // CK_EVERY) for n in lens]
    ck_starts = torch.tensor([0, *torch.tensor(counts).cumsum(0).tolist()], dtype=torch.int64, device=dev)
    rows = sum(counts)
    ck = torch.zeros(rows, H, D, D, dtype=torch.bfloat16, device=dev)
    launch = kda_b200.prepare_plain(q, k, v, g, beta, D ** -0.5, pool, False, cu, dynamic_layout=True,
                                    ssm_state_indices=slots, state_checkpoints=ck, checkpoint_cu_starts=ck_starts,
                                    checkpoint_every_n_tokens=CK_EVERY)
    # kernels of this library per step: planner + chunk kernel, and with cut capacity the scan of cut chains + the
    # chunk kernel's second launch (both run every step; they find no work when the planner cuts nothing)
    launches_per_step = 4 if launch._args.max_cut_pieces > 0 else 2

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    # ---- verification, before timing and again after an in-place refill of every input (the launch re-reads the same
    # buffers), as the reference's own benchmark does (kda/b200/bench.py:182-187): two heads of this rank's shard
    # against the fp64 recurrence on the CPU.
    verified = None
    if not args.no_verify:
        heads = sorted({0, H - 1})
        pool0 = pool.clone()
        res = launch()
        torch.cuda.synchronize()
        rel = verify_serving((q, k, v, g, beta), lens, pool0, slots, CK_EVERY, res, heads)
        q2, k2, v2, g2, beta2 = make_device_inputs(H, lens, 500 + rank, dev)
        for dst_, src_ in ((q, q2), (k, k2), (v, v2), (g, g2), (beta, beta2)):
            dst_.copy_(src_)
        del q2, k2, v2, g2, beta2
        pool.copy_(pool0)
        ck.zero_()
        res = launch()
        torch.cuda.synchronize()
        rel = max(rel, verify_serving((q, k, v, g, beta), lens, pool0, slots, CK_EVERY, res, heads))
        del pool0
        verified = {"verified": True, "rel_l2_max": rel, "heads_checked": heads,
                    "what": "output, touched pool slots and bf16 checkpoint rows vs the fp64 recurrence, before timing "
                            "and after an in-place refill of q, k, v, g, beta"}

    sampler = ClockSampler(local) if rank == 0 else None
    for _ in range(args.warmup):
        launch()
    barrier()
    if kda_b200.status_bits(launch) != 0 or kda_b200.kernel_error(launch) != 0:
        raise SystemExit("bench: the launch reported a table or kernel error")
    t_load = time.perf_counter()
    while rank == 0 and time.perf_counter() - t_load < 0.6:     # keep the GPU busy until nvidia-smi has sampled
        launch()
    barrier()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier()
    e0.record()
    for _ in range(args.steps):
        launch()
    e1.record()
    barrier()
    ms = e0.elapsed_time(e1) / args.steps
    if world > 1:
        t = torch.tensor([ms], device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    clocks = sampler.stop() if sampler else None

    # ---- end to end through the public call with HOST buffers: pinned inputs -> device -> prefill -> output to host.
    # The requests are served in a few groups of consecutive sequences, each with its own prepared launch over slices of
    # the same buffers, so that the host-to-device copy of the next group, the prefill of the current one and the
    # device-to-host copy of the previous one overlap (the step is bound by the PCIe link, which is full duplex).
    e2e = None
    if args.e2e_steps > 0:
        n_groups = max(1, min(args.e2e_groups, N))
        target, acc, cuts = T / n_groups, 0, [0]
        for i, n in enumerate(lens):
            acc += n
            if acc >= target * len(cuts) and len(cuts) < n_groups and i + 1 < N:
                cuts.append(i + 1)
        cuts.append(N)
        cu_l, ck_l = [0, *torch.tensor(lens).cumsum(0).tolist()], [0, *torch.tensor(counts).cumsum(0).tolist()]
        groups, h2d = [], 0
        for a_, b_ in zip(cuts[:-1], cuts[1:]):
            ta, tb, ra, rb = cu_l[a_], cu_l[b_], ck_l[a_], ck_l[b_]
            dv = [q[:, ta:tb], k[:, ta:tb], v[:, ta:tb], g[:, ta:tb], beta[:, ta:tb],
                  (cu[a_:b_ + 1] - cu[a_]).contiguous(), slots[a_:b_].contiguous(), (ck_starts[a_:b_ + 1] - ck_starts[a_]).contiguous()]
            hv = [t.cpu().pin_memory() for t in dv]
            h2d += sum(t.numel() * t.element_size() for t in hv)
            lg = kda_b200.prepare_plain(dv[0], dv[1], dv[2], dv[3], dv[4], D ** -0.5, pool, False, dv[5], dynamic_layout=True,
                                        ssm_state_indices=dv[6], state_checkpoints=ck[ra:rb], checkpoint_cu_starts=dv[7],
                                        checkpoint_every_n_tokens=CK_EVERY)
            groups.append((dv, hv, lg, ta, tb))
        out_host = torch.empty((1, T, H, D), dtype=torch.bfloat16).pin_memory()
        d2h = out_host.numel() * out_host.element_size()
        s_in, s_out = torch.cuda.Stream(dev), torch.cuda.Stream(dev)
        main = torch.cuda.current_stream(dev)

        def step():
            s_in.wait_stream(main)                       # the previous step's prefills have read the input buffers
            done = []
            for dv, hv, lg, ta, tb in groups:
                with torch.cuda.stream(s_in):
                    for d_, h_ in zip(dv, hv):
                        d_.copy_(h_, non_blocking=True)
                    ev = torch.cuda.Event()
                    ev.record(s_in)
                main.wait_event(ev)
                res = lg()
                ev2 = torch.cuda.Event()
                ev2.record(main)
                with torch.cuda.stream(s_out):
                    s_out.wait_event(ev2)
                    out_host[:, ta:tb].copy_(res[0], non_blocking=True)
                done.append(res)
            main.wait_stream(s_out)
            return done

        step()
        barrier()
        for dv, hv, lg, ta, tb in groups:
            if kda_b200.status_bits(lg) != 0 or kda_b200.kernel_error(lg) != 0:
                raise SystemExit("bench: an end-to-end launch reported a table or kernel error")
        e0.record()
        for _ in range(args.e2e_steps):
            step()
        e1.record()
        barrier()
        ems = e0.elapsed_time(e1) / args.e2e_steps
        if world > 1:
            t = torch.tensor([ems], device=dev)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ems = float(t.item())
        e2e = {"value": T / (ems * 1e-3), "unit": "tokens/s", "ms_per_step": ems, "h2d_bytes_per_step": h2d * world,
               "d2h_bytes_per_step": d2h * world, "groups": len(groups)}

    # ---- N > 1: the context-parallel configuration as well, after the headline timing, so that one
    # launch per N yields both scaling curves.  The serving tensors are released first.
    planner_counts = dict(zip(("tasks_first_launch", "tasks_second_launch", "cut_sequences"), launch.plan_counts()))
    longctx = None
    if world > 1 and not args.no_longctx and not args.small:
        del launch, q, k, v, g, beta, pool, ck
        if args.e2e_steps > 0:
            del groups, out_host
        torch.cuda.empty_cache()
        lc = measure_longctx(args, world, rank, dev, max(3, min(args.steps, 5)), 2, verify=not args.no_verify)
        if rank == 0:
            longctx = {kk: lc[kk] for kk in ("metric", "value", "unit", "ms_per_step", "steps", "config", "verification",
                                               "verified", "roofline", "phases_ms_rank0", "segments_ms_per_rank", "fixup")}

    if rank == 0:
        pk = peaks()
        algo_bytes = T * H * BYTES_PER_TOKEN_HEAD + N * H * 2 * D * D * 4 + rows * H * D * D * 2
        achieved = algo_bytes / (ms * 1e-3) / 1e9
        flops = T * H * FLOP_PER_TOKEN_HEAD
        tf = flops / (ms * 1e-3) / 1e12
        line = {
            "metric": METRIC, "value": T / (ms * 1e-3), "unit": "tokens/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "strong", "vs_baseline": None,
            "dtype": "bf16", "data": "synthetic",
            "config": {"workload": "configs[2]: serving call, H=64 (sharded by heads over the GPUs), K=V=128, 48 requests, "
                                   "lengths lognormal(ln1024,0.8) clipped [16,8192], fp32 pool of 256 slots, bf16 checkpoints "
                                   "every 1024 tokens, pre-activated bf16 q/k/v + fp32 g/beta" + (" [--small]" if args.small else ""),
                       "tokens": T, "requests": N, "heads_per_gpu": H, "checkpoint_rows": rows,
                       "planner": planner_counts,
                       "l2": "inputs (GBs per step) far exceed L2; no flush needed", "parallelism": f"hp{world}"},
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": pk["hbm_gbs"], "unit": "GB/s",
                         "frac": achieved / pk["hbm_gbs"], "traffic": None, "peak_source": pk["src"],
                         "kernel": "kda_chunk_umma_kernel (the step also holds kda_plan_kernel, 0.9 % of the time)",
                         "algorithmic_bytes_per_launch": algo_bytes},
            "tensor": {"achieved": tf, "peak": pk["tf"], "unit": "TFLOP/s", "frac": tf / pk["tf"],
                       "peak_burst": pk["tf_burst"], "frac_of_burst": tf / pk["tf_burst"],
                       "flops_per_launch": flops,
                       "note": "dense count 163840 FLOP per token-head (chunk 64 convention); `peak` is the sustained "
                               "bf16 figure, `peak_burst` the burst one: the timed region lies between the two definitions"},
            "e2e": e2e, "gpu_launches": launches_per_step * args.steps, "clocks": clocks,
        }
        if verified is not None:
            line.update(verified=True, verification=verified)
        if longctx is not None:
            line["longctx"] = longctx
        if NCU_DRAM_BYTES_PER_TOKEN_HEAD is not None:
            line["roofline"]["traffic"] = NCU_DRAM_BYTES_PER_TOKEN_HEAD * T * H
        if world == 1 and not args.no_cpu_baseline:
            line["cpu_baseline"], _, _ = cpu_baseline(lens, H_TOTAL)
        print(json.dumps(line))
    if world > 1:
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    raise SystemExit(main())
