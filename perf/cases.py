"""The work that a user of this package has it do, as measurable cases.

A case is one call of a public entry point of `kda_b200` on one batch:

    call      how the user's program calls: "plain" = `chunk_kda`, "prefill" = `kda_prefill`, "launch" = a launch made once
              by `prepare` / `prepare_plain` and called again and again, "graph" = such a launch replayed from a CUDA graph
              that was captured once for a capacity of sequences, "context" = `parallel.context_parallel_prefill`
    raw       1: bf16 gate and beta logits, activation and q/k L2 norm in the kernel; 0: fp32 log-decay and beta, normalised q/k
    heads     heads on this GPU
    requests, lengths, low, high, layout
              the batch: `requests` sequence lengths drawn from `layout` (a seed) by the rule `lengths`:
              "one" = a single sequence of `high` tokens, "equal" = all of `high` tokens, "uniform" in [low, high],
              "lognormal" around 1024 (sigma 0.8) clipped to [low, high], "fill" = uniform in [low, high] until `tokens`
              tokens are full
    pool      slots of the fp32 state pool that is updated in place (0: one state per sequence, final state returned)
    every     checkpoint rows of the state after every so many tokens (0: none), in `rows` ("bf16" or "fp32")
    slow      1: slowly decaying gates (long memory)
    capacity  sequences the captured graph is laid out for ("graph" only)
"""
import math
import random
import sys
from pathlib import Path

import torch

sys.path.insert(0, str(Path("eat-kernels_b200").resolve()))
import kda_b200  # noqa: E402
from kda_b200 import parallel  # noqa: E402

D = 128
DEV = "cuda:0"


def _case(name, call, raw, heads, lengths, high, requests=1, low=1, layout=0, tokens=0, pool=0, every=0, rows="", slow=0, capacity=0):
    return {"name": name, "call": call, "raw": raw, "heads": heads, "lengths": lengths, "requests": requests, "low": low,
            "high": high, "layout": layout, "tokens": tokens, "pool": pool, "every": every, "rows": rows, "slow": slow,
            "capacity": capacity}


def listed():
    return [
        # one short user turn appended to a conversation, on one GPU's share of the heads: latency and launches count
        _case("short_turn", "prefill", 1, 16, "one", 77, pool=8),
        # the plain call on a small batch-1 sequence (a unit of research code, or of a small model)
        _case("plain_small", "plain", 0, 4, "one", 512),
        # a handful of short ragged requests with a prefix cache in fp32
        _case("ragged_turns", "prefill", 1, 12, "uniform", 700, requests=7, low=1, layout=11, pool=32, every=64, rows="fp32"),
        # equal requests with the gate activation in the kernel
        _case("batch_1024", "launch", 1, 64, "equal", 1024, requests=8),
        # one long prompt, the whole call each time
        _case("one_8192", "prefill", 1, 96, "one", 8192),
        # one very long prompt on one GPU's share of the heads, with dense prefix-cache checkpoints
        _case("prefix_cache_32768", "launch", 1, 16, "one", 32768, pool=4, every=64, rows="bf16"),
        # packed variable-length batch through the plain call, initial and final states
        _case("plain_varlen", "plain", 0, 32, "uniform", 4096, requests=16, low=128, layout=1),
        # a serving batch: paged pool, bf16 checkpoints
        _case("serving_48", "launch", 0, 64, "lognormal", 8192, requests=48, low=16, layout=2, pool=256, every=1024, rows="bf16"),
        # the same batch on an eighth of the heads (head-parallel over eight GPUs)
        _case("serving_48_shard", "launch", 0, 8, "lognormal", 8192, requests=48, low=16, layout=2, pool=256, every=1024, rows="bf16"),
        # one captured graph laid out for 512 sequences, replayed over many short requests ...
        _case("graph_512x64", "graph", 0, 64, "equal", 64, requests=512, pool=1024, slow=1, capacity=512),
        # ... and over a few long ones
        _case("graph_mix", "graph", 0, 64, "fill", 4096, tokens=32768, layout=5, pool=1024, slow=1, capacity=512),
        # a very long context on one GPU, cut into pieces that fill it
        _case("long_context", "context", 0, 96, "one", 131072, slow=1),
    ]


def _spread(rng, low, high):
    """A whole number in [low, high], even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["turn", "turns", "plain", "plain_varlen", "launch", "serving", "prefix", "graph", "context"])
    heads = rng.choice([4, 8, 12, 16, 24, 32, 48, 64, 96])
    raw, slow, layout = rng.randint(0, 1), rng.randint(0, 1), rng.randrange(1 << 20)
    if kind == "turn":
        c = _case("", "prefill", 1, heads, "one", _spread(rng, 1, 2048), pool=rng.choice([0, 8, 32]), slow=slow)
    elif kind == "turns":
        c = _case("", "prefill", 1, heads, "uniform", _spread(rng, 64, 2048), requests=rng.randint(2, 24), layout=layout,
                  pool=rng.choice([0, 32]), slow=slow)
        if c["pool"] and rng.random() < 0.5:
            c.update(every=rng.choice([32, 64, 256]), rows=rng.choice(["fp32", "bf16"]))
    elif kind == "plain":
        c = _case("", "plain", 0, heads, "one", _spread(rng, 16, 16384), slow=slow)
    elif kind == "plain_varlen":
        c = _case("", "plain", 0, heads, "uniform", _spread(rng, 256, 4096), requests=rng.randint(2, 32), low=16, layout=layout, slow=slow)
    elif kind == "launch":
        c = _case("", "launch", raw, heads, rng.choice(["equal", "uniform"]), _spread(rng, 100, 8192), requests=rng.randint(1, 14),
                  layout=layout, slow=slow)
    elif kind == "serving":
        c = _case("", "launch", raw, heads, "lognormal", rng.choice([4096, 8192]), requests=rng.randint(8, 64), low=16, layout=layout,
                  pool=128, every=rng.choice([0, 256, 1024]), rows="bf16", slow=slow)
        if not c["every"]:
            c["rows"] = ""
    elif kind == "prefix":
        c = _case("", "launch", raw, rng.choice([4, 8, 12, 16, 24]), "one", _spread(rng, 4096, 65536), pool=4,
                  every=rng.choice([64, 128, 1024]), rows=rng.choice(["fp32", "bf16"]), slow=slow)
        while c["every"] == 64 and c["rows"] == "fp32" and c["high"] * c["heads"] > 16 * 32768:
            c["high"] //= 2
    elif kind == "graph":
        c = _case("", "graph", raw, rng.choice([8, 16, 32, 64]), "fill", _spread(rng, 48, 8192), tokens=rng.choice([8192, 16384, 32768]),
                  low=16, layout=layout, pool=512, slow=slow, capacity=rng.choice([64, 256, 512]))
        c["low"] = max(c["low"], -(-c["tokens"] // c["capacity"]))           # the requests fit the graph's capacity
        c["high"] = max(c["high"], c["low"])
    else:
        c = _case("", "context", raw, heads, "one", _spread(rng, 16384, 131072), slow=slow)
    del c["name"]
    return c


def _lengths(case):
    rng, n, low, high = random.Random(case["layout"]), case["requests"], case["low"], case["high"]
    if case["lengths"] in ("one", "equal"):
        return [high] * n
    if case["lengths"] == "uniform":
        return [rng.randint(min(low, high), high) for _ in range(n)]
    if case["lengths"] == "lognormal":
        return [int(round(min(high, max(low, 1024.0 * math.exp(0.8 * rng.gauss(0.0, 1.0)))))) for _ in range(n)]
    lens, left = [], case["tokens"]
    while left > 0:
        lens.append(min(left, rng.randint(low, high)))
        left -= lens[-1]
    return lens


def _starts(counts, total=0):
    c = [0]
    for n in counts:
        c.append(c[-1] + n)
    return torch.tensor(c + [c[-1]] * (total + 1 - len(c)), dtype=torch.int64, device=DEV)


def _normal(gen, T, H, mean=0.0, unit=False, out=torch.bfloat16, act=None):
    """[1, T, H, 128] normal values (unit: L2-normalised per head), made in slices so that no large fp32 copy is held."""
    x = torch.empty(1, T, H, D, dtype=out, device=DEV)
    step = max(1, (1 << 26) // (H * D))
    for t in range(0, T, step):
        n = min(step, T - t)
        y = torch.randn(1, n, H, D, generator=gen, device=DEV)
        if mean:
            y += mean
        if unit:
            y = torch.nn.functional.normalize(y, dim=-1)
        x[:, t:t + n] = act(y) if act is not None else y
    return x


def prepare(case, seed):
    H, lens, raw = case["heads"], _lengths(case), case["raw"]
    T, N = sum(lens), len(lens)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    s = {"call": case["call"], "raw": raw, "scale": D ** -0.5}
    s["q"], s["k"] = _normal(gen, T, H, unit=not raw), _normal(gen, T, H, unit=not raw)
    s["v"] = _normal(gen, T, H)
    if raw:
        s["g"] = _normal(gen, T, H)
        s["beta"] = torch.randn(1, T, H, generator=gen, device=DEV).to(torch.bfloat16)
        s["A_log"] = torch.zeros(H, device=DEV)
        s["dt_bias"] = torch.rand(H * D, generator=gen, device=DEV) * 6.0 - 12.0 if case["slow"] else torch.zeros(H * D, device=DEV)
    else:
        s["g"] = _normal(gen, T, H, mean=2.0 if case["slow"] else 0.0, out=torch.float32, act=torch.nn.functional.logsigmoid)
        s["beta"] = torch.sigmoid(torch.randn(1, T, H, generator=gen, device=DEV))
    slots = max(case["pool"], case["capacity"], N) if case["pool"] else N
    s["state"] = torch.randn(slots, H, D, D, generator=gen, device=DEV) * 0.05
    s["cu"] = _starts(lens, case["capacity"])
    s["serving"] = {}
    if case["pool"]:
        ids = torch.randperm(slots, generator=torch.Generator().manual_seed(seed))[:max(N, case["capacity"])]
        s["serving"]["ssm_state_indices"] = ids.to(torch.int32).to(DEV)
    if case["every"]:
        counts = [-(-n // case["every"]) for n in lens]
        s["serving"].update(state_checkpoints=torch.zeros(sum(counts), H, D, D, device=DEV, dtype=torch.bfloat16 if case["rows"] == "bf16" else torch.float32),
                            checkpoint_cu_starts=_starts(counts), checkpoint_every_n_tokens=case["every"])
    if case["call"] in ("launch", "graph"):
        if raw:
            s["launch"] = kda_b200.prepare(s["q"], s["k"], s["v"], s["g"], s["beta"], s["A_log"], s["dt_bias"], s["scale"], s["state"],
                                           s["cu"], dynamic_layout=True, **s["serving"])
        else:
            s["launch"] = kda_b200.prepare_plain(s["q"], s["k"], s["v"], s["g"], s["beta"], s["scale"], s["state"], True, s["cu"],
                                                 dynamic_layout=True, **s["serving"])
    if case["call"] == "graph":
        s["result"] = s["launch"]()                 # warm-up before the capture
        torch.cuda.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            s["launch"]()
    if case["call"] == "context":
        s["backend"] = parallel.CudaBackend(reuse=True)
    return s


def run(s):
    if s["call"] == "launch":
        return s["launch"]()
    if s["call"] == "graph":
        s["graph"].replay()
        return s["result"]
    if s["call"] == "plain":
        return kda_b200.chunk_kda(s["q"], s["k"], s["v"], s["g"], s["beta"], initial_state=s["state"], output_final_state=True,
                                  cu_seqlens=s["cu"])
    if s["call"] == "prefill":
        return kda_b200.kda_prefill(s["q"], s["k"], s["v"], s["g"], s["beta"], s["A_log"], s["dt_bias"], s["state"], s["cu"], **s["serving"])
    return parallel.context_parallel_prefill(s["q"], s["k"], s["v"], s["g"], s["beta"], s.get("A_log"), s.get("dt_bias"), s["scale"],
                                             s["state"], raw=bool(s["raw"]), backend=s["backend"])


def work(case):
    """q, k, v, the gate and beta read once, the output written once, each sequence's state read and written once, each
    checkpoint row written once; operations of the chunked form over 64-token chunks (per token and head: three
    products with the 128 x 128 state and the intra-chunk products)."""
    lens, H = _lengths(case), case["heads"]
    token = 3 * D * 2 + D * (2 if case["raw"] else 4) + (2 if case["raw"] else 4) + D * 2
    bytes_ = sum(lens) * H * token + len(lens) * H * 2 * D * D * 4
    if case["every"]:
        bytes_ += sum(-(-n // case["every"]) for n in lens) * H * D * D * (2 if case["rows"] == "bf16" else 4)
    return {"bytes": bytes_, "flops": sum(lens) * H * (6 * D * D + 4 * 64 * 2 * D)}


def tolerance(case):
    # bf16 inputs and outputs, products of bf16 / tf32 operands with fp32 accumulation (two such implementations, each
    # within about 4e-3 of the exact recurrence in the 2-norm)
    return {"rel": 1e-2}
