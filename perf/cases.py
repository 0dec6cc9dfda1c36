"""The work that a user of fast_b200 on one B200 has it do, as measurable cases.

Four paths, each through its public entry points:

  moe       forward of one routed-expert layer (``MoELayer``): decode steps of a few tokens, prefills of thousands,
            bf16 or e4m3 dispatch, eager or as the captured CUDA graph
  train     one training step of the MoE block (``MixtralBlockModel`` forward and backward, ``FusedAdamW`` on every parameter)
  a2av      an all-to-all(v) of several ranks on one GPU (``LocalGroup``): tiny, large and skewed, two-tier, ragged element counts
  schedule  what a rank pays on the host for a traffic matrix that it has not seen before (``schedule``: plan, check, lower, upload)

The shapes are those of ``fast_b200.models.configs`` (the Mixtral-8x7B-shaped block; the DeepSeek-V3-like layer with
the 32 experts per GPU of ``fast_b200.bench.moe_fwd``) and a small generic one.
"""
from __future__ import annotations

import numpy as np
import torch

from fast_b200 import sched
from fast_b200.models import MixtralBlockModel, MoELayer
from fast_b200.parallel import Communicator, LocalGroup
from fast_b200.sched import PlanKind, Topology
from fast_b200.utils import FusedAdamW

# hidden, FFN width of an expert, experts on the GPU, experts per token
SHAPES = {
    "mixtral": (4096, 14336, 8, 2),
    "deepseek": (7168, 2048, 32, 8),
    "small": (1024, 3584, 8, 2),
}
VOCAB = 32000
SMS = 148
MAX_ITEMS = 32768   # more work items than one rank of any case here has


def _moe(name, shape, tokens, fp8=False, graph=False):
    return {"name": name, "path": "moe", "shape": shape, "tokens": tokens, "fp8": fp8, "graph": graph}


def _train(name, shape, tokens):
    return {"name": name, "path": "train", "shape": shape, "tokens": tokens}


def _a2av(name, servers, gpus, row_units, unit_bytes, skew, kind="staged"):
    return {"name": name, "path": "a2av", "servers": servers, "gpus": gpus, "row_units": row_units, "unit_bytes": unit_bytes, "skew": skew, "kind": kind}


def _schedule(name, servers, gpus, row_bytes, skew, kind="staged"):
    return {"name": name, "path": "schedule", "servers": servers, "gpus": gpus, "row_bytes": row_bytes, "skew": skew, "kind": kind}


def listed():
    return [
        # One user's chat: a decode step of a single token through the eager layer.
        _moe("decode_1", "mixtral", 1),
        # A serving batch of decode steps, replayed as the captured graph.
        _moe("decode_64_graph", "mixtral", 64, graph=True),
        # A decode batch of the layer with many small experts, e4m3 rows on the wire.
        _moe("decode_128_fp8", "deepseek", 128, fp8=True),
        # A prefill of an odd prompt length.
        _moe("prefill_2501", "mixtral", 2501),
        # The forward benchmark's prefill: 4096 tokens, skewed routing, e4m3 dispatch.
        _moe("prefill_4096_fp8", "deepseek", 4096, fp8=True),
        # Trying a recipe out on a small model: a step bound by launches and host work.
        _train("train_small_1022", "small", 1022),
        # Fine-tuning with one sequence per GPU and step.
        _train("train_4096", "mixtral", 4096),
        # The training benchmark's step: eight sequences of 4096 tokens.
        _train("train_32768", "mixtral", 32768),
        # Control messages: 1 KiB per rank, where only latency counts.
        _a2av("a2av_8x1KiB", 8, 1, 1024, 1, 0.0),
        # Skewed expert traffic: 256 MiB per rank, Zipf 1.0, the staged plan.
        _a2av("a2av_8x256MiB_zipf", 8, 1, 256 << 20, 1, 1.0),
        # Two servers of four GPUs; odd counts of 2-byte elements, so that segments start on any even address.
        _a2av("a2av_2x4_ragged", 2, 4, 8388607, 2, 0.5),
        # New routing in every step: the host's part of a collective whose matrix was never seen.
        _schedule("schedule_8", 8, 1, 256 << 20, 1.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    path = rng.choice(("moe", "moe", "train", "a2av", "schedule"))
    if path == "moe":
        graph = rng.random() < 0.3
        c = _moe("", rng.choice(sorted(SHAPES)), _log_int(rng, 2, 512 if graph else 8192), fp8=not graph and rng.random() < 0.4, graph=graph)
    elif path == "train":
        c = _train("", rng.choice(("mixtral", "small")), _log_int(rng, 64, 16384))
    else:
        servers, gpus = rng.choice(((2, 1), (3, 1), (4, 1), (6, 1), (8, 1), (2, 2), (2, 4), (4, 2)))
        skew, kind = rng.choice((0.0, 0.5, 1.0, 1.5)), rng.choice(("staged", "fanout"))
        if path == "a2av":
            unit = rng.choice((1, 2, 8))   # bytes in multiples of 16, bf16 elements and 8-byte words in any number
            c = _a2av("", servers, gpus, _log_int(rng, 1024, 128 << 20) // unit, unit, skew, kind)
        else:
            c = _schedule("", servers, gpus, _log_int(rng, 1 << 16, 1 << 30), skew, kind)
    del c["name"]
    return c


def _matrix(case, seed, row_units, quantum):
    n = case["servers"] * case["gpus"]
    return sched.workload_zipf_rows(n, case["skew"], row_units // quantum * quantum, seed, quantum)


def _prepare_moe(case, seed):
    H, I, E, K = SHAPES[case["shape"]]
    T = case["tokens"]
    rows = (T * min(K, E) + 256 * E + 255) // 256 * 256
    comm = Communicator(heap_bytes=rows * H * (4 if not case["fp8"] else 3) + rows * (H // 128) * 4 + (64 << 20))
    skewed = case["shape"] == "deepseek"   # a balance bias per expert, as that router has
    layer = MoELayer(comm, H, I, E, K, max_tokens=T, fp8_dispatch=case["fp8"], router_bias=skewed, training=False, graph_mode=case["graph"], seed=seed)
    layer.eval()
    g = torch.Generator(device="cuda").manual_seed(seed + 7)
    if skewed:
        layer.router_bias.data.copy_(torch.randn(E, generator=g, device="cuda") * 1.5)
    x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    if case["graph"]:
        layer.capture(T)
    return {"case": case, "layer": layer, "x": x}


def _prepare_train(case, seed):
    H, I, E, K = SHAPES[case["shape"]]
    T = case["tokens"]
    rows = T * min(K, E) + 256 * E + 256
    comm = Communicator(heap_bytes=4 * rows * H * 2 + (64 << 20))
    model = MixtralBlockModel(comm, vocab=VOCAB, hidden=H, inter=I, num_experts=E, top_k=K, max_tokens=T, seed=seed)
    experts = FusedAdamW(model.expert_parameters(), lr=1e-5, weight_decay=0.01)
    # The replicated parameters stand at the first step of their warm-up (rate 0): the update runs as always, and the
    # routing of a later pass on the same state does not hang on the last bit of an earlier pass' router gradient.
    replicated = FusedAdamW(model.replicated_parameters(), lr=0.0, weight_decay=0.0)
    g = torch.Generator(device="cuda").manual_seed(seed + 7)
    ids = torch.randint(0, VOCAB, (1, T), generator=g, device="cuda")
    names = {p: n for n, p in model.named_parameters()}
    return {"case": case, "model": model, "opts": (experts, replicated), "ids": ids, "names": names}


def _prepare_a2av(case, seed):
    topo = Topology(case["servers"], case["gpus"])
    ub = case["unit_bytes"]
    m = _matrix(case, 7, case["row_units"], 16 if ub == 1 else 1)   # the sizes belong to the case, the bytes come from the seed
    kind = PlanKind.STAGED if case["kind"] == "staged" else PlanKind.FANOUT
    plan = sched.build_plan(m, topo, kind=kind, split_align=max(1, 16 // ub))
    need = sum(int(b) * ub + 4096 for b in plan.buffers.max(axis=0)[1:])
    group = LocalGroup(topo.ranks, heap_bytes=need + (1 << 20), topo=topo, ctas=SMS // topo.ranks, threads=512)
    scheds = group.schedule(m, unit_bytes=ub, kind=kind)
    g = torch.Generator(device="cuda").manual_seed(seed + 7)
    ins = [torch.randint(0, 256, (max(s.input_bytes, 1),), generator=g, device="cuda", dtype=torch.uint8) for s in scheds]
    recv = [c.alloc(max(scheds[0].max_bytes["output"], 1), torch.uint8) for c in group.comms]
    return {"case": case, "group": group, "scheds": scheds, "ins": ins, "outs": [t[: s.output_bytes] for t, s in zip(recv, scheds)]}


def _prepare_schedule(case, seed):
    topo = Topology(case["servers"], case["gpus"])
    group = LocalGroup(topo.ranks, heap_bytes=1 << 20, topo=topo, ctas=SMS)
    return {"case": case, "group": group, "next": seed * 1000003, "items": np.zeros((MAX_ITEMS, 10), np.int64), "filled": 0}


def prepare(case, seed):
    return {"moe": _prepare_moe, "train": _prepare_train, "a2av": _prepare_a2av, "schedule": _prepare_schedule}[case["path"]](case, seed)


def _run_moe(s):
    with torch.no_grad():
        return s["layer"].forward_graphed(s["x"]) if s["case"]["graph"] else s["layer"](s["x"])


def _run_train(s):
    model = s["model"]
    for o in s["opts"]:
        o.zero_grad()
    loss = model(s["ids"])
    loss.backward()
    for o in s["opts"]:
        o.step()
    out = {"loss": loss.detach()}
    for o in s["opts"]:
        for p in o.params:
            out[s["names"][p]] = (p.detach(), p.grad, *o.state[p])   # parameter, gradient, master copy, first and second moment
    return out


def _run_a2av(s):
    s["group"].all_to_all_v(s["outs"], s["ins"], s["scheds"])
    return s["outs"]


def _run_schedule(s):
    # One rank of the job plans the matrix of its next step.
    c = s["case"]
    s["next"] += 1
    # A new step's tokens: other destinations, and up to a quarter fewer of them.
    m = _matrix(c, s["next"], c["row_bytes"] - 16 * (s["next"] * 7919 % (c["row_bytes"] // 64)), 16)
    got = s["group"].comms[0].schedule(m, unit_bytes=1, kind=PlanKind.STAGED if c["kind"] == "staged" else PlanKind.FANOUT)
    items, k = got.lowered["items"], len(got.lowered["items"])   # a list of any length, followed by zeros
    s["items"][:k] = items
    s["items"][k: s["filled"]] = 0
    s["filled"] = k
    return {"items": s["items"], "count": k, "output": got.output_bytes, "max": got.max_bytes}


def run(state):
    return {"moe": _run_moe, "train": _run_train, "a2av": _run_a2av, "schedule": _run_schedule}[state["case"]["path"]](state)


def work(case):
    if case["path"] in ("moe", "train"):
        H, I, E, K = SHAPES[case["shape"]]
        T = case["tokens"]
        touched = E * (1.0 - (1.0 - K / E) ** T)          # experts that get a token, for even routing
        if case["path"] == "moe":
            return {"bytes": 2.0 * touched * 3 * H * I + 2.0 * E * H + 2.0 * 2 * T * H, "flops": 6.0 * T * K * H * I + 2.0 * T * H * E}
        params = 3.0 * E * H * I + VOCAB * H + E * H + H
        # bf16 parameters and three fp32 states read and written, gradients written, ids read
        return {"bytes": 30.0 * params + 8.0 * T, "flops": 18.0 * T * K * H * I + 6.0 * T * H * E}
    n = case["servers"] * case["gpus"]
    if case["path"] == "a2av":
        return {"bytes": 2.0 * n * case["row_units"] * case["unit_bytes"], "flops": 0.0}
    # the matrix in, one rank's work list out (a chunk of up to 1 MiB is one item of ten words)
    return {"bytes": 8.0 * n * n + 80.0 * max(n - 1, case["row_bytes"] / (1 << 18)), "flops": 0.0}


def tolerance(case):
    if case["path"] in ("a2av", "schedule"):
        return "exact"                                     # bytes and whole numbers
    if case["path"] == "moe":
        return {"rel": 1e-2, "max": 0.3}                   # bf16 activations, rounded between the two projections
    return {"rel": 1e-2, "max": 0.3}                       # bf16 gradients of bf16 activations; squared in the second moment
