"""The calls that a program using this framework makes, over the sizes it makes them at.

Five kinds of case, all through the public entry points:

``call``       ``all2all.custom_kernel`` on device tensors: one rank's whole step (dispatch, expert
               placeholder, combine) on a GPU of its own, as a serving loop calls it once a layer.
``host``       the same call on pinned host tensors: copies in, step, copy out.
``ranks``      ``local_world.LocalWorld.forward_pipelined``: the roles of the one-launch kernel for
               every rank of a group, stepped on one GPU -- the senders, routers, expert blocks and
               combine that a group of GPUs runs.
``phases``     ``LocalWorld.forward_phases``: routing, sending, receiving, the expert op and the
               combine as calls of their own, which is how a program with its own expert kernels
               drives the path.
``histogram``  ``histogram.custom_kernel``: counts of the byte values of a buffer.

Problem sizes are the configurations of ``task.py`` and of the histogram's task, and generic ones
between and around them: expert layouts (experts, top-k, hidden size) as they occur there, one token
to a prefill batch of 2048, ragged token counts, buffers from a few kilobytes to half a gigabyte.
"""
import math
from types import SimpleNamespace

import torch

from gpu_mode_kernels_b200.all2all import custom_kernel
from gpu_mode_kernels_b200.histogram import custom_kernel as histogram_kernel
from gpu_mode_kernels_b200.local_world import LocalWorld
from gpu_mode_kernels_b200.task import MoEConfig

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}

# (experts, top-k, hidden) as they occur together in the task's shapes and the benchmark workloads
LAYOUTS = [(8, 2, 6144), (8, 2, 2048), (64, 6, 2048), (128, 4, 2880), (128, 8, 4096), (256, 8, 7168)]


def _moe(name, kind, layout, max_tokens, tokens, dtype="bf16", world=1, payload="dedup", combine="push",
         routing="uniform", weights="softmax"):
    experts, topk, hidden = layout
    case = dict(kind=kind, experts=experts, topk=topk, hidden=hidden, max_tokens=max_tokens, tokens=tokens,
                dtype=dtype, world=world, payload=payload, combine=combine, routing=routing, weights=weights)
    return dict(case, name=name) if name else case


def _bytes(name, size, contention, offset=0):
    case = dict(kind="histogram", size=size, contention=contention, offset=offset)
    return dict(case, name=name) if name else case


def listed():
    return [
        # one token being decoded, in the task's own number format: nothing but latency
        _moe("decode_one_token", "call", (64, 6, 2048), 4, 1, dtype="fp16", weights="rand"),
        # a decode batch that does not fill its buffers, rows that are no multiple of 2 KB
        _moe("decode_batch_ragged", "call", (128, 4, 2880), 128, 93, dtype="fp16", weights="rand"),
        # the workload the framework's headline figure is quoted on, one GPU's share of tokens
        _moe("headline", "call", (256, 8, 7168), 256, 256),
        # a prefill batch of the same model
        _moe("prefill", "call", (256, 8, 7168), 2048, 2048),
        # a caller whose activations live in pinned host memory
        _moe("headline_from_host", "host", (256, 8, 7168), 256, 256),
        # the headline workload over eight ranks
        _moe("ranks8_headline", "ranks", (256, 8, 7168), 256, 256, world=8),
        # skewed expert popularity over eight ranks: some ranks get several times the rows of others
        _moe("ranks8_skewed", "ranks", (64, 6, 2048), 256, 256, world=8, routing="zipf"),
        # the headline workload with rows quantised to eight bits on the wire
        _moe("ranks8_fp8", "ranks", (256, 8, 7168), 256, 256, world=8, payload="fp8"),
        # a program with its own expert kernels: one call per phase, a row per pair sent into its slab
        _moe("phases4", "phases", (128, 8, 4096), 128, 117, dtype="fp16", world=4, payload="direct", combine="pull",
             weights="rand"),
        # the histogram task's small, contended case; its largest benchmark; a large ragged buffer
        _bytes("histogram_30k", 30080, 90),
        _bytes("histogram_10m", 10485760, 10),
        _bytes("histogram_512m", 536870917, 40),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["call", "call", "call", "host", "ranks", "ranks", "phases", "histogram", "histogram"])
    if kind == "histogram":
        return _bytes(None, _log_int(rng, 5120, 536870912), rng.choice([0, 10, 40, 90, rng.randint(0, 95)]),
                      rng.choice([0, 0, rng.randint(1, 15)]))
    experts, topk, hidden = rng.choice(LAYOUTS)
    if rng.random() < 0.3:
        hidden = 8 * rng.randint(64, hidden // 8)
    world = rng.choice([2, 4, 8]) if kind in ("ranks", "phases") else 1
    max_tokens = _log_int(rng, 1, {"call": 2048, "host": 512}.get(kind, 256))
    tokens = rng.choice([max_tokens, rng.randint((max_tokens + 1) // 2, max_tokens)])
    # eight-bit wire rows need a hidden size that is a multiple of their scale block
    fp8 = hidden % 128 == 0 and rng.random() < 0.25
    payload = "fp8" if fp8 else (rng.choice(["direct", "dedup"]) if kind == "phases" else "dedup")
    combine = "pull" if kind == "phases" or rng.random() < 0.2 else "push"
    task_style = rng.random() < 0.4
    return _moe(None, kind, (experts, topk, hidden), max_tokens, tokens, dtype="fp16" if task_style else "bf16",
                world=world, payload=payload, combine=combine,
                routing="zipf" if experts >= 64 and rng.random() < 0.25 else "uniform",
                weights="rand" if task_style else "softmax")


def _rank_data(case, gen):
    n, e, k = case["tokens"], case["experts"], case["topk"]
    dev = gen.device
    # k distinct experts per token: the k largest of independent keys (Gumbel keys where popularity is skewed)
    keys = torch.rand(n, e, generator=gen, device=dev)
    if case["routing"] == "zipf":
        popularity = -1.2 * torch.log(torch.arange(1, e + 1, device=dev, dtype=torch.float32))
        keys = popularity - torch.log(-torch.log(keys.clamp(1e-7, 1 - 1e-6)))
    indices = keys.topk(k, dim=1).indices.to(torch.int32)
    if case["weights"] == "softmax":
        w = torch.softmax(torch.randn(n, k, generator=gen, device=dev), dim=-1)
    else:
        w = torch.rand(n, k, generator=gen, device=dev)
    x = torch.randn(n, case["hidden"], generator=gen, device=dev).to(DTYPES[case["dtype"]])
    return SimpleNamespace(num_tokens=n, x=x, indices=indices.contiguous(), weights=w.contiguous())


# A program sets its group up once and keeps it; the group of the last shape asked for is kept here.
_world = {}


def _world_for(case, cfg):
    schedule = "phased" if case["kind"] == "phases" else "pipelined"
    key = (cfg.num_experts, cfg.experts_per_token, cfg.hidden_dim, cfg.max_num_tokens, cfg.in_dtype,
           case["world"], case["payload"], schedule, case["combine"])
    if key not in _world:
        for old in _world.values():
            old.close()
        _world.clear()
        _world[key] = LocalWorld(cfg, case["world"], payload=case["payload"], schedule=schedule,
                                 combine=case["combine"])
    return _world[key]


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind == "histogram":
        data = torch.randint(0, 256, (case["size"] + case["offset"],), dtype=torch.uint8, generator=gen, device="cuda")
        often = int(torch.randint(0, 256, (1,), generator=gen, device="cuda"))
        for lo in range(0, data.numel(), 1 << 26):  # a slice at a time: the random keys are four times the data
            part = data[lo:lo + (1 << 26)]
            part[torch.rand(part.numel(), generator=gen, device="cuda") < case["contention"] / 100] = often
        return kind, (data[case["offset"]:], torch.empty(256, dtype=torch.int64, device="cuda"))
    dtype = DTYPES[case["dtype"]]
    cfg = MoEConfig(case["experts"], case["topk"], case["hidden"], case["max_tokens"], dtype, dtype)
    data = [_rank_data(case, gen) for _ in range(case["world"])]
    if kind in ("ranks", "phases"):
        return kind, (_world_for(case, cfg), data)
    rank_data = data[0]
    if kind == "host":
        for name in ("x", "indices", "weights"):
            setattr(rank_data, name, getattr(rank_data, name).cpu().pin_memory())
    return kind, ((cfg, rank_data, 0, 1), case["payload"], case["combine"])


def run(state):
    kind, what = state
    if kind == "histogram":
        return histogram_kernel(what)
    if kind == "ranks":
        world, data = what
        return world.forward_pipelined(data)
    if kind == "phases":
        world, data = what
        return world.forward_phases(data)
    data, payload, combine = what
    return custom_kernel(data, payload=payload, combine=combine)


def work(case):
    if case["kind"] == "histogram":
        return {"bytes": case["size"] + 256 * 8, "flops": 0}
    n, k, h = case["tokens"] * case["world"], case["topk"], case["hidden"]
    # token rows in, one row per (token, expert) written into the experts' buffers, output rows out, and the
    # top-k indices and weights; a multiply per dispatched element, a multiply-add for its share of the output
    return {"bytes": n * (2 + k) * h * 2 + n * k * 8, "flops": 3 * n * k * h}


def tolerance(case):
    if case["kind"] == "histogram":
        return "exact"
    # Roundings of the output to its element type, one, and with the reduction at the expert ranks one more per
    # contributing rank; four times what the path differs by from the same sums in 64 bits (2-norm 1.7e-3 to
    # 2.2e-3 in bf16, 2.1e-4 to 2.9e-4 in fp16; largest single difference 7.3e-3 in bf16, 9.4e-4 in fp16).
    bf16 = case["dtype"] == "bf16"
    return {"rel": 8e-3, "max": 3e-2} if bf16 else {"rel": 1.2e-3, "max": 4e-3}
