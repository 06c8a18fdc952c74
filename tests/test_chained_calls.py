"""Calls back to back on each other's outputs, as layers follow one another: a launch may be resident while the one
before it still writes what it will read, and the results are those of calls that wait for one another."""
import glob
import os
import re

import pytest
import torch

import gpu_mode_kernels_b200 as pkg
from gpu_mode_kernels_b200.all2all import A2AContext
from gpu_mode_kernels_b200.local_world import LocalWorld

DEV = "cuda:0"
CALLS = 50


def bits(t):
    return t.contiguous().view(torch.int16)


def test_no_kernel_of_the_path_reads_through_the_read_only_cache():
    """Loads that promise memory nobody writes during the kernel; an input may be the output of the launch before."""
    csrc = os.path.join(os.path.dirname(pkg.__file__), "csrc")
    files = glob.glob(os.path.join(csrc, "a2a*.cuh"))
    assert len(files) >= 5
    for path in files:
        with open(path) as f:
            assert not re.search(r"__ldg\s*\(|\.nc\.|__restrict__", f.read()), path


def rank_datas(E, K, H, T, ws):
    """Weights of a token add up to between 0.7 and 1 over the factors of the ranks: fifty calls stay in range, and every
    call changes every row."""
    rds = [pkg.generate_input(E, K, H, T, seed=51, rank=r, world_size=ws)[1].to(DEV) for r in range(ws)]
    for rd in rds:
        scale = 1.0 + (rd.indices // (E // ws)).float()
        share = torch.rand_like(rd.weights) + 0.1
        total = torch.linspace(0.7, 1.0, rd.num_tokens, device=DEV)[:, None]
        rd.weights = (share / share.sum(1, keepdim=True) * total / scale).contiguous()
    return rds


def chained(step, xs, wait):
    for i in range(CALLS):
        xs = step(xs)
        if wait:
            torch.cuda.synchronize()
        if i % 7 == 3:  # another program's kernel in between
            for x in xs:
                x.mul_(1.25)
            if wait:
                torch.cuda.synchronize()
    torch.cuda.synchronize()
    return [bits(x) for x in xs]


def same(step, rds):
    first = [rd.x.clone() for rd in rds]
    want = chained(step, [x.clone() for x in first], wait=True)
    assert all(w.bool().any() for w in want)
    for _ in range(3):
        got = chained(step, [x.clone() for x in first], wait=False)
        assert all(torch.equal(g, w) for g, w in zip(got, want))


@pytest.mark.gpu
@pytest.mark.parametrize("place", ["new outputs", "two buffers", "in place"])
@pytest.mark.parametrize("E,K,H,T,payload,schedule", [
    (64, 6, 2048, 1, "dedup", "pipelined"), (128, 4, 2880, 93, "dedup", "pipelined"), (256, 8, 7168, 256, "fp8", "pipelined"),
    (8, 2, 2048, 1300, "dedup", "pipelined"),  # routing and rows as two launches
    (16, 4, 1024, 70, "dedup", "phased"),      # one cooperative launch
])
def test_one_rank(E, K, H, T, payload, schedule, place):
    rd = rank_datas(E, K, H, T, 1)[0]
    ctx = A2AContext(pkg.MoEConfig(E, K, H, T), 0, 1, device=0, payload=payload, schedule=schedule,
                     combine="push" if schedule == "pipelined" else "pull")
    spare = [torch.empty_like(rd.x)]

    def step(xs):
        x = xs[0]
        if place == "new outputs":
            return [ctx.forward(x, rd.indices, rd.weights)]
        y = x
        if place == "two buffers":
            y, spare[0] = spare[0], x
        return [ctx.forward(x, rd.indices, rd.weights, y)]

    try:
        same(step, [rd])
        ctx.check()
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("schedule,payload,combine", [
    ("pipelined", "dedup", "push"), ("pipelined", "dedup", "pull"), ("pipelined", "fp8", "push"),
    ("phased", "direct", "pull"), ("phased", "dedup", "pull"), ("phased", "fp8", "pull"),
])
@pytest.mark.parametrize("E,K,H,T,ws", [(8, 2, 2048, 3, 2), (64, 6, 2048, 100, 4), (32, 8, 4096, 64, 8)])
def test_a_group(schedule, payload, combine, E, K, H, T, ws):
    rds = rank_datas(E, K, H, T, ws)
    world = LocalWorld(pkg.MoEConfig(E, K, H, T), ws, payload=payload, schedule=schedule, combine=combine)
    forward = world.forward_pipelined if schedule == "pipelined" else world.forward_phases

    def step(xs):
        for rd, x in zip(rds, xs):
            rd.x = x
        return forward(rds)

    try:
        same(step, rds)
        world.check()
    finally:
        world.close()
