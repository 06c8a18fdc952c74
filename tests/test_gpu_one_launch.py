"""The kernel that a group with a GPU per rank runs -- senders in their form for distant peers, watchers, flags and
fences at system scope, all roles at the same time -- held to the oracle on one GPU: every rank's blocks in one
cooperative launch, and the same roles rank by rank.  ``LocalWorld``'s steps, which the other tests call, run
variants for peers on the same GPU."""
import pytest
import torch

import gpu_mode_kernels_b200 as pkg
from gpu_mode_kernels_b200 import _lib
from gpu_mode_kernels_b200.all2all import A2AError
from gpu_mode_kernels_b200.local_world import LocalWorld
from oracle import a2a_oracle as O
from parity import check_y, tol
from test_gpu_group import rank_by_rank
from test_gpu_pipelined import check_pipelined_dispatch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
HOW = {"one_launch": LocalWorld.forward_one_launch, "rank_by_rank": rank_by_rank}


def bits(t):
    return t.contiguous().view(torch.int16)


def run_case(cfg, ws, rds_cpu, how, payload, combine, calls=1):
    """`calls` calls against the oracle; the outputs bit for bit those of the roles in lock-step."""
    disp, ys = O.simulate(cfg, ws, rds_cpu)
    rds = [rd.to(DEV) for rd in rds_cpu]
    world = LocalWorld(cfg, ws, payload=payload, schedule="pipelined", combine=combine)
    try:
        for _ in range(calls):
            before = [c.launches for c in world.ctxs]
            out = HOW[how](world, rds)
            torch.cuda.synchronize()
            world.check()
            assert all(c.launches - b == (1 if how == "one_launch" else 3) for c, b in zip(world.ctxs, before))
            check_pipelined_dispatch(world, disp, cfg.in_dtype, payload)
            check_y(cfg, ws, rds_cpu, out, ys, payload, [r for r in range(ws) if rds_cpu[r].num_tokens])
        ref = world.forward_pipelined(rds)
        assert all(torch.equal(bits(a), bits(b)) for a, b in zip(out, ref))
        world.check()
        return out
    finally:
        torch.cuda.synchronize()
        world.close()


@pytest.mark.parametrize("how", list(HOW))
@pytest.mark.parametrize("combine", ["push", "pull"])
def test_golden_cases(golden, combine, how):
    if golden.ws == 1:
        pytest.skip("one rank has a kernel of its own")
    rds = [golden.rank_data(r) for r in range(golden.ws)]
    out = run_case(golden.cfg, golden.ws, rds, how, "dedup", combine)
    for r in range(golden.ws):
        torch.testing.assert_close(out[r].cpu().float(), golden.expected_y(r).float(), **tol(golden.cfg.in_dtype))


@pytest.mark.parametrize("how", list(HOW))
@pytest.mark.parametrize("name,ws,payload,combine", [
    ("c2", 8, "dedup", "push"), ("c3", 8, "dedup", "push"), ("c4", 8, "dedup", "push"), ("c4", 8, "dedup", "pull"),
    ("c4", 2, "dedup", "push"), ("c5", 8, "fp8", "push"), ("c5", 4, "fp8", "pull"),
])
def test_benchmark_workloads_full_size(name, ws, payload, combine, how):
    datas = [pkg.workload_input(name, r, ws) for r in range(ws)]
    run_case(datas[0][0], ws, [d[1] for d in datas], how, payload, combine)


@pytest.mark.parametrize("payload", ["dedup", "fp8"])
@pytest.mark.parametrize("combine", ["push", "pull"])
@pytest.mark.parametrize("E,K,H,T,ws,dtype", [
    (8, 1, 128, 1, 8, torch.bfloat16),       # one token, one expert per rank
    (12, 3, 2944, 70, 3, torch.float16),     # ranks that do not divide the grid, rows that end inside a piece
    (16, 4, 9216, 70, 2, torch.bfloat16),    # a row larger than one stage of the senders' ring
    (32, 4, 256, 700, 4, torch.bfloat16),    # several rounds of 256 tokens
])
def test_edge_shapes(E, K, H, T, ws, dtype, combine, payload):
    datas = [pkg.generate_input(E, K, H, T, seed=5, rank=r, world_size=ws, dtype=dtype, ragged=T > 2) for r in range(ws)]
    rds = [d[1] for d in datas]
    if ws == 3:  # a rank without tokens still serves the others
        rds[1].num_tokens = 0
        rds[1].x, rds[1].indices, rds[1].weights = rds[1].x[:0], rds[1].indices[:0], rds[1].weights[:0]
    run_case(datas[0][0], ws, rds, "one_launch", payload, combine, calls=2)


@pytest.mark.parametrize("payload", ["dedup", "fp8"])
@pytest.mark.parametrize("combine", ["push", "pull"])
def test_repeated_calls_without_host_sync(combine, payload):
    """Back-to-back calls on alternating inputs, one launch and steps mixed: nothing of an earlier call is taken
    for this one's."""
    ws, cfg = 4, pkg.MoEConfig(32, 4, 512, 64)
    sets = []
    for seed in (1, 2):
        datas = [pkg.generate_input(32, 4, 512, 64, seed=seed, rank=r, world_size=ws, ragged=True) for r in range(ws)]
        sets.append([d[1].to(DEV) for d in datas])
    world = LocalWorld(cfg, ws, payload=payload, schedule="pipelined", combine=combine)
    try:
        want = [[bits(y) for y in world.forward_pipelined(rds)] for rds in sets]
        outs = []
        for i in range(40):
            call = world.forward_pipelined if i % 5 == 4 else world.forward_one_launch
            outs.append(call(sets[i % 2]))
        torch.cuda.synchronize()
        world.check()
        for i, out in enumerate(outs):
            assert all(torch.equal(bits(a), b) for a, b in zip(out, want[i % 2])), i
    finally:
        torch.cuda.synchronize()
        world.close()


def test_what_is_no_group_call_is_refused():
    rds = [pkg.generate_input(8, 2, 64, 4, seed=1, rank=r, world_size=2)[1].to(DEV) for r in range(2)]
    cfg = pkg.MoEConfig(8, 2, 64, 4)
    for ws, schedule, payload, code in ((2, "phased", "dedup", _lib.A2A_ERR_STATE), (1, "pipelined", "dedup", _lib.A2A_ERR_CONFIG)):
        world = LocalWorld(cfg, ws, payload=payload, schedule=schedule, combine="pull")
        try:
            with pytest.raises(A2AError) as refused:
                world.forward_one_launch(rds[:ws])
            assert refused.value.code == code and all(c.launches == 0 for c in world.ctxs)
        finally:
            world.close()
