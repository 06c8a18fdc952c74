"""One launch per phase for a whole group on one GPU: the same bits as the phases called rank by rank, and
nothing begun when one rank's arguments are refused."""
import ctypes as C

import pytest
import torch

import gpu_mode_kernels_b200 as pkg
from gpu_mode_kernels_b200 import _lib
from gpu_mode_kernels_b200.all2all import A2AError
from gpu_mode_kernels_b200.local_world import LocalWorld

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def bits(t):
    return t.contiguous().view(torch.int16)


def rank_by_rank(world, rds):
    if world.ctxs[0].schedule == "pipelined":
        for c, rd in zip(world.ctxs, rds):
            c.pipe_step(0, rd.x, rd.indices, rd.weights)
        for c in world.ctxs:
            c.pipe_step(1)
        return [c.pipe_step(2) for c in world.ctxs]
    for c, rd in zip(world.ctxs, rds):
        c.route(rd.indices)
    for c, rd in zip(world.ctxs, rds):
        c.dispatch_send(rd.x)
    for c in world.ctxs:
        c.dispatch_recv()
    for c in world.ctxs:
        c.expert_placeholder()
    return [c.combine(rd.weights) for c, rd in zip(world.ctxs, rds)]


def state(world):
    return [t for c in world.ctxs for t in c.route_tables() + c.export_dispatch()]


@pytest.mark.parametrize("schedule,payload,combine", [
    ("pipelined", "dedup", "push"), ("pipelined", "dedup", "pull"), ("pipelined", "fp8", "push"),
    ("phased", "direct", "pull"), ("phased", "dedup", "pull"), ("phased", "fp8", "pull"),
])
@pytest.mark.parametrize("E,K,H,T,ws", [
    (8, 2, 128, 1, 2),       # one token: fewer wire rows than sender blocks
    (12, 3, 2944, 70, 3),    # ranks that do not divide the grid, rows that end inside a warp's piece
    (64, 6, 2048, 300, 8),   # more than one round of 256 tokens
])
def test_group_launches_equal_the_phases_rank_by_rank(schedule, payload, combine, E, K, H, T, ws):
    sets = [[pkg.generate_input(E, K, H, T, seed=s, rank=r, world_size=ws, ragged=T > 1) for r in range(ws)] for s in (3, 4)]
    world = LocalWorld(sets[0][0][0], ws, payload=payload, schedule=schedule, combine=combine)
    grouped = world.forward_pipelined if schedule == "pipelined" else world.forward_phases
    try:
        for datas in sets:  # ranks of different token counts, then others on the same contexts
            rds = [d[1].to(DEV) for d in datas]
            want = [bits(y) for y in rank_by_rank(world, rds)]
            tables = state(world)
            before = [c.launches for c in world.ctxs]
            got = grouped(rds)
            assert all(c.launches - b == (3 if schedule == "pipelined" else 4) for c, b in zip(world.ctxs, before))
            assert all(torch.equal(bits(g), w) for g, w in zip(got, want))
            assert all(torch.equal(a, b) for a, b in zip(state(world), tables))
        world.ctxs[1].trace_enable()  # traced contexts are launched one by one
        got = grouped(rds)
        assert all(torch.equal(bits(g), w) for g, w in zip(got, want))
        assert bool((world.ctxs[1].trace_read()[:2, 1] != 0).all())  # blocks that every phase's launch has
        world.check()
    finally:
        world.close()


def test_nothing_begins_when_one_rank_is_refused():
    cfg = pkg.MoEConfig(8, 2, 64, 4)
    datas = [pkg.generate_input(8, 2, 64, 4, seed=1, rank=r, world_size=2) for r in range(2)]
    rds = [d[1].to(DEV) for d in datas]
    world = LocalWorld(cfg, 2, payload="dedup", schedule="pipelined", combine="push")
    try:
        want = [bits(y) for y in world.forward_pipelined(rds)]
        bad = [rds[0], rds[1].to(DEV)]
        bad[1].weights = bad[1].weights.double()
        with pytest.raises(A2AError):
            world.forward_pipelined(bad)
        lib, before = world.ctxs[0].lib, [c.launches for c in world.ctxs]
        handles = (C.c_void_p * 2)(*[c._h for c in world.ctxs])
        calls = (_lib.Call * 2)()
        for call, rd in zip(calls, rds):
            call.x, call.topk_idx, call.topk_weights = rd.x.data_ptr(), rd.indices.data_ptr(), rd.weights.data_ptr()
            call.y, call.num_tokens = rd.x.data_ptr(), 4
        calls[1].num_tokens = 5  # more than the contexts were made for
        assert lib.a2a_group_step(handles, _lib.GROUP_PHASE["pipe_send"], calls, None) == _lib.A2A_ERR_CONFIG
        assert lib.a2a_group_step(handles, _lib.GROUP_PHASE["pipe_send"], None, None) == _lib.A2A_ERR_CONFIG
        assert lib.a2a_group_step((C.c_void_p * 2)(handles[1], handles[0]), 0, calls, None) == _lib.A2A_ERR_CONFIG
        assert lib.a2a_group_step(handles, 8, calls, None) == _lib.A2A_ERR_CONFIG
        assert [c.launches for c in world.ctxs] == before
        got = world.forward_pipelined(rds)  # the ranks' call counters are still level
        assert all(torch.equal(bits(g), w) for g, w in zip(got, want))
        world.check()
    finally:
        world.close()


@pytest.mark.parametrize("schedule,payload,combine", [("pipelined", "dedup", "push"), ("phased", "direct", "pull")])
def test_contexts_that_are_no_group_are_refused(schedule, payload, combine):
    """Contexts of two equal groups mixed, and ranks that are not at the same call."""
    cfg = pkg.MoEConfig(8, 2, 64, 4)
    rds = [pkg.generate_input(8, 2, 64, 4, seed=2, rank=r, world_size=2)[1].to(DEV) for r in range(2)]
    worlds = [LocalWorld(cfg, 2, payload=payload, schedule=schedule, combine=combine) for _ in range(2)]

    def forward(world):
        return [bits(y) for y in (world.forward_pipelined if schedule == "pipelined" else world.forward_phases)(rds)]

    def launches():
        return [c.launches for w in worlds for c in w.ctxs]

    try:
        want = forward(worlds[0])
        assert all(torch.equal(a, b) for a, b in zip(forward(worlds[1]), want))
        mixed = object.__new__(LocalWorld)
        mixed.cfg, mixed.world_size, mixed.ctxs = cfg, 2, [worlds[0].ctxs[0], worlds[1].ctxs[1]]
        before = launches()
        with pytest.raises(A2AError) as refused:
            forward(mixed)
        assert refused.value.code == _lib.A2A_ERR_CONFIG and launches() == before
        for c in worlds[0].ctxs:  # one rank begins a call by itself, then the other
            c.route(rds[0].indices)
            if c.rank == 0:
                before = launches()
                with pytest.raises(A2AError) as refused:
                    forward(worlds[0])
                assert refused.value.code == _lib.A2A_ERR_STATE and launches() == before
        for w in worlds:
            assert all(torch.equal(a, b) for a, b in zip(forward(w), want))
            w.check()
    finally:
        for w in worlds:
            w.close()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("schedule,payload,combine", [("pipelined", "dedup", "push"), ("phased", "direct", "pull")])
def test_expert_op_on_every_bit_pattern(dtype, schedule, payload, combine):
    """Subnormals, overflow, infinities and signed zeros included: dtype(float(x) * (1 + rank)) to the bit on all
    eight ranks (a NaN stays one, whatever its payload)."""
    ws, T, H = 8, 64, 1024
    x = torch.arange(1 << 16, dtype=torch.int32).to(torch.int16).view(dtype).view(T, H)
    idx = torch.arange(ws, dtype=torch.int32).expand(T, ws).contiguous()  # every token to every rank's one expert
    w = torch.ones(T, ws)
    world = LocalWorld(pkg.MoEConfig(ws, ws, H, T, dtype, dtype), ws, payload=payload, schedule=schedule, combine=combine)
    try:
        rds = []
        for _ in range(ws):
            rd = object.__new__(pkg.RankTestData)
            rd.num_tokens, rd.x, rd.indices, rd.weights = T, x.to(DEV), idx.to(DEV), w.to(DEV)
            rds.append(rd)
        (world.forward_pipelined if schedule == "pipelined" else world.forward_phases)(rds)
        for r, c in enumerate(world.ctxs):
            _, rows, _ = c.export_dispatch()
            want = (x.float() * (1.0 + r)).to(dtype)
            for s in range(ws):  # the rows of source s, tokens in order
                got = rows[0, s * T:(s + 1) * T].cpu()
                assert torch.equal(got.isnan(), want.isnan())
                assert torch.equal(bits(got)[~got.isnan()], bits(want)[~want.isnan()])
        world.check()
    finally:
        world.close()


@pytest.mark.parametrize("payload,combine", [("dedup", "push"), ("dedup", "pull"), ("fp8", "push")])
@pytest.mark.parametrize("together", [(True, False, False), (True, True, False), (True, False, True),
                                      (False, True, True), (False, True, False), (False, False, True)])
def test_a_call_goes_on_in_the_form_it_was_begun_in(payload, combine, together):
    """Roles for the whole group and roles rank by rank, mixed inside one call: the same bits."""
    ws, T, H = 3, 40, 2944
    rds = [pkg.generate_input(12, 3, H, T, seed=5, rank=r, world_size=ws, ragged=True)[1].to(DEV) for r in range(ws)]
    world = LocalWorld(pkg.MoEConfig(12, 3, H, T), ws, payload=payload, schedule="pipelined", combine=combine)
    try:
        want = [bits(y) for y in rank_by_rank(world, rds)]
        tables = state(world)
        for _ in range(2):
            if together[0]:
                calls, ys = world._whole_calls(rds)
                world._step("pipe_send", calls)
                world._begun(rds, ys)
            else:
                for c, rd in zip(world.ctxs, rds):
                    c.pipe_step(0, rd.x, rd.indices, rd.weights)
                ys = [c._y for c in world.ctxs]
            for role, phase in ((1, "pipe_expert"), (2, "pipe_combine")):
                if together[role]:
                    world._step(phase)
                else:
                    for c in world.ctxs:
                        c.pipe_step(role)
            assert all(torch.equal(bits(y), w) for y, w in zip(ys, want))
            assert all(torch.equal(a, b) for a, b in zip(state(world), tables))
        world.check()
    finally:
        world.close()


@pytest.mark.parametrize("T", [8, 130])  # 1 MB of expert rows, and 18
def test_a_rank_without_rows_need_not_run_its_expert_phase(T):
    """Phases called rank by rank by a program that steps only the ranks with rows; the combine for all ranks together."""
    ws, E, K, H = 4, 16, 4, 4096
    rds = [pkg.generate_input(E, K, H, T, seed=6, rank=r, world_size=ws)[1].to(DEV) for r in range(ws)]
    for rd in rds:  # no expert of the last rank
        rd.indices = torch.rand(T, E - E // ws, device=DEV).topk(K, dim=1).indices.int()
    world = LocalWorld(pkg.MoEConfig(E, K, H, T), ws, payload="direct", timeout_ms=300)
    try:
        want = [bits(y) for y in world.forward_phases(rds)]
        for run in (ws - 1, 0):
            world._send(rds)
            for c in world.ctxs[:run]:
                c.dispatch_recv()
                c.expert_placeholder()
            ys = world._combine(rds)
            torch.cuda.synchronize()
            if run:
                assert all(torch.equal(bits(y), w) for y, w in zip(ys, want))
                world.check()
        for c in world.ctxs:  # nobody's expert phase ran: every rank ran out of its budget, once
            assert c.peek() == _lib.A2A_ERR_TIMEOUT
            c.clear_status()
        assert all(torch.equal(bits(y), w) for y, w in zip(world.forward_phases(rds), want))
        world.check()
    finally:
        world.close()


@pytest.mark.parametrize("payload,combine", [("dedup", "push"), ("dedup", "pull"), ("fp8", "push")])
def test_a_call_begun_rank_by_rank_goes_on_in_one_launch_a_role(payload, combine):
    from cuda.bindings import runtime

    ws, T, H = 3, 40, 2944
    rds = [pkg.generate_input(12, 3, H, T, seed=7, rank=r, world_size=ws, ragged=True)[1].to(DEV) for r in range(ws)]
    world = LocalWorld(pkg.MoEConfig(12, 3, H, T), ws, payload=payload, schedule="pipelined", combine=combine)
    try:
        want = [bits(y) for y in rank_by_rank(world, rds)]
        for c, rd in zip(world.ctxs, rds):
            c.pipe_step(0, rd.x, rd.indices, rd.weights)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph):
            world._step("pipe_expert")
            world._step("pipe_combine")
        status, _, nodes = runtime.cudaGraphGetNodes(runtime.cudaGraph_t(graph.raw_cuda_graph()), 0)
        assert int(status) == 0 and nodes == 2
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(bits(c._y), w) for c, w in zip(world.ctxs, want))
        world.check()
    finally:
        world.close()


@pytest.mark.parametrize("payload,combine", [("dedup", "push"), ("dedup", "pull"), ("fp8", "push"), ("fp8", "pull")])
@pytest.mark.parametrize("E,K,H,T,ws", [
    (12, 3, 640, 33, 3),     # one token more than a routing block takes, rows that end inside a warp's piece
    (16, 7, 6144, 200, 8),   # the wide form of role 1, for many stores a load
    (8, 2, 2816, 400, 4),    # and for few
    (8, 2, 128, 1100, 2),    # routing blocks of 64 tokens
    (8, 2, 128, 8200, 2),    # of 256
])
def test_a_whole_call_equals_its_roles(payload, combine, E, K, H, T, ws):
    """Outputs from the expert pass, against the forms of distant ranks, to the bit: in one call, role by role, and with
    outputs over inputs (of the same rank, of another, and across two), where partial rows are added up."""
    rds = [pkg.generate_input(E, K, H, T, seed=8, rank=r, world_size=ws)[1].to(DEV) for r in range(ws)]
    for name in ("x", "indices", "weights"):  # a rank without tokens, one with few
        setattr(rds[1], name, getattr(rds[1], name)[:0].contiguous())
        setattr(rds[-1], name, getattr(rds[-1], name)[:1 if ws > 2 else 0].contiguous())
    rds[0].indices[0, :] = rds[0].indices[0, 0]  # repeats, and a token without a valid expert: dropped, zero
    rds[0].indices[T - 1, :] = E
    for rd in rds:
        rd.num_tokens = rd.x.shape[0]
    world = LocalWorld(pkg.MoEConfig(E, K, H, T), ws, payload=payload, schedule="pipelined", combine=combine)
    phases = (C.c_int32 * 3)(*[_lib.GROUP_PHASE[name] for name in ("pipe_send", "pipe_expert", "pipe_combine")])
    handles = (C.c_void_p * ws)(*[c._h.value for c in world.ctxs])

    def clear():
        for c in world.ctxs:
            assert c.peek() in (0, _lib.A2A_ERR_ROUTING)
            c.clear_status()

    def steps(xs, ys, whole):
        calls, done = (_lib.Call * ws)(), C.c_int32()
        for call, rd, x, y in zip(calls, rds, xs, ys):
            call.x, call.topk_idx, call.topk_weights = x.data_ptr(), rd.indices.data_ptr(), rd.weights.data_ptr()
            call.y, call.num_tokens = y.data_ptr(), x.shape[0]
        if whole:
            _lib.check(world.ctxs[0].lib.a2a_group_steps(handles, phases, 3, calls, _lib.current_stream(), C.byref(done)))
            assert done.value == 3
        else:
            for name in ("pipe_send", "pipe_expert", "pipe_combine"):
                world._step(name, calls)
        torch.cuda.synchronize()
        clear()
        for c, x in zip(world.ctxs, xs):
            c._num_tokens = x.shape[0]
        return [bits(y) for y in ys]

    try:
        want = [bits(y) for y in rank_by_rank(world, rds)]
        clear()
        tables = state(world)
        for whole in (True, False):
            got = steps([rd.x for rd in rds], [torch.full_like(rd.x, 3) for rd in rds], whole)
            assert all(torch.equal(a, b) for a, b in zip(got, want))
            assert all(torch.equal(a, b) for a, b in zip(state(world), tables))
            xs = [rd.x.clone() for rd in rds]
            assert all(torch.equal(a, b) for a, b in zip(steps(xs, xs, whole), want))
            xs = [rd.x.clone() for rd in rds]
            ys = [torch.empty_like(x) for x in xs]
            ys[-1] = xs[0][:xs[-1].shape[0]]  # over rows of another rank
            assert all(torch.equal(a, b) for a, b in zip(steps(xs, ys, whole), want))
            room, xs, ys, at = torch.empty(sum(rd.x.numel() for rd in rds) + 8 * H, dtype=rds[0].x.dtype, device=DEV), [], [], 0
            for rd in rds:  # outputs that begin three rows into the inputs: over rows of two ranks
                n = rd.x.numel()
                xs.append(room[at:at + n].view_as(rd.x).copy_(rd.x))
                ys.append(room[at + 3 * H:at + 3 * H + n].view_as(rd.x))
                at += n
            assert all(torch.equal(a, b) for a, b in zip(steps(xs, ys, whole), want))
            assert all(torch.equal(a, b) for a, b in zip(state(world), tables))
    finally:
        world.close()


@pytest.mark.parametrize("payload", ["direct", "dedup", "fp8"])
@pytest.mark.parametrize("E,K,H,T,ws", [
    (12, 3, 640, 33, 3),      # ranks that do not divide the grid, rows that end inside a warp's piece
    (48, 11, 1152, 70, 2),    # more pairs than are requested together
    (8, 2, 7168, 300, 8),     # 1 KB a warp in every phase; 69 MB of rows: phases that begin with the last rows
    (256, 32, 128, 20, 8),    # the most experts a token, a row of one scale block
])
def test_phases_of_a_group_equal_those_rank_by_rank(payload, E, K, H, T, ws):
    """In one call, with receiving and expert op in one launch, phase by phase, sent rank by rank and received together, and
    the other way round."""
    rds = [pkg.generate_input(E, K, H, T, seed=9, rank=r, world_size=ws)[1].to(DEV) for r in range(ws)]
    for name in ("x", "indices", "weights"):  # a rank without tokens
        setattr(rds[1], name, getattr(rds[1], name)[:0].contiguous())
    rds[1].num_tokens = 0
    rds[0].indices[3, :] = rds[0].indices[3, 0]  # repeats, and a token without a valid expert: dropped, zero
    rds[0].indices[T - 1, :] = E
    world = LocalWorld(pkg.MoEConfig(E, K, H, T), ws, payload=payload)

    def by_steps(send, recv):
        if send:
            world._send(rds)
        else:
            for c, rd in zip(world.ctxs, rds):
                c.route(rd.indices)
                c.dispatch_send(rd.x)
        if recv:
            world._step("recv")
            world._step("expert")
            return world._combine(rds)
        for c in world.ctxs[:-1]:
            c.dispatch_recv()
            c.expert_placeholder()
        world.ctxs[-1].dispatch_recv_expert()
        return [c.combine(rd.weights) for c, rd in zip(world.ctxs, rds)]

    try:
        want = [bits(y) for y in rank_by_rank(world, rds)]
        tables = state(world)
        for run in (lambda: world.forward_phases(rds), lambda: world.forward(rds), lambda: by_steps(True, True), lambda: by_steps(False, True),
                    lambda: by_steps(True, False)):
            for c in world.ctxs:
                c.expert_buffers()[0].zero_()
            assert all(torch.equal(bits(g), w) for g, w in zip(run(), want))
            assert all(torch.equal(a, b) for a, b in zip(state(world), tables))
        assert not want[0][T - 1].any()
        assert [c.peek() for c in world.ctxs] == [_lib.A2A_ERR_ROUTING] + [0] * (ws - 1)
    finally:
        world.close()


@pytest.mark.parametrize("names", [("send", "recv", "expert", "combine"), ("send", "recv_expert", "combine")])
@pytest.mark.parametrize("payload", ["direct", "fp8"])
def test_phases_go_on_after_a_refused_combine(names, payload):
    """What was launched before the refusal stands as if it had been called phase by phase: the combine follows, for all
    ranks together or rank by rank, and waits for nothing that never comes."""
    ws, E, K, H, T = 3, 12, 3, 640, 33
    rds = [pkg.generate_input(E, K, H, T, seed=10, rank=r, world_size=ws)[1].to(DEV) for r in range(ws)]
    world = LocalWorld(pkg.MoEConfig(E, K, H, T), ws, payload=payload, timeout_ms=300)
    lib, handles = world.ctxs[0].lib, (C.c_void_p * ws)(*[c._h.value for c in world.ctxs])
    phases = (C.c_int32 * len(names))(*[_lib.GROUP_PHASE[name] for name in names])
    try:
        want = [bits(y) for y in world.forward_phases(rds)]
        tables = state(world)
        for field, wrong in (("y", 0), ("y", 2), ("topk_weights", 0)):  # missing, off a 16-byte boundary, missing
            for together in (True, False):
                ys, calls, done = [torch.full_like(rd.x, 3) for rd in rds], (_lib.Call * ws)(), C.c_int32()
                for c, call, rd, y in zip(world.ctxs, calls, rds, ys):
                    call.x, call.topk_idx, call.topk_weights = rd.x.data_ptr(), rd.indices.data_ptr(), rd.weights.data_ptr()
                    call.y, call.num_tokens = y.data_ptr(), rd.num_tokens
                    c._num_tokens = rd.num_tokens
                good = getattr(calls[ws - 1], field)
                setattr(calls[ws - 1], field, good + wrong if wrong else None)
                rc = lib.a2a_group_steps(handles, phases, len(names), calls, _lib.current_stream(), C.byref(done))
                assert rc == _lib.A2A_ERR_CONFIG and done.value == len(names) - 1
                setattr(calls[ws - 1], field, good)
                if together:
                    world._step("combine", calls)
                else:
                    ys = [c.combine(rd.weights) for c, rd in zip(world.ctxs, rds)]
                torch.cuda.synchronize()
                world.check()
                assert all(torch.equal(bits(y), w) for y, w in zip(ys, want))
                assert all(torch.equal(a, b) for a, b in zip(state(world), tables))
        assert all(torch.equal(bits(y), w) for y, w in zip(world.forward_phases(rds), want))
        world.check()
    finally:
        world.close()


@pytest.mark.parametrize("payload", ["dedup", "fp8"])
@pytest.mark.parametrize("E,K,H,T,ws", [(12, 3, 640, 33, 3), (16, 8, 2944, 70, 2)])
def test_a_combine_of_all_ranks_finds_rows_by_their_slots(payload, E, K, H, T, ws):
    """After calls that leave no list of places, the one launch and the roles rank by rank: the bits of the PULL combine, dropped
    pairs among them."""
    rds = [pkg.generate_input(E, K, H, T, seed=11, rank=r, world_size=ws)[1].to(DEV) for r in range(ws)]
    rds[0].indices[3, :] = rds[0].indices[3, 0]
    rds[0].indices[T - 1, :] = E
    world = LocalWorld(pkg.MoEConfig(E, K, H, T), ws, payload=payload, schedule="pipelined", combine="pull")
    try:
        for run in (lambda: world.forward_one_launch(rds), lambda: rank_by_rank(world, rds), lambda: world.forward_pipelined(rds)):
            want = [bits(y) for y in run()]
            for c, rd in zip(world.ctxs, rds):
                c._num_tokens = T
            assert all(torch.equal(bits(y), w) for y, w in zip(world._combine(rds), want))
        assert [c.peek() for c in world.ctxs] == [_lib.A2A_ERR_ROUTING] + [0] * (ws - 1)
    finally:
        world.close()
