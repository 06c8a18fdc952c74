"""The one-launch kernel of world size 1 where its split can go wrong: rows that end inside a warp's
item, one token, more tokens per block than it resolves at a time, K beyond one vector of indices,
token counts whose stepped roles need more than half an SM's shared memory.

Dispatch is held bit for bit against the CPU checker; outputs against the same sums in 64 bits within
the roundings the kernel makes, and bit for bit against the stepped roles, which are other kernels.
"""
import pytest
import torch

import gpu_mode_kernels_b200 as pkg
from gpu_mode_kernels_b200 import _lib
from gpu_mode_kernels_b200.all2all import A2AContext
from gpu_mode_kernels_b200.local_world import LocalWorld
from oracle import a2a_oracle as O
from parity import fp8_roundtrip

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def bits(t):
    return t.contiguous().view(torch.int16)


@pytest.mark.parametrize("E,K,H,T,n,dtype,payload", [
    (8, 1, 8, 1, 1, torch.bfloat16, "dedup"),         # a row of one vector
    (6, 3, 520, 33, 20, torch.float16, "dedup"),      # 65 vectors: one past two lanes' worth
    (64, 6, 2048, 4, 0, torch.float16, "dedup"),      # no tokens
    (1024, 32, 128, 40, 40, torch.bfloat16, "dedup"), # limits of E and K
    (8, 2, 72, 6000, 5003, torch.bfloat16, "dedup"),  # 17 tokens per block: a second round for some blocks
    (256, 8, 7168, 256, 255, torch.bfloat16, "dedup"),
    (256, 8, 64, 2048, 2048, torch.float16, "dedup"), # stepped roles: 133 KB of routing tables
    (6, 3, 640, 33, 33, torch.float16, "fp8"),
    (32, 4, 7168, 200, 199, torch.bfloat16, "fp8"),
])
def test_forward_against_the_checker_and_the_stepped_roles(E, K, H, T, n, dtype, payload):
    cfg, rd, _, _ = pkg.generate_input(E, K, H, T, seed=11, rank=0, world_size=1, dtype=dtype, weights="rand")
    rd.num_tokens = n
    rd.x, rd.indices, rd.weights = rd.x[:n], rd.indices[:n], rd.weights[:n]
    disp, _ = O.simulate(cfg, 1, [rd])
    ctx = A2AContext(cfg, 0, 1, device=0, payload=payload, schedule="pipelined", combine="push")
    world = LocalWorld(cfg, 1, payload=payload, schedule="pipelined", combine="push")
    try:
        d = rd.to(DEV)
        before = ctx.launches
        y = ctx.forward(d.x, d.indices, d.weights)
        assert ctx.launches == before + 1
        slots, sent = ctx.route_tables()
        counts, rows, meta = ctx.export_dispatch()
        torch.cuda.synchronize()
        ctx.check()
        want_slots, want_sent = O.route_tables(rd.indices, E)
        assert torch.equal(slots.cpu(), want_slots) and torch.equal(sent.cpu(), want_sent)
        assert torch.equal(counts.cpu(), disp[0].expert_num_tokens)
        held = counts.cpu().tolist()
        got = torch.cat([rows[e, :h] for e, h in enumerate(held)], 0).cpu()
        assert torch.equal(torch.cat([meta[e, :h] for e, h in enumerate(held)], 0).cpu(), disp[0].meta)
        want = disp[0].rows
        if payload == "fp8":
            want = fp8_roundtrip(want, dtype)
        assert torch.equal(bits(got), bits(want))  # rank 0: the placeholder op multiplies by one
        # K fp32 multiply-adds (each within 2^-24 of the terms' magnitudes), then one rounding to the element
        # type (half an ulp: a bf16 significand has 8 bits, so 2^-8 of the result; fp16 11 bits, 2^-11; 2^-25 where fp16 is subnormal)
        x = (fp8_roundtrip(rd.x, dtype) if payload == "fp8" and n else rd.x).double()
        w = rd.weights.double()
        exact, terms = x * w.sum(1, keepdim=True), x.abs() * w.sum(1, keepdim=True)
        bound = exact.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) + 2.0 ** -25 + (K + 1) * 2.0 ** -24 * terms
        assert bool(((y.cpu().double() - exact).abs() <= bound).all())
        ref = world.forward_pipelined([d])[0]
        torch.cuda.synchronize()
        world.check()
        assert torch.equal(bits(ref), bits(y))
    finally:
        ctx.close()
        world.close()


@pytest.mark.parametrize("E,K,H,T,n,dtype,payload", [
    (8, 2, 2048, 1280, 1280, torch.bfloat16, "dedup"),  # the fewest tokens, whole blocks of 64
    (64, 6, 520, 2100, 2049, torch.float16, "dedup"),   # one token in the last routing block, rows that end inside a warp
    (40, 32, 264, 1300, 1283, torch.bfloat16, "dedup"), # the most experts a token
    (256, 8, 640, 1344, 1343, torch.bfloat16, "fp8"),
    (8, 2, 2048, 1280, 1279, torch.bfloat16, "dedup"),  # one token fewer: one launch
])
def test_many_tokens_match_the_stepped_roles(E, K, H, T, n, dtype, payload):
    """Routing and rows as two launches; repeated and out-of-range experts on both sides of a 32- and a 64-token edge."""
    cfg, rd, _, _ = pkg.generate_input(E, K, H, T, seed=13, rank=0, world_size=1, dtype=dtype, weights="rand")
    rd.num_tokens = n
    rd.x, rd.indices, rd.weights = rd.x[:n], rd.indices[:n], rd.weights[:n]
    for t in (31, 32, 63, 64, 127, n - 1):
        rd.indices[t, K - 1] = rd.indices[t, 0]
    rd.indices[95], rd.indices[96, 0] = -1, E
    ctx = A2AContext(cfg, 0, 1, device=0, payload=payload, schedule="pipelined", combine="push", timeout_ms=500)
    world = LocalWorld(cfg, 1, payload=payload, schedule="pipelined", combine="push")
    try:
        d = rd.to(DEV)
        before = ctx.launches
        y = ctx.forward(d.x, d.indices, d.weights)
        assert ctx.launches == before + (2 if n >= 1280 else 1)
        ref = world.forward_pipelined([d])[0]
        got, want = ctx.route_tables() + ctx.export_dispatch(), world.ctxs[0].route_tables() + world.ctxs[0].export_dispatch()
        again = torch.empty_like(y)  # a combine called on its own finds the flags up
        _lib.check(ctx.lib.a2a_combine(ctx._h, d.weights.data_ptr(), again.data_ptr(), torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert ctx.peek() == _lib.A2A_ERR_ROUTING
        assert all(torch.equal(a, b) for a, b in zip(got, want))
        assert torch.equal(bits(ref), bits(y)) and torch.equal(bits(again), bits(y)) and not y[95].any()
    finally:
        ctx.close()
        world.close()


@pytest.mark.parametrize("E,K,H,T,launches", [
    (64, 8, 4096, 640, 2), (64, 8, 4096, 639, 1),    # 40 MB of expert rows, and a token less
    (32, 6, 2048, 800, 2), (32, 6, 2048, 799, 1),    # 800 tokens of more than 16 MB, and 799
    (16, 4, 2624, 800, 2), (16, 4, 2616, 800, 1),    # just above 16 MB, and below
    (8, 2, 824, 1280, 2), (8, 2, 816, 1280, 1),      # 1280 tokens of 4 MB, and of less
])
def test_where_a_call_takes_two_launches(E, K, H, T, launches):
    cfg, rd, _, _ = pkg.generate_input(E, K, H, T, seed=14, rank=0, world_size=1)
    ctx = A2AContext(cfg, 0, 1, device=0, payload="dedup", schedule="pipelined", combine="push", timeout_ms=500)
    world = LocalWorld(cfg, 1, payload="dedup", schedule="pipelined", combine="push")
    try:
        d = rd.to(DEV)
        before = ctx.launches
        y = ctx.forward(d.x, d.indices, d.weights)
        assert ctx.launches == before + launches
        ref = world.forward_pipelined([d])[0]
        got, want = ctx.route_tables() + ctx.export_dispatch(), world.ctxs[0].route_tables() + world.ctxs[0].export_dispatch()
        torch.cuda.synchronize()
        ctx.check()
        assert torch.equal(bits(ref), bits(y)) and all(torch.equal(a, b) for a, b in zip(got, want))
    finally:
        ctx.close()
        world.close()


@pytest.mark.parametrize("E,K,H,T", [(16, 4, 72, 100), (64, 12, 1024, 300), (16, 8, 4096, 900)])
def test_indices_wherever_they_begin(E, K, H, T):
    """Indices in whole 16-byte vectors and one to three words past them: one launch, two, a group and its phases."""
    rds = [pkg.generate_input(E, K, H, T, seed=15, rank=r, world_size=2)[1].to(DEV) for r in range(2)]
    for rd in rds:
        rd.indices[T - 2, K - 1] = rd.indices[T - 2, 0]
    cfg = pkg.MoEConfig(E, K, H, T)
    ctx = A2AContext(cfg, 0, 1, device=0, payload="dedup", schedule="pipelined", combine="push")
    worlds = [LocalWorld(cfg, 2, payload="dedup", schedule="pipelined", combine="push"), LocalWorld(cfg, 2)]
    base = torch.empty(2, T * K + 4, dtype=torch.int32, device=DEV)
    want = None
    try:
        for off in range(4):
            for r, rd in enumerate(rds):
                place = base[r, off:off + T * K].view(T, K)
                place.copy_(rd.indices.clone())
                rd.indices = place
            got = [ctx.forward(rds[0].x, rds[0].indices, rds[0].weights)] + worlds[0].forward_pipelined(rds) + worlds[1].forward_phases(rds)
            got = [bits(y) for y in got] + list(ctx.route_tables()) + [t for w in worlds for c in w.ctxs for t in c.route_tables()]
            torch.cuda.synchronize()
            want = want or got
            assert all(torch.equal(a, b) for a, b in zip(got, want))
        slots = torch.zeros_like(got[-2])
        sent = torch.zeros(E, dtype=torch.int32, device=DEV)
        lib = _lib.load()
        assert lib.a2a_route_noalloc(rds[1].indices.data_ptr(), T, E, K, slots.data_ptr(), sent.data_ptr(), None) == 0
        torch.cuda.synchronize()
        assert torch.equal(got[-2], slots) and torch.equal(got[-1], sent)
    finally:
        ctx.close()
        for w in worlds:
            w.close()


def test_dropped_pairs_match_the_stepped_roles_and_phases_can_follow():
    """Indices out of range and repeated, the repeats also across the eight indices the kernel loads
    together and in tokens before the reading block's own; then a combine called on its own, which
    must find the flags of the forward up."""
    E, K, H, T = 16, 11, 2048, 300
    cfg, rd, _, _ = pkg.generate_input(E, K, H, T, seed=12, rank=0, world_size=1, weights="rand")
    rd.indices[3, 9] = rd.indices[3, 1]
    rd.indices[3, 2] = rd.indices[3, 1]
    rd.indices[150, 10] = rd.indices[150, 8]
    rd.indices[299] = -1
    rd.indices[20, 0] = E
    ctx = A2AContext(cfg, 0, 1, device=0, payload="dedup", schedule="pipelined", combine="push", timeout_ms=500)
    world = LocalWorld(cfg, 1, payload="dedup", schedule="pipelined", combine="push")
    try:
        d = rd.to(DEV)
        y = ctx.forward(d.x, d.indices, d.weights)
        ref = world.forward_pipelined([d])[0]
        tables, want = ctx.route_tables(), world.ctxs[0].route_tables()
        again = torch.empty_like(y)
        _lib.check(ctx.lib.a2a_combine(ctx._h, d.weights.data_ptr(), again.data_ptr(), torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert ctx.peek() == _lib.A2A_ERR_ROUTING and world.ctxs[0].peek() == _lib.A2A_ERR_ROUTING
        assert all(torch.equal(a, b) for a, b in zip(tables, want))
        assert torch.equal(bits(ref), bits(y)) and torch.equal(bits(again), bits(y))
        assert not y[299].any()
    finally:
        ctx.close()
        world.close()


@pytest.mark.parametrize("place", ["pinned", "pageable", "pinned_x_only", "off_alignment", "in_place", "spans_two"])
@pytest.mark.parametrize("K,H,T,n,payload", [(2, 8, 1, 1, "dedup"), (6, 2056, 93, 80, "dedup"), (8, 1024, 300, 300, "fp8")])
def test_host_tensors_wherever_they_live(place, K, H, T, n, payload):
    """Pinned rows are read and written by the kernel itself, all others copied: the bits of the device call
    either way."""
    cfg, rd, _, _ = pkg.generate_input(16, K, H, T, seed=21, rank=0, world_size=1, weights="rand")
    x, idx, w = rd.x[:n].contiguous(), rd.indices[:n].contiguous(), rd.weights[:n].contiguous()
    ctx = A2AContext(cfg, 0, 1, device=0, payload=payload, schedule="pipelined", combine="push")
    pinned = []
    try:
        want = bits(ctx.forward(x.to(DEV), idx.to(DEV), w.to(DEV))).cpu()
        y = torch.empty(n, H, dtype=cfg.out_dtype, pin_memory=place != "pageable")
        if place != "pageable":
            x = x.pin_memory()
        if place in ("pinned", "in_place"):
            idx, w = idx.pin_memory(), w.pin_memory()
        if place == "off_alignment":  # two bytes past a 16-byte boundary
            base = torch.empty(n * H + 8, dtype=x.dtype, pin_memory=True)
            x = base[1:1 + n * H].view(n, H).copy_(x)
        if place == "in_place":
            y = x
        if place == "spans_two":  # only the first page of the rows is registered
            base = torch.empty(n * H * 2 + 8192, dtype=torch.uint8)
            at = -base.data_ptr() % 4096
            x = base[at:at + n * H * 2].view(x.dtype).view(n, H).copy_(x)
            assert torch.cuda.cudart().cudaHostRegister(x.data_ptr(), 4096, 0) == torch.cuda.cudart().cudaError.success
            pinned.append(x.data_ptr())
        if place == "spans_two" and n * H * 2 > 4096:  # the copy refuses such rows; so does what replaces it
            with pytest.raises(_lib.A2AError):
                ctx.forward_host(x, idx, w, y)
            return
        got = ctx.forward_host(x, idx, w, y)
        torch.cuda.synchronize()
        ctx.check()
        assert torch.equal(bits(got), want)
        again = torch.empty(n, H, dtype=cfg.out_dtype, device=DEV)  # the phases after it find what they need
        _lib.check(ctx.lib.a2a_combine(ctx._h, w.to(DEV).data_ptr(), again.data_ptr(), torch.cuda.current_stream().cuda_stream))
        assert torch.equal(bits(again).cpu(), want)
    finally:
        torch.cuda.synchronize()
        for ptr in pinned:
            torch.cuda.cudart().cudaHostUnregister(ptr)
        ctx.close()


@pytest.mark.parametrize("combine", ["push", "pull"])
def test_roles_are_refused_where_the_call_was_not_begun_by_role_0(combine):
    """The one launch writes none of the records that roles 1 and 2 work from: what lies there is of an earlier,
    larger call."""
    cfg, rd, _, _ = pkg.generate_input(8, 2, 64, 40, seed=31, rank=0, world_size=1)
    big, n = rd.to(DEV), 5
    few = [t[:n].contiguous() for t in (rd.x, rd.indices, rd.weights)]
    ctx = A2AContext(cfg, 0, 1, device=0, payload="dedup", schedule="pipelined", combine=combine)
    try:
        def step_all():
            ctx.pipe_step(0, big.x, big.indices, big.weights)
            ctx.pipe_step(1)
            return ctx.pipe_step(2)

        want = bits(step_all())
        assert torch.equal(bits(ctx.forward(big.x, big.indices, big.weights)), want)
        by_phases = [t.to(DEV) for t in few]

        def begin_phases():
            ctx.route(by_phases[1])
            ctx.dispatch_send(by_phases[0])

        for begin in (lambda: ctx.forward(*by_phases), lambda: ctx.forward_host(*few),
                      lambda: ctx.forward_host(*[t.pin_memory() for t in few]), begin_phases):
            begin()
            before = ctx.launches
            for role in (1, 2):
                with pytest.raises(_lib.A2AError) as refused:
                    ctx.pipe_step(role)
                assert refused.value.code == _lib.A2A_ERR_STATE
            assert ctx.launches == before
            assert torch.equal(bits(step_all()), want)
        ctx.check()
    finally:
        torch.cuda.synchronize()
        ctx.close()


@pytest.mark.parametrize("over", ["weights", "x"])
@pytest.mark.parametrize("payload,H", [("dedup", 72), ("fp8", 128)])
def test_output_laid_over_an_input(payload, H, over):
    """More tokens than the blocks resolve at a time: the weights of a block's second round lie under output
    rows of its first."""
    T, K = 6000, 2
    cfg, rd, _, _ = pkg.generate_input(8, K, H, T, seed=41, rank=0, world_size=1, weights="rand")
    d = rd.to(DEV)
    ctx = A2AContext(cfg, 0, 1, device=0, payload=payload, schedule="pipelined", combine="push")
    try:
        want = bits(ctx.forward(d.x, d.indices, d.weights))
        y = torch.empty_like(d.x)
        x, w = d.x, d.weights
        if over == "x":
            x = y.copy_(d.x)
        else:
            w = y.view(-1)[8:8 + 2 * T * K].view(torch.float32).view(T, K).copy_(d.weights)
        assert torch.equal(bits(ctx.forward(x, d.indices, w, y)), want)
        ctx.check()
    finally:
        torch.cuda.synchronize()
        ctx.close()


@pytest.mark.parametrize("over", ["weights", "indices"])
@pytest.mark.parametrize("combine", ["push", "pull"])
@pytest.mark.parametrize("payload,H,T,K", [("dedup", 72, 6000, 2), ("dedup", 2056, 37, 5), ("fp8", 256, 700, 8), ("dedup", 64, 1, 3)])
def test_weights_and_indices_are_read_before_the_first_row_is_written(payload, H, T, K, combine, over):
    """An output laid over them, with a repeat and a token without a valid expert, in every combine mode: slots and
    outputs to the bit."""
    cfg, rd, _, _ = pkg.generate_input(8, K, H, T, seed=42, rank=0, world_size=1, weights="rand")
    rd.indices[T - 1, :] = 8
    rd.indices[0, K - 1] = rd.indices[0, 0]
    d = rd.to(DEV)
    ctx = A2AContext(cfg, 0, 1, device=0, payload=payload, schedule="pipelined", combine=combine)
    try:
        want = bits(ctx.forward(d.x, d.indices, d.weights))
        tables = [t.clone() for t in ctx.route_tables() + ctx.export_dispatch()]
        for at in (0, 8, (T * H - 2 * T * K) // 8 * 8):
            if at + 2 * T * K > T * H:
                continue
            y = torch.full_like(d.x, 7)
            idx, w = d.indices, d.weights
            place = y.view(-1)[at:at + 2 * T * K]
            if over == "weights":
                w = place.view(torch.float32).view(T, K).copy_(d.weights)
            else:
                idx = place.view(torch.int32).view(T, K).copy_(d.indices)
            assert torch.equal(bits(ctx.forward(d.x, idx, w, y)), want)
            assert all(torch.equal(a, b) for a, b in zip(ctx.route_tables() + ctx.export_dispatch(), tables))
        assert ctx.peek() == _lib.A2A_ERR_ROUTING and not want[T - 1].any()
    finally:
        torch.cuda.synchronize()
        ctx.close()
