"""The compiled part of the Python layer: the same answers and errors as the Python code behind it, for plain and
for unusual inputs."""
from types import SimpleNamespace

import pytest
import torch

import gpu_mode_kernels_b200 as pkg
from gpu_mode_kernels_b200 import _lib, all2all, histogram
from gpu_mode_kernels_b200.all2all import A2AContext, A2AError, custom_kernel, release_contexts
from gpu_mode_kernels_b200.local_world import LocalWorld

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


class Sub(torch.Tensor):
    pass


def bits(t):
    return t.contiguous().view(torch.int16)


def data_of(rd, **changed):
    return SimpleNamespace(**{**dict(num_tokens=rd.num_tokens, x=rd.x, indices=rd.indices, weights=rd.weights), **changed})


FORMS = {
    "plain": lambda rd: {},
    "strided x": lambda rd: dict(x=rd.x.t().contiguous().t()),
    "every second row": lambda rd: dict(x=rd.x.repeat_interleave(2, 0)[::2]),
    "int64 indices": lambda rd: dict(indices=rd.indices.long()),
    "strided indices": lambda rd: dict(indices=rd.indices.t().contiguous().t()),
    "double weights": lambda rd: dict(weights=rd.weights.double()),
    "a subclass": lambda rd: dict(x=rd.x.as_subclass(Sub)),
    "needs a gradient": lambda rd: dict(x=rd.x.clone().requires_grad_()),
    "no tokens": lambda rd: dict(x=rd.x[:0], indices=rd.indices[:0], weights=rd.weights[:0]),
}


@pytest.mark.parametrize("form", FORMS)
def test_what_was_accepted_gives_the_same_bits(form):
    cfg, rd, _, _ = pkg.generate_input(8, 3, 264, 9, seed=3, rank=0, world_size=1, device=DEV)
    ctx = A2AContext(cfg, 0, 1, device=0, payload="dedup", schedule="pipelined", combine="push")
    try:
        d = data_of(rd, **FORMS[form](rd))
        want = torch.empty(d.x.shape, dtype=rd.x.dtype, device=DEV)  # an output of its own: the code behind the compiled part
        want = ctx.forward(d.x.contiguous(), d.indices.to(torch.int32).contiguous(), d.weights.float().contiguous(), want)
        y = custom_kernel((cfg, d, 0, 1))
        assert type(y) is torch.Tensor and y.dtype == want.dtype and not y.requires_grad and torch.equal(bits(y), bits(want))
    finally:
        ctx.close()
        release_contexts(barrier=False)


@pytest.mark.parametrize("wrong", [
    dict(x=lambda t: t.half()), dict(x=lambda t: t[:, :-8]), dict(x=lambda t: t[0]), dict(x=lambda t: t.cpu(), indices=None),
    dict(indices=lambda t: t[:-1].contiguous()), dict(weights=lambda t: t[:, :1].contiguous()), dict(weights=lambda t: t.cpu()),
])
def test_what_was_refused_is_refused(wrong):
    cfg, rd, _, _ = pkg.generate_input(8, 3, 264, 9, seed=3, rank=0, world_size=1, device=DEV)
    ctx = A2AContext(cfg, 0, 1, device=0, payload="dedup", schedule="pipelined", combine="push")
    try:
        d = data_of(rd, **{k: f(getattr(rd, k)) for k, f in wrong.items() if f})
        for call in (lambda: ctx.forward(d.x, d.indices, d.weights), lambda: custom_kernel((cfg, d, 0, 1))):
            with pytest.raises(A2AError) as refused:
                call()
            assert refused.value.code == _lib.A2A_ERR_CONFIG
        with pytest.raises(A2AError) as refused:  # more tokens than the context was made for
            ctx.forward(rd.x.repeat(2, 1), rd.indices.repeat(2, 1), rd.weights.repeat(2, 1))
        assert refused.value.code == _lib.A2A_ERR_CONFIG
        ctx.close()
        with pytest.raises(A2AError):
            ctx.forward(rd.x, rd.indices, rd.weights)
    finally:
        ctx.close()
        release_contexts(barrier=False)


@pytest.mark.parametrize("schedule,payload,combine", [("pipelined", "dedup", "push"), ("phased", "direct", "pull")])
def test_a_group_with_unusual_data(schedule, payload, combine):
    rds = [pkg.generate_input(8, 2, 264, 6, seed=4, rank=r, world_size=2)[1].to(DEV) for r in range(2)]
    world = LocalWorld(pkg.MoEConfig(8, 2, 264, 6), 2, payload=payload, schedule=schedule, combine=combine)
    forward = world.forward_pipelined if schedule == "pipelined" else world.forward_phases
    try:
        want = [bits(y) for y in forward(rds)]
        def kept(datas, ys):
            for c, d, y in zip(world.ctxs, datas, ys):
                held = [d.x, d.indices, d.weights, y] if schedule == "pipelined" else [d.indices, d.x, d.weights]
                assert [t.data_ptr() for t in c._keep] == [t.data_ptr() for t in held]
                assert schedule != "pipelined" or c._y is y

        ys = forward(rds)
        kept(rds, ys)
        odd = [data_of(rds[0], x=rds[0].x.as_subclass(Sub)), rds[1]]  # goes through the Python code
        ys = forward(tuple(odd))
        assert all(torch.equal(bits(y), w) for y, w in zip(ys, want))
        kept(odd, ys)
        assert [c._num_tokens for c in world.ctxs] == [6, 6]
        with pytest.raises(A2AError) as refused:
            forward(rds[:1])
        assert refused.value.code == _lib.A2A_ERR_STATE
        before = [c.launches for c in world.ctxs]
        with pytest.raises(A2AError):
            big = data_of(rds[0], x=rds[0].x.repeat(2, 1), indices=rds[0].indices.repeat(2, 1), weights=rds[0].weights.repeat(2, 1))
            forward([big, rds[1]])
        assert [c.launches for c in world.ctxs] == before
        assert all(torch.equal(bits(y), w) for y, w in zip(forward(rds), want))
        world.check()
    finally:
        world.close()


def test_histogram_of_unusual_tensors():
    data = torch.randint(0, 256, (5000,), dtype=torch.uint8, device=DEV)
    want = torch.bincount(data.cpu(), minlength=256)
    out = torch.empty(256, dtype=torch.int64, device=DEV)
    assert histogram.custom_kernel((data, out)) is out and torch.equal(out.cpu(), want)
    assert torch.equal(histogram.custom_kernel((data.as_subclass(Sub), out.view(16, 16))).cpu().view(256), want)
    for bad in ((data.cpu(), out), (data.int(), out), (data[::2], out), (data.view(50, 100), out), (data, out[:128]), (data, out.cpu())):
        with pytest.raises(A2AError) as refused:
            histogram.custom_kernel(bad)
        assert refused.value.code == _lib.A2A_ERR_CONFIG


def test_side_streams_and_threads():
    """Calls go to the caller's current stream, from whichever thread."""
    import threading

    cfg, rd, _, _ = pkg.generate_input(8, 3, 264, 9, seed=3, rank=0, world_size=1, device=DEV)
    ctxs = [A2AContext(cfg, 0, 1, device=0, payload="dedup", schedule="pipelined", combine="push") for _ in range(3)]
    got = [None] * 3
    try:
        want = bits(ctxs[0].forward(rd.x, rd.indices, rd.weights))
        torch.cuda.synchronize()

        def work(i):
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(50):
                    y = ctxs[i].forward(rd.x, rd.indices, rd.weights)
                torch.cuda.current_stream().synchronize()
                got[i] = y

        threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
        [t.start() for t in threads]
        [t.join() for t in threads]
        assert all(torch.equal(bits(y), want) for y in got)
    finally:
        [c.close() for c in ctxs]
    assert all2all._CONTEXTS == {}


@pytest.mark.parametrize("what", ["one rank", "many tokens", "group", "phases", "histogram"])
def test_calls_under_graph_capture(what):
    """Captured launches, those that overlap included, replayed on other inputs."""
    ws, E, K, H, T = 2, 8, 2, 2048, 1300 if what == "many tokens" else 40
    sets = [[pkg.generate_input(E, K, H, T, seed=s, rank=r, world_size=ws)[1].to(DEV) for r in range(ws)] for s in (1, 2)]
    cfg = pkg.MoEConfig(E, K, H, T)
    data, counts = torch.zeros(300000, dtype=torch.uint8, device=DEV), torch.empty(256, dtype=torch.int64, device=DEV)
    held = [data_of(rd, x=rd.x.clone(), indices=rd.indices.clone(), weights=rd.weights.clone()) for rd in sets[0]]
    world = None
    if what in ("group", "phases"):
        world = LocalWorld(cfg, ws, payload="dedup" if what == "group" else "direct",
                           schedule="pipelined" if what == "group" else "phased", combine="push" if what == "group" else "pull")
    try:
        def call():
            if what == "histogram":
                return [histogram.custom_kernel((data, counts))]
            if world is None:
                return [custom_kernel((cfg, held[0], 0, 1))]
            return world.forward_pipelined(held) if what == "group" else world.forward_phases(held)

        call()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs = [o for _ in range(3) for o in call()]
        for rds in sets[::-1]:
            for h, rd in zip(held, rds):
                h.x.copy_(rd.x), h.indices.copy_(rd.indices), h.weights.copy_(rd.weights)
            data.random_(0, 256)
            graph.replay()
            torch.cuda.synchronize()
            got = [o.clone() for o in outs]
            want = [o.clone() for o in call()] * 3
            assert all(torch.equal(a, b) for a, b in zip(got, want))
        if what == "histogram":
            assert torch.equal(counts.cpu(), torch.bincount(data.cpu(), minlength=256))
    finally:
        if world is not None:
            world.close()
        release_contexts(barrier=False)


def test_a_dispatch_mode_still_hears_of_the_outputs():
    """Outputs are allocated without the dispatcher only where no mode listens."""
    from torch.utils._python_dispatch import TorchDispatchMode

    class Listen(TorchDispatchMode):
        def __init__(self):
            super().__init__()
            self.shapes = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            out = func(*args, **(kwargs or {}))
            if "empty" in func.name():
                self.shapes.append(tuple(out.shape))
            return out

    cfg = pkg.MoEConfig(8, 2, 64, 4)
    rds = [pkg.generate_input(8, 2, 64, 4, seed=1, rank=r, world_size=2)[1].to(DEV) for r in range(2)]
    ctx = A2AContext(cfg, 0, 1, device=0, payload="dedup", schedule="pipelined", combine="push")
    world = LocalWorld(cfg, 2, payload="dedup", schedule="pipelined", combine="push")
    try:
        want = [ctx.forward(rds[0].x, rds[0].indices, rds[0].weights)] + world.forward_pipelined(rds)
        with Listen() as heard:
            got = [ctx.forward(rds[0].x, rds[0].indices, rds[0].weights)] + world.forward_pipelined(rds)
        assert heard.shapes == [(4, 64)] * 3
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    finally:
        ctx.close()
        world.close()


def test_a_profiler_still_sees_the_outputs():
    """Observers of operators are no modes; they too hear of every output."""
    from torch.profiler import ProfilerActivity, profile

    cfg = pkg.MoEConfig(8, 2, 64, 4)
    rds = [pkg.generate_input(8, 2, 64, 4, seed=1, rank=r, world_size=2)[1].to(DEV) for r in range(2)]
    ctx = A2AContext(cfg, 0, 1, device=0, payload="dedup", schedule="pipelined", combine="push")
    world = LocalWorld(cfg, 2, payload="dedup", schedule="pipelined", combine="push")
    try:
        want = [ctx.forward(rds[0].x, rds[0].indices, rds[0].weights)] + world.forward_pipelined(rds)
        with profile(activities=[ProfilerActivity.CPU]) as seen:
            got = [ctx.forward(rds[0].x, rds[0].indices, rds[0].weights)] + world.forward_pipelined(rds)
        assert [e.name for e in seen.events()].count("aten::empty") == 3
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    finally:
        ctx.close()
        world.close()
