"""Several ranks on ONE GPU, run phase by phase in one process.

Kernels that wait on a peer must never share a GPU with the kernel they wait
for, so the ranks here are stepped in lock-step: one launch runs a phase of every
rank, the sending phase before any waiting one, on one stream, and each wait finds its
flag already set.  Routing, rows, flag values and epochs are those of a group
with a GPU per rank; what depends on where a peer is, is not: flags are awaited at gpu
scope without watchers, rows are read where they lie and written where they belong instead of being sent to a
stage, and a token's output is added up where its expert rows are written (csrc/a2a_near.cuh).  The forms for
distant peers run in ``forward_one_launch``, which puts every rank's blocks into one cooperative
launch, and in the phases called context by context.
Validation tool: parity tests and the smoke check use it to cover world sizes
2, 4 and 8 on a single device.  What it takes is the time of ranks that share a GPU, by kernels for near peers; it
says nothing of a group with a GPU per rank, which runs the one-launch kernel (csrc/a2a_pipe.cuh) over links.
"""
from __future__ import annotations

import ctypes as C
from typing import List, Sequence

import torch

from . import _lib
from .all2all import A2AContext
from .task import MoEConfig

# what a call's launches are, in order
_PHASES, _FUSED, _ROLES = (tuple(_lib.GROUP_PHASE[name] for name in names) for names in (
    ("send", "recv", "expert", "combine"), ("send", "recv_expert", "combine"), ("pipe_send", "pipe_expert", "pipe_combine")))


class LocalWorld:
    def __init__(self, cfg: MoEConfig, world_size: int, *, payload: str = "direct", schedule: str = "phased",
                 combine: str = "pull", timeout_ms: int = 2000, device: int = 0):
        self.cfg, self.world_size = cfg, world_size
        self.ctxs: List[A2AContext] = [
            A2AContext(cfg, r, world_size, device=device, payload=payload, schedule=schedule, combine=combine,
                       timeout_ms=timeout_ms, connect=False)
            for r in range(world_size)
        ]
        A2AContext.attach_local(self.ctxs)

    def _calls(self, rank_datas: Sequence):
        """One empty call per rank; a rank without data would pass for one that has no tokens."""
        if len(rank_datas) < self.world_size:
            raise _lib.A2AError(_lib.A2A_ERR_STATE, f"{self.world_size} ranks, but data for {len(rank_datas)}")
        return (_lib.Call * self.world_size)()

    def _step(self, phase: str, calls=None) -> None:
        handles = (C.c_void_p * self.world_size)(*[c._h.value for c in self.ctxs])
        _lib.check(self.ctxs[0].lib.a2a_group_step(handles, _lib.GROUP_PHASE[phase], calls, _lib.current_stream()))

    def _quick(self, rank_datas, phases, pipelined):
        """The phases of a whole call without the interpreter in between, or None where something needs a second look."""
        if len(self.ctxs) != self.world_size:
            return None
        out = _lib.host().group_forward(self.ctxs, rank_datas, phases, pipelined)
        return out if type(out) is not int else _lib.check(out)

    def _send(self, rank_datas: Sequence) -> None:
        """route + dispatch_send on every rank, in one launch."""
        calls = self._calls(rank_datas)
        for call, c, rd in zip(calls, self.ctxs, rank_datas):
            assert rd.indices.dtype == torch.int32 and rd.indices.is_contiguous() and rd.indices.is_cuda
            assert rd.x.dtype == self.cfg.in_dtype and rd.x.is_contiguous() and rd.x.is_cuda
            call.x, call.topk_idx, call.num_tokens = rd.x.data_ptr(), rd.indices.data_ptr(), rd.indices.shape[0]
        self._step("send", calls)
        for c, rd in zip(self.ctxs, rank_datas):
            c._num_tokens, c._keep = rd.indices.shape[0], [rd.indices, rd.x]

    def _combine(self, rank_datas: Sequence) -> List[torch.Tensor]:
        calls, ys = (_lib.Call * self.world_size)(), []
        for call, c, rd in zip(calls, self.ctxs, rank_datas):
            assert rd.weights.dtype == torch.float32 and rd.weights.is_contiguous() and rd.weights.is_cuda
            ys.append(torch.empty(c._num_tokens, self.cfg.hidden_dim, dtype=self.cfg.out_dtype, device=c.device))
            call.topk_weights, call.y = rd.weights.data_ptr(), ys[-1].data_ptr()
            c._keep.append(rd.weights)
        self._step("combine", calls)
        return ys

    def dispatch(self, rank_datas: Sequence) -> None:
        """route + dispatch on every rank (rank_datas hold device tensors)."""
        self._send(rank_datas)
        self._step("recv")

    def forward_phases(self, rank_datas: Sequence) -> List[torch.Tensor]:
        """The four public phases, one after the other and handed on from one to the next: a program with expert kernels of its
        own calls them one by one, in which each launch also raises and awaits flags."""
        ys = self._quick(rank_datas, _PHASES, False)
        if ys is not None:
            return ys
        self.dispatch(rank_datas)
        self._step("expert")
        return self._combine(rank_datas)

    def forward(self, rank_datas: Sequence) -> List[torch.Tensor]:
        """The kernels a2a_forward launches (send, recv+expert fused, combine), in lock-step."""
        ys = self._quick(rank_datas, _FUSED, False)
        if ys is not None:
            return ys
        self._send(rank_datas)
        self._step("recv_expert")
        return self._combine(rank_datas)

    def forward_pipelined(self, rank_datas: Sequence) -> List[torch.Tensor]:
        """The roles of the pipelined one-launch kernel as three launches, in lock-step and in the forms of ranks on one GPU:
        every rank's routers, then every rank's expert blocks, then every rank's combine.  Nothing of the caller's
        runs in between, so the second writes the outputs too where they do not lie over inputs (csrc/a2a_near.cuh)."""
        ys = self._quick(rank_datas, _ROLES, True)
        if ys is not None:
            return ys
        calls, ys = self._whole_calls(rank_datas)
        self._step("pipe_send", calls)
        self._begun(rank_datas, ys)
        self._step("pipe_expert")
        self._step("pipe_combine")
        return ys

    def forward_one_launch(self, rank_datas: Sequence) -> List[torch.Tensor]:
        """The pipelined one-launch kernel of every rank, as a group with a GPU per rank runs it, in one cooperative
        launch: every block of every rank is running, so the waits of one rank for another are safe here."""
        calls, ys = self._whole_calls(rank_datas)
        handles = (C.c_void_p * self.world_size)(*[c._h.value for c in self.ctxs])
        _lib.check(self.ctxs[0].lib.a2a_group_forward(handles, calls, _lib.current_stream()))
        self._begun(rank_datas, ys)
        return ys

    def _whole_calls(self, rank_datas: Sequence):
        calls, ys = self._calls(rank_datas), []
        for call, c, rd in zip(calls, self.ctxs, rank_datas):
            n = c._check_inputs(rd.x, rd.indices, rd.weights, None, on_device=True)
            ys.append(torch.empty(n, self.cfg.hidden_dim, dtype=self.cfg.out_dtype, device=c.device))
            call.x, call.topk_idx, call.topk_weights = rd.x.data_ptr(), rd.indices.data_ptr(), rd.weights.data_ptr()
            call.y, call.num_tokens = ys[-1].data_ptr(), n
        return calls, ys

    def _begun(self, rank_datas: Sequence, ys) -> None:
        for c, rd, y in zip(self.ctxs, rank_datas, ys):
            c._num_tokens, c._y, c._keep = y.shape[0], y, [rd.x, rd.indices, rd.weights, y]

    def check(self) -> None:
        for c in self.ctxs:
            c.check()

    def close(self) -> None:
        torch.cuda.synchronize()
        for c in self.ctxs:
            c.close()
