"""CPU checks of the host side of a group on one GPU."""
from types import SimpleNamespace

import pytest
import torch

import gpu_mode_kernels_b200 as pkg
from gpu_mode_kernels_b200 import _lib
from gpu_mode_kernels_b200.local_world import LocalWorld


@pytest.mark.parametrize("entry", ["dispatch", "forward_phases", "forward", "forward_pipelined"])
@pytest.mark.parametrize("given", [0, 1, 2])
def test_data_for_every_rank_is_asked_for(entry, given, monkeypatch):
    monkeypatch.setattr(_lib, "current_stream", lambda: 0)
    cfg, rd, _, _ = pkg.generate_input(6, 2, 64, 4, seed=1, rank=0, world_size=3)
    tensors = [SimpleNamespace(is_cuda=True, is_contiguous=lambda: True, dtype=t.dtype, shape=t.shape, data_ptr=lambda: 0)
               for t in (rd.x, rd.indices, rd.weights)]
    data = SimpleNamespace(x=tensors[0], indices=tensors[1], weights=tensors[2])
    world, launched = object.__new__(LocalWorld), []
    lib = SimpleNamespace(a2a_group_step=lambda *a: launched.append(a) or 0)
    world.cfg, world.world_size = cfg, 3
    world.ctxs = [SimpleNamespace(_h=SimpleNamespace(value=1), lib=lib, device=torch.device("cpu"), _num_tokens=4, _keep=[],
                                  _check_inputs=lambda *a, **k: 4) for _ in range(3)]
    with pytest.raises(_lib.A2AError) as refused:
        getattr(world, entry)([data] * given)
    assert refused.value.code == _lib.A2A_ERR_STATE and not launched
