"""The compiled part of the Python layer belongs to one Python and one torch; without it the same calls run."""
import os
import sysconfig

import pytest
import torch

import gpu_mode_kernels_b200 as pkg
from gpu_mode_kernels_b200 import _lib, all2all, build, histogram
from gpu_mode_kernels_b200.local_world import LocalWorld

DEV = "cuda:0"


def test_the_file_is_this_pythons_and_this_torchs(monkeypatch, tmp_path):
    assert _lib.host() is not _lib.Interpreted
    monkeypatch.setattr(build, "PKG_DIR", str(tmp_path))
    monkeypatch.setattr(build, "LIB_PATH", str(tmp_path / "liba2a.so"))
    here = build.host_path()
    assert os.path.basename(here) == f"_host.{sysconfig.get_config_var('SOABI')}.torch-{torch.__version__}.so"
    assert build.needs_build()
    for path in (build.LIB_PATH, here):  # newer than every source
        open(path, "w").close()
    assert not build.needs_build()
    monkeypatch.setattr(torch, "__version__", "0.0.1+other")
    assert build.host_path() != here and build.needs_build()


@pytest.mark.parametrize("there", ["nothing", "no library"])
def test_without_it_calls_go_through_python(monkeypatch, tmp_path, there):
    path = os.path.join(tmp_path, "_host.other.so")
    if there == "no library":
        with open(path, "w") as f:
            f.write("text")
    monkeypatch.setattr(_lib, "host_path", lambda: path)
    monkeypatch.setattr(_lib, "_host", None)
    with pytest.warns(RuntimeWarning, match="build.py"):
        assert _lib.host() is _lib.Interpreted
    assert _lib.host().Rank(1, 0, 8, 64, torch.bfloat16).forward(None, None, None, True) is None


@pytest.mark.gpu
def test_the_same_bits_without_it(monkeypatch):
    def everything():
        cfg, rd, _, _ = pkg.generate_input(8, 3, 264, 9, seed=3, rank=0, world_size=1, device=DEV)
        got = [all2all.custom_kernel((cfg, rd, 0, 1))]
        all2all.release_contexts(barrier=False)
        rds = [pkg.generate_input(8, 2, 264, 6, seed=4, rank=r, world_size=2)[1].to(DEV) for r in range(2)]
        for schedule, payload, combine in (("pipelined", "dedup", "push"), ("phased", "direct", "pull")):
            world = LocalWorld(pkg.MoEConfig(8, 2, 264, 6), 2, payload=payload, schedule=schedule, combine=combine)
            got += (world.forward_pipelined if schedule == "pipelined" else world.forward_phases)(rds)
            assert [c._num_tokens for c in world.ctxs] == [6, 6]
            world.check()
            world.close()
        data = torch.arange(5000, device=DEV).to(torch.uint8)
        return got + [histogram.custom_kernel((data, torch.empty(256, dtype=torch.int64, device=DEV)))]

    assert _lib.host() is not _lib.Interpreted
    want = everything()
    monkeypatch.setattr(_lib, "_host", _lib.Interpreted)
    assert all(torch.equal(a, b) for a, b in zip(everything(), want))
