"""The 256-bin byte histogram (the reference repository's second task, pmpp_v2/histogram_py).

CPU: the checker (the reference's own ``torch.bincount`` call) against an operator-free restatement,
hand-written answers and the committed fixture.  GPU: the kernel through the C ABI against the
checker, bit-exact (integer work), on the task's own test and benchmark sizes and contentions, on
ragged sizes, unaligned starts and degenerate inputs."""
import ctypes as C
import os

import numpy as np
import pytest
import torch

from oracle import histogram_oracle as HO

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "histogram.npz")


def test_checker_known_answers():
    data = torch.tensor([0, 0, 255, 7, 7, 7, 200], dtype=torch.uint8)
    want = np.zeros(256, dtype=np.int64)
    want[0], want[255], want[7], want[200] = 2, 1, 3, 1
    assert np.array_equal(HO.ref_histogram(data).numpy(), want)
    assert np.array_equal(HO.count_bytes(data), want)
    empty = torch.zeros(0, dtype=torch.uint8)
    assert int(HO.ref_histogram(empty).sum()) == 0 and HO.ref_histogram(empty).shape == (256,)


@pytest.mark.parametrize("size,seed,contention", HO.REFERENCE_TESTS)
def test_checker_agrees_with_its_restatement(size, seed, contention):
    data, out = HO.generate_input(size, contention, seed)
    h = HO.ref_histogram(data)
    assert h.dtype == torch.int64 and int(h.sum()) == size
    assert np.array_equal(h.numpy(), HO.count_bytes(data))
    # the generator's "evil" value really dominates at high contention
    if contention >= 90:
        assert int(h.max()) > 0.85 * size
    assert out.shape == (256,) and out.dtype == torch.int64


def test_checker_reproduces_the_committed_fixture():
    z = np.load(GOLDEN)
    for i in range(int(z["cases"])):
        size, seed, contention = (int(v) for v in z[f"c{i}_spec"])
        data, _ = HO.generate_input(size, contention, seed)
        assert np.array_equal(data.numpy(), z[f"c{i}_data"])
        assert np.array_equal(HO.ref_histogram(data).numpy(), z[f"c{i}_hist"])


def _run(data_gpu):
    from gpu_mode_kernels_b200.histogram import custom_kernel

    out = torch.full((256,), -5, dtype=torch.int64, device=data_gpu.device)  # stale content must be overwritten
    got = custom_kernel((data_gpu, out))
    torch.cuda.synchronize()
    assert got is out
    return out.cpu()


@pytest.mark.gpu
@pytest.mark.parametrize("size,seed,contention", HO.REFERENCE_TESTS + HO.REFERENCE_BENCHMARKS)
def test_reference_task_cases(size, seed, contention):
    data, _ = HO.generate_input(size, contention, seed)
    assert torch.equal(_run(data.to("cuda:0")), HO.ref_histogram(data))


@pytest.mark.gpu
def test_committed_fixture_on_the_gpu():
    z = np.load(GOLDEN)
    for i in range(int(z["cases"])):
        data = torch.from_numpy(z[f"c{i}_data"].copy())
        assert np.array_equal(_run(data.to("cuda:0")).numpy(), z[f"c{i}_hist"])


@pytest.mark.gpu
@pytest.mark.parametrize("size", [0, 1, 15, 16, 17, 31, 33, 4095, 4097, 1 << 20])
@pytest.mark.parametrize("offset", [0, 1, 7])
def test_ragged_sizes_and_unaligned_starts(size, offset):
    g = torch.Generator().manual_seed(size * 8 + offset)
    base = torch.randint(0, 256, (size + offset,), dtype=torch.uint8, generator=g)
    data = base.to("cuda:0")[offset:]  # starts `offset` bytes past an aligned allocation
    assert torch.equal(_run(data.contiguous() if offset == 0 else data), HO.ref_histogram(base[offset:]))


@pytest.mark.gpu
@pytest.mark.parametrize("size", [
    (1 << 18) - 1, 1 << 18, (1 << 18) + 1,
    148 * 512 * 16 + 5,                             # a vector per thread of a block per SM; a third of the blocks count
    148 * 512 * 4 * 16, 148 * 512 * 4 * 16 + 21,    # one round of that grid; one vector and five bytes more
    (1 << 25) - 1, 1 << 25, (1 << 25) + 31,
])
@pytest.mark.parametrize("offset,frequent", [(0, 0.0), (9, 0.9)])
def test_either_side_of_the_launch_rules(size, offset, frequent):
    """One cluster / two launches, one block / two blocks per SM, one vector more than a round of the grid takes;
    twice into the same output, the second time on other data."""
    g = torch.Generator().manual_seed(size + offset)
    out = torch.full((256,), 3, dtype=torch.int64, device="cuda:0")
    from gpu_mode_kernels_b200.histogram import histogram256

    for value in (0, 255):
        base = torch.randint(0, 256, (size + offset,), dtype=torch.uint8, generator=g)
        base[torch.rand(base.numel(), generator=g) < frequent] = value
        histogram256(base.to("cuda:0")[offset:], out)
        assert torch.equal(out.cpu(), HO.ref_histogram(base[offset:]))


@pytest.mark.gpu
def test_degenerate_inputs_and_two_calls_in_a_row():
    same = torch.full((1 << 22,), 200, dtype=torch.uint8)
    h = _run(same.to("cuda:0"))
    assert int(h[200]) == 1 << 22 and int(h.sum()) == 1 << 22
    ramp = (torch.arange(1 << 16) % 256).to(torch.uint8)
    assert torch.equal(_run(ramp.to("cuda:0")), torch.full((256,), 256, dtype=torch.int64))


@pytest.mark.gpu
def test_arguments_are_checked():
    from gpu_mode_kernels_b200 import _lib
    from gpu_mode_kernels_b200.histogram import histogram256

    data = torch.zeros(64, dtype=torch.uint8, device="cuda:0")
    out = torch.zeros(256, dtype=torch.int64, device="cuda:0")
    for bad in ((data.to(torch.int32), out), (data, out.to(torch.int32)), (data, out[:100]), (data.cpu(), out)):
        with pytest.raises(_lib.A2AError):
            histogram256(*bad)
    lib = _lib.load()
    assert lib.a2a_histogram256(None, 16, C.c_void_p(out.data_ptr()), None) == _lib.A2A_ERR_CONFIG
    assert lib.a2a_histogram256(C.c_void_p(data.data_ptr()), 16, None, None) == _lib.A2A_ERR_CONFIG


@pytest.mark.gpu
@pytest.mark.parametrize("size", [2048, 200000, 148 * 4096, 148 * 4096 + 1, 5 << 20])
def test_calls_that_overlap_read_what_the_stream_wrote(size):
    """A call may be resident while the launch before it still writes its data -- a copy, or the call before, whose counts are
    the next call's bytes; and while the call before it still adds to the same output."""
    from gpu_mode_kernels_b200.histogram import histogram256

    g = torch.Generator().manual_seed(size)
    sets = [torch.randint(0, 256, (size,), dtype=torch.uint8, generator=g) for _ in range(3)]
    want = [HO.ref_histogram(s) for s in sets]
    want_of_counts = [HO.ref_histogram(w.view(torch.uint8)) for w in want]
    on_gpu, data = [s.to("cuda:0") for s in sets], torch.empty(size, dtype=torch.uint8, device="cuda:0")
    out = torch.empty(256, dtype=torch.int64, device="cuda:0")
    got = []
    for i in range(60):
        data.copy_(on_gpu[i % 3])
        histogram256(data, out)
        chained = histogram256(out.view(torch.uint8), torch.empty_like(out))
        got.append((out.clone(), chained))
        histogram256(on_gpu[(i + 1) % 3], out)
    torch.cuda.synchronize()
    for i, (counts, chained) in enumerate(got):
        assert torch.equal(counts.cpu(), want[i % 3]) and torch.equal(chained.cpu(), want_of_counts[i % 3])
