"""The 3D trace's charge and current: cells of many records, and few records on many nodes."""

from __future__ import annotations

import numpy as np
import pytest

from tests.golden.cases import copy_args
from tests.gpu_util import load_golden, to_device, to_host

pytestmark = pytest.mark.gpu

CHARGE, CURRENT = 37, 39


@pytest.mark.parametrize("copies", [1, 2, 33, 400])
@pytest.mark.parametrize("name", ["trace3d_i0_r0_m1_b0_j1", "trace3d_i1_r1_m0_b1_j1"])
def test_current_of_many_copies(name, copies):
    """Cells whose records fill part of a warp to many warps: copies of a case's trajectories
    leave as many times its charge and current (1e-12 of the largest)."""
    from beamtracer_b200.kernels import KERNELS

    args, out = load_golden(name)
    n = args[1].shape[1]
    big = copy_args(args)
    big[0] = np.arange(n * copies, dtype=np.int64)
    for i in (1, 2):
        big[i] = np.tile(args[i], (1, copies))
    for i in (3, 4, 5, 6, 7):
        big[i] = np.tile(args[i], copies)
    big[33] = np.full(n * copies, -1, dtype=np.int64)  # no kept paths
    big[31] = np.zeros((n * copies,) + args[31].shape[1:])
    big[32] = np.zeros((n * copies, args[32].shape[1]), dtype=np.int64)
    device = to_device(big)
    KERNELS["trace_trajectories_3d"](*device)
    got = to_host(device)
    for i in (CHARGE, CURRENT):
        want = copies * out[i].sum(axis=0)
        assert float(np.abs(got[i].sum(axis=0) - want).max()) <= 1e-12 * float(np.abs(want).max())


def test_scratch_of_few_trajectories_on_many_nodes():
    """Three trajectories with the current on 129^3 nodes: straight lines, whose charge is their
    time and whose current their displacement (1e-12), in a few words of scratch a node (one
    slab of the pool and 32 bytes a node at most; a record a node would be 192)."""
    import threading

    import torch

    from beamtracer_b200.kernels import KERNELS

    N, h, n = 129, 1e-3, 3
    up, nodes = h * (N - 1), 129**3

    def zeros(*shape):
        return torch.zeros(shape, dtype=torch.float64, device="cuda")

    def ints(a):
        return torch.as_tensor(np.asarray(a, dtype=np.int64)).cuda()

    def reals(a):
        return torch.as_tensor(np.asarray(a, dtype=float)).cuda()

    x = [[1e-6] * n, [0.3 * up, 0.5 * up, 0.7 * up], [0.5 * up, 0.2 * up, 0.4 * up]]
    v = [[3e5] * n, [1e4, -2e4, 0.0], [0.0, 1e4, 3e4]]
    args = [ints(range(n)), reals(x), reals(v), reals([9.58e7] * n), reals([1.0] * n), ints([0] * n),
            ints([-1] * n), ints([-1] * n), zeros((N + 1) * N * N), zeros((N + 1) * N * N),
            zeros((N + 1) * N * N), ints([[N, N, N, 0, 0, 0, 0, 0]]),
            reals([[0.0, 0.0, 0.0, h, 0.0, 0.0, 0.0, up, up, up]]), zeros(1), 0, 0.0, 0.0, 0.0, h,
            up, up, up, 0, 0, 0, 0.5, 10_000,
            torch.full(((N - 1) ** 3,), -1, dtype=torch.int64, device="cuda"), ints([-1]), 1,
            reals([1e9]), zeros(n, 1, 1, 8), ints(np.zeros((n, 1))), ints([-1] * n), zeros(1, 1, 3),
            ints([0]), 1, zeros(1, nodes), 1, zeros(1, 3 * nodes), 0.0]  # fmt: skip
    used = []

    def run():  # a thread has a context, and so scratch, of its own
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        KERNELS["trace_trajectories_3d"](*args)
        torch.cuda.synchronize()
        used.append(before - torch.cuda.mem_get_info()[0])

    thread = threading.Thread(target=run)
    thread.start()
    thread.join()
    assert used and used[0] <= (128 << 20) + (16 << 20) + 32 * nodes
    moved = args[1].cpu().numpy() - np.array(x)
    time = moved[0] / 3e5
    assert args[6].tolist() == [0] * n
    assert float(args[CHARGE].sum()) == pytest.approx(time.sum(), rel=1e-12)
    np.testing.assert_allclose(args[CURRENT].reshape(3, -1).sum(1).cpu().numpy(), moved.sum(1),
                               rtol=0, atol=1e-12 * np.abs(moved).max())  # fmt: skip


def test_current_of_a_long_window():
    """A window whose records are fewer than 2^32, though the shares of their current are more:
    the outputs of the default window."""
    import threading

    import torch

    from beamtracer_b200.kernels import KERNELS

    if torch.cuda.mem_get_info()[0] < 100 << 30:
        pytest.skip("the window's records take 62 GB")
    args, _ = load_golden("trace3d_i0_r0_m1_b0_j1")
    n = args[1].shape[1]
    window = 2**32 // (24 * n) + 1
    results = []

    def run():  # in a thread: its context gives the scratch back
        for steps in (0, window):
            device = to_device(args)
            KERNELS["trace_trajectories_3d"](*device, window=steps)
            results.append(to_host(device))

    thread = threading.Thread(target=run)
    thread.start()
    thread.join()
    assert len(results) == 2
    for short, long in zip(*results, strict=True):
        if isinstance(short, np.ndarray):
            scale = max(float(np.abs(short).max()), 1e-300) if short.size else 1.0
            np.testing.assert_allclose(long, short, rtol=0, atol=1e-13 * scale)
