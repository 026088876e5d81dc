"""A deposit whose first call on a context is recorded in a CUDA graph."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("replay", [False, True])
def test_first_deposit_under_capture(replay):
    """What a first call leaves for the later ones must not depend on its having run: the
    context's next deposit, before a replay or after one, and the replay's own are right.  (The
    scratch comes from blocks that a closed context gave back, filled with what it left.)"""
    import torch

    from beamtracer_b200 import _lib

    lib = _lib.lib()
    rng = np.random.default_rng(8)
    nx, ny, n = 200, 300, 20_000
    px = torch.from_numpy(rng.uniform(0.0, 0.1 * nx, n)).cuda()
    py = torch.from_numpy(rng.uniform(0.0, 0.1 * ny, n)).cuda()
    q = torch.from_numpy(rng.normal(size=n)).cuda()

    def deposit(ctx, charge):
        _lib.check(lib.bt_deposit_trajectories_2d(
            ctx.handle, _lib.dptr(px), _lib.dptr(py), _lib.dptr(q), n, 0.0, 0.0, 0.1, 0,
            _lib.dptr(charge), nx, ny))  # fmt: skip

    def zeros():
        return torch.zeros((nx, ny), dtype=torch.float64, device="cuda")

    stream = torch.cuda.Stream()
    expected, recorded, after = zeros(), zeros(), zeros()
    torch.cuda.synchronize()
    before = _lib.Context(torch.cuda.current_device())
    deposit(before, expected)
    before.synchronize()
    before.close()
    ctx = _lib.Context(torch.cuda.current_device())
    ctx.use_stream(stream.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        deposit(ctx, recorded)
    if replay:
        with torch.cuda.stream(stream):
            graph.replay()
    deposit(ctx, after)
    ctx.synchronize()
    assert torch.equal(after, expected)
    assert torch.equal(recorded, expected if replay else zeros())
    torch.cuda.synchronize()
    del graph
    ctx.close()
