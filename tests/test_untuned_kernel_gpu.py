"""Steps too short for the autotuner: launches at first, the flow kernel once
100 (large grids: 200) sweeps have been asked for since the reset, and launches
of tall regions on grids of more than 1800x1800; the oracle's states, bit for
bit, through the change and after a new reset."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import cjacobi

pytestmark = pytest.mark.gpu


def _inputs(n, m, seed):
    rng = np.random.default_rng(seed)
    mask = (rng.random((n, m)) < 0.97).astype(np.int32)
    mask[n // 2:, m // 3:] = 1
    mask[: n // 4, : m // 4] = 0
    tgt = rng.uniform(0, 255, (n, m, 3)).astype(np.float32)
    grad = rng.uniform(-30, 30, (n, m, 3)).astype(np.float32)
    grad[mask == 0] = 0
    return mask, tgt, grad


@pytest.mark.parametrize("size,flow_from", [((845, 850), 100), ((100, 8000), 100), ((1500, 1500), 100),
                                            ((1500, 1501), 200), ((1800, 1800), 200), ((1801, 1800), 0)])
def test_kernel_by_the_sweeps_since_the_reset(size, flow_from):
    from fpie_gb300 import backend

    s = backend.GridSolver(8, 8)
    early, late = ("p16w8k16", "p16w8k12d") if flow_from else ("p22w8k16", "p22w8k16")
    for seed in (1, 2):
        mask, tgt, grad = _inputs(*size, seed)
        s.reset(mask.size, mask, tgt, grad)
        assert s.resident == ""
        o = cjacobi.CGrid(mask, tgt, grad)
        for k, kernel in ((8, early), (max(flow_from, 100) - 56, early),
                          (47, early), (48, late), (47, early), (100, late), (1, early)):
            s.step(k)
            o.sweep(k)
            assert s.kernel == kernel
            np.testing.assert_array_equal(s.state(), o.x)


@pytest.mark.parametrize("size", [(1, 1), (143, 95), (144, 96), (145, 97), (300, 210)])
def test_tall_regions_at_their_edges(size):
    from fpie_gb300 import backend

    mask, tgt, grad = _inputs(*size, 3)
    s = backend.GridSolver(8, 8)
    s.set_kernel("p22w8k16")
    s.reset(mask.size, mask, tgt, grad)
    o = cjacobi.CGrid(mask, tgt, grad)
    for k in (1, 15, 16, 64, 37):
        s.step(k)
        o.sweep(k)
        np.testing.assert_array_equal(s.state(), o.x)


@pytest.mark.parametrize("size,warm", [((902, 902), 1), ((902, 902), 3), ((194, 194), 1), ((1900, 1810), 1)])
def test_a_short_step_in_a_captured_graph(size, warm):
    """One warm-up step is enough to capture the next, although that one passes
    the number of sweeps from which the flow kernel is taken."""
    import torch

    from fpie_gb300 import backend

    mask, tgt, grad = _inputs(*size, 4)
    stream = torch.cuda.Stream()
    s = backend.GridSolver(8, 8)
    s.set_stream(stream.cuda_stream)
    dev = [torch.from_numpy(a).cuda() for a in (mask, tgt, grad)]
    img = torch.empty((*size, 3), dtype=torch.uint8, device="cuda")
    err = torch.empty(3, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    s.reset_tensors(*dev)
    for _ in range(warm):
        s.step_tensors(50, img, err)
    s.sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        s.step_tensors(50, img, err)
    with torch.cuda.stream(stream):
        graph.replay()
    torch.cuda.synchronize()
    o = cjacobi.CGrid(mask, tgt, grad)
    o.sweep(50 * (warm + 1))
    np.testing.assert_array_equal(img.cpu().numpy(), o.image())
