"""Steps captured into a CUDA graph after one step outside it: nothing is
allocated, replays of an even number of launches advance the state, and what a
capture only recorded (tile flags) is not taken for built."""

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


class _Captured:
    def __init__(self, size):
        import torch

        from fpie_gb300 import backend

        self.torch = torch
        self.stream = torch.cuda.Stream()
        self.s = backend.GridSolver(8, 8)
        self.s.set_stream(self.stream.cuda_stream)
        self.img = torch.empty((*size, 3), dtype=torch.uint8, device="cuda")
        self.err = torch.empty(3, dtype=torch.float32, device="cuda")

    def reset(self, *arrays):
        self.dev = [self.torch.from_numpy(a).cuda() for a in arrays]
        self.torch.cuda.synchronize()
        self.s.reset_tensors(*self.dev)

    def step(self, k):
        self.s.step_tensors(k, self.img, self.err)
        self.s.sync()

    def capture(self, k):
        graph = self.torch.cuda.CUDAGraph()
        with self.torch.cuda.graph(graph, stream=self.stream):
            self.s.step_tensors(k, self.img, self.err)
        return graph

    def replay(self, graph):
        with self.torch.cuda.stream(self.stream):
            graph.replay()
        self.torch.cuda.synchronize()
        return self.img.cpu().numpy()


@pytest.mark.parametrize("size,warm,k", [
    ((38, 38), 3, 3), ((38, 38), 3, 20), ((194, 194), 8, 8), ((194, 194), 8, 20), ((194, 194), 50, 50),
    ((194, 194), 50, 128), ((333, 517), 100, 64), ((802, 802), 16, 32), ((902, 902), 150, 20),
    ((902, 902), 150, 8), ((902, 902), 10, 120), ((1900, 1810), 20, 20), ((1900, 1810), 70, 30)])
def test_replays_after_one_step(size, warm, k):
    arrays = _inputs(*size, 4)
    c = _Captured(size)
    c.reset(*arrays)
    c.step(warm)
    graph = c.capture(k)
    o = cjacobi.CGrid(*arrays)
    o.sweep(warm)
    for replay in range(3):
        got = c.replay(graph)
        if replay == 0 or -(-k // 16) % 2 == 0:  # an odd number of launches repeats itself
            o.sweep(k)
        np.testing.assert_array_equal(got, o.image())


@pytest.mark.parametrize("size", [(194, 194), (902, 902), (1900, 1810)])
def test_a_capture_without_a_replay_leaves_no_trace(size):
    """A new mask activates other tiles; the step after the capture needs its
    own flags although the capture recorded the kernel that makes them."""
    first = _inputs(*size, 5)
    small = first[0].copy()
    small[20:] = 0
    c = _Captured(size)
    c.reset(small, first[1], (first[2] * small[..., None]).astype(np.float32))
    for _ in range(2):
        c.step(20)
    second = _inputs(*size, 6)
    c.reset(*second)
    graph = c.capture(20)
    o = cjacobi.CGrid(*second)
    for k in (12, 20, 7):
        c.step(k)
        o.sweep(k)
        np.testing.assert_array_equal(c.s.state(), o.x)
    del graph


@pytest.mark.parametrize("order", ["jacobi", "red_black"])
def test_equation_systems(order):
    import torch

    from fpie_gb300 import backend

    rng = np.random.default_rng(7)
    src, tgt = (torch.from_numpy(rng.integers(0, 256, (150, 170, 3), dtype=np.uint8)).cuda()
                for _ in range(2))
    mask = torch.full((150, 170), 255, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    s, ref = (backend.EquSolver(256, order=order) for _ in range(2))
    s.set_stream(stream.cuda_stream)
    n = s.reset_images(src, mask, tgt, (0, 0), (0, 0), "max")[0]
    ref.reset_images(src, mask, tgt, (0, 0), (0, 0), "max")
    x = torch.empty((n, 3), dtype=torch.uint8, device="cuda")
    s.step_tensors(12, x)
    s.sync()
    ref.step(12)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        s.step_tensors(32, x)
    for _ in range(3):
        with torch.cuda.stream(stream):
            graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(x.cpu().numpy(), ref.step(32)[0])
