"""Reset and finish kernels at the edges of their vector accesses.

The GPU-side reset against the host construction (the same integers, so equal)
for widths around its 16-pixel and 4-column groups, mask channels, and device
images whose first byte has every alignment; the finish kernel's image (equal
to the oracle's) and residual sums for widths around its 4-column groups and
128-column warps, into tensors of every alignment.  The sums are float32
roundings of sums that are exact to far better than 1e-7, against the oracle's
float64 sum: rtol 1e-6.
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle import np_jacobi

pytestmark = pytest.mark.gpu


def _unaligned(a, off):
    """`a` on the GPU with its first byte `off` bytes into an allocation."""
    import torch

    buf = torch.empty(a.size + 64, dtype=torch.uint8, device="cuda")
    t = buf[off:off + a.size].view(a.shape)
    t.copy_(torch.from_numpy(a))
    return t


@pytest.mark.parametrize("gradient", ["src", "avg", "max"])
@pytest.mark.parametrize("size", [(3, 3), (5, 9), (17, 15), (16, 16), (9, 33), (40, 131), (130, 21)])
def test_reset_images_any_width_and_alignment(size, gradient):
    import torch

    from fpie_gb300 import backend, prep

    rng = np.random.default_rng(size[0] * 131 + size[1])
    h, w = size
    s = backend.GridSolver(8, 8)
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    for channels, off in ((1, 0), (1, 3), (3, 0), (3, 5)):
        shape = (h, w) if channels == 1 else (h, w, 3)
        mask = rng.integers(0, 256, shape, np.uint8)
        mask[h // 2, w // 2] = 255
        src = rng.integers(0, 256, (h + 3, w + 2, 3), np.uint8)
        tgt = rng.integers(0, 256, (h + 1, w + 4, 3), np.uint8)
        mc, t, g, crop = prep.grid_inputs(src, mask, tgt, (2, 1), (1, 3), gradient)
        box = s.reset_images(_unaligned(src, off), _unaligned(mask, off), _unaligned(tgt, off + 1),
                             (2, 1), (1, 3), gradient)
        assert box == (crop.x0, crop.x1, crop.y0, crop.y1)
        gm, gg = s.inputs()
        np.testing.assert_array_equal(gm, mc)
        np.testing.assert_array_equal(gg, g)
        np.testing.assert_array_equal(s.state(), t)


def test_reset_images_larger_than_one_pass():
    """More groups than the device has threads: strided loops, several rows
    per thread."""
    import torch

    from fpie_gb300 import backend, prep

    rng = np.random.default_rng(3)
    h, w = 2501, 2063
    mask = rng.integers(0, 256, (h, w), np.uint8)
    src, tgt = (rng.integers(0, 256, (h, w, 3), np.uint8) for _ in range(2))
    mc, t, g, _ = prep.grid_inputs(src, mask, tgt, (0, 0), (0, 0), "max")
    s = backend.GridSolver(8, 8)
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    s.reset_images(*(torch.from_numpy(a).cuda() for a in (src, mask, tgt)), (0, 0), (0, 0), "max")
    gm, gg = s.inputs()
    np.testing.assert_array_equal(gm, mc)
    np.testing.assert_array_equal(gg, g)
    img, err = s.step(0)
    o = np_jacobi.GridJacobi(mc, t, g)
    np.testing.assert_array_equal(img, o.image())
    np.testing.assert_allclose(err, o.err64(), rtol=1e-6)


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 7, 127, 128, 129, 130, 131, 255, 257, 385])
def test_finish_any_width_and_alignment(m):
    import torch

    from fpie_gb300 import backend

    rng = np.random.default_rng(m)
    n = 7
    mask = (rng.random((n, m)) < 0.8).astype(np.int32)
    tgt = rng.uniform(-50, 300, (n, m, 3)).astype(np.float32)
    grad = rng.uniform(-30, 30, (n, m, 3)).astype(np.float32)
    s = backend.GridSolver(8, 8)
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    s.reset(mask.size, mask, tgt, grad)
    o = np_jacobi.GridJacobi(mask, tgt, grad)
    for off in range(4):
        buf = torch.full((n * m * 3 + 16,), 77, dtype=torch.uint8, device="cuda")
        img = buf[off:off + n * m * 3].view(n, m, 3)
        err = torch.empty(3, dtype=torch.float32, device="cuda")
        s.step_tensors(3, img, err)
        o.sweep(3)
        np.testing.assert_array_equal(img.cpu().numpy(), o.image())
        assert (buf[:off] == 77).all() and (buf[off + n * m * 3:] == 77).all()
        np.testing.assert_allclose(err.cpu().numpy(), o.err64(), rtol=1e-6, atol=1e-30)


def test_finish_sums_that_overflow_or_are_no_number():
    from fpie_gb300 import backend

    mask = np.ones((6, 40), np.int32)
    tgt = np.full((6, 40, 3), 3e37, np.float32)
    tgt[2, 3, 1] = np.nan
    grad = np.zeros_like(tgt)
    s = backend.GridSolver(8, 8)
    s.reset(mask.size, mask, tgt, grad)
    img, err = s.step(0)
    o = np_jacobi.GridJacobi(mask, tgt, grad)
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(err, o.err64().astype(np.float32))


@pytest.mark.parametrize("shape", [(1, 1), (5, 3), (9, 130), (40, 259), (333, 517), (1700, 2100)])
def test_norms_any_shape(shape):
    """max |r| exactly, sum |r| to 1e-14 of the float64 sum (its terms are
    float32 values, summed without FP64 rounding to 2^-52)."""
    from fpie_gb300 import backend

    n, m = shape
    rng = np.random.default_rng(n * 7 + m)
    mask = (rng.random((n, m)) < 0.8).astype(np.int32)
    tgt = rng.uniform(-50, 300, (n, m, 3)).astype(np.float32)
    grad = rng.uniform(-30, 30, (n, m, 3)).astype(np.float32)
    s = backend.GridSolver(8, 8)
    s.reset(mask.size, mask, tgt, grad)
    for _ in range(2):
        r = np.abs(_residual(mask, tgt, grad)).astype(np.float64)
        mx, sm = s.residual_norms()
        np.testing.assert_array_equal(mx, r.max((0, 1)))
        np.testing.assert_allclose(sm, [np.sum(np.sort(r[..., c].ravel())) for c in range(3)], rtol=1e-14)


def _residual(mask, x, g):
    """The oracle's float32 residual, numpy order, 0 outside the mask."""
    p = np.pad(x, ((1, 1), (1, 1), (0, 0)))
    four = np.float32(4)
    r = four * x - g
    for nb in (p[:-2, 1:-1], p[2:, 1:-1], p[1:-1, :-2], p[1:-1, 2:]):
        r = r - nb
    r[mask == 0] = 0
    return r


@pytest.mark.parametrize("scale", [1e36, 1e-42])
def test_norms_of_huge_and_tiny_residuals(scale):
    from fpie_gb300 import backend

    rng = np.random.default_rng(1)
    mask = np.ones((50, 70), np.int32)
    tgt = (rng.uniform(-1, 1, (50, 70, 3)) * scale).astype(np.float32)
    tgt[:, :35] *= np.float32(1e-20) if scale > 1 else np.float32(1)
    grad = np.zeros_like(tgt)
    s = backend.GridSolver(8, 8)
    s.reset(mask.size, mask, tgt, grad)
    r = np.abs(_residual(mask, tgt, grad)).astype(np.float64)
    mx, sm = s.residual_norms()
    np.testing.assert_array_equal(mx, r.max((0, 1)))
    np.testing.assert_allclose(sm, r.sum((0, 1)), rtol=1e-13)
