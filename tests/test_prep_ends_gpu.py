"""The GPU-side reset where the crop reaches the first and last bytes of images
that start and end at every alignment: equal to the host construction."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(3, 3), (3, 4), (4, 5), (5, 6), (3, 7), (6, 8), (7, 129), (33, 3)])
@pytest.mark.parametrize("off", [0, 1, 2, 3])
def test_crops_as_large_as_the_images(size, off):
    import torch

    from fpie_gb300 import backend, prep

    rng = np.random.default_rng(size[0] * 131 + size[1])
    src, tgt = (rng.integers(0, 256, (*size, 3), np.uint8) for _ in range(2))
    mask = np.full(size, 255, np.uint8)

    def device(a, shift):
        buf = torch.empty(shift + a.size, dtype=torch.uint8, device="cuda")
        t = buf[shift:].view(a.shape)
        t.copy_(torch.from_numpy(a))
        return t

    mc, t, g, crop = prep.grid_inputs(src, mask, tgt, (0, 0), (0, 0), "max")
    assert (crop.x0, crop.x1, crop.y0, crop.y1) == (0, size[0], 0, size[1])
    s = backend.GridSolver(8, 8)
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    s.reset_images(device(src, off), torch.from_numpy(mask).cuda(), device(tgt, 3 - off), (0, 0),
                   (0, 0), "max")
    gm, gg = s.inputs()
    np.testing.assert_array_equal(gm, mc)
    np.testing.assert_array_equal(gg, g)
    np.testing.assert_array_equal(s.state(), t)
