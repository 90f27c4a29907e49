"""Steps that store the picture straight into the target image.

The composed target must equal, byte for byte, the one that numpy composes
from step()'s result, for the targets that native code stores into and for
those that it leaves to numpy (other strides, negative or wrong coordinates).
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _images(h, w, seed, fill=0.6):
    rng = np.random.default_rng(seed)
    src = rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
    tgt = rng.integers(0, 256, (h + 9, w + 13, 3), dtype=np.uint8)
    mask = np.where(rng.random((h, w)) < fill, 255, 0).astype(np.uint8)
    mask[h // 2, w // 2] = 255
    return src, mask, tgt


SIZES = [(3, 3), (5, 64), (61, 47), (180, 301)]


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("device_prep", [True, False])
def test_grid_target_equals_numpy(size, device_prep):
    from fpie_gb300.process import GridProcessor

    src, mask, tgt = _images(*size, seed=size[1])
    a, b = (GridProcessor("max", device_prep=device_prep) for _ in range(2))
    for p in (a, b):
        p.reset(src, mask, tgt, (0, 0), (4, 7))
    want = tgt.copy()
    for k in (1, 0, 30):
        out, err = a.step(k)
        img, err_b = b.core.step(k)
        want[b.x0:b.x1, b.y0:b.y1] = img
        assert out is a.tgt
        np.testing.assert_array_equal(out, want)
        np.testing.assert_array_equal(err, err_b)
    # A view with other strides: numpy stores the picture.
    wide = np.zeros((tgt.shape[0], 2 * tgt.shape[1], 3), np.uint8)
    a.tgt = wide[:, ::2]
    a.tgt[:] = want
    img, _ = b.core.step(5)
    want[b.x0:b.x1, b.y0:b.y1] = img
    np.testing.assert_array_equal(a.step(5)[0], want)
    assert not wide[:, 1::2].any()


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("backend", ["gb300", "gb300-rb"])
@pytest.mark.parametrize("device_prep", [True, False])
def test_equ_target_equals_numpy(size, backend, device_prep):
    from fpie_gb300.process import EquProcessor

    src, mask, tgt = _images(*size, seed=size[0])
    a, b = (EquProcessor("max", backend=backend, device_prep=device_prep) for _ in range(2))
    for p in (a, b):
        p.reset(src, mask, tgt, (0, 0), (4, 7))
        assert all(i.dtype == np.int64 for i in p.tgt_index)
    want = tgt.copy()
    for k in (1, 0, 30):
        out, err = a.step(k)
        x, err_b = b.core.step(k)
        want[b.tgt_index] = x[1:]
        np.testing.assert_array_equal(out, want)
        np.testing.assert_array_equal(err, err_b)
    # Coordinates from the end of the image, as numpy reads them.
    rows, cols = b.tgt_index
    a.tgt_index = (rows - tgt.shape[0], cols)
    x, _ = b.core.step(5)
    want[b.tgt_index] = x[1:]
    np.testing.assert_array_equal(a.step(5)[0], want)
    # A coordinate outside: refused, the target keeps its bytes.
    bad = cols.copy()
    bad[-1] = tgt.shape[1]
    a.tgt_index = (rows, bad)
    with pytest.raises(IndexError):
        a.step(5)
    np.testing.assert_array_equal(a.tgt, want)
    a.tgt_index = (rows, cols)
    x, _ = b.core.step(5)
    want[b.tgt_index] = x[1:]
    np.testing.assert_array_equal(a.step(0)[0], want)


def test_index_arrays_across_systems_of_other_sizes():
    from fpie_gb300.backend import EquSolver

    s = EquSolver()
    for size in [(40, 50), (180, 301), (9, 9), (61, 47)]:
        src, mask, tgt = _images(*size, seed=7)
        n, box, (rows, cols) = s.reset_images(src, mask, tgt, (0, 0), (4, 7), "src")
        on = mask >= 128
        on[0] = on[-1] = on[:, 0] = on[:, -1] = False
        r, c = np.nonzero(on)
        assert n == r.size + 1
        np.testing.assert_array_equal(rows, r + 4)
        np.testing.assert_array_equal(cols, c + 7)


def test_a_step_that_gave_up_waiting_leaves_the_target():
    from fpie_gb300 import _abi
    from fpie_gb300.process import GridProcessor

    src, mask, tgt = _images(300, 300, 8, fill=0.9)
    p = GridProcessor("max", device_prep=True)
    p.core.set_kernel("p12w8x128k16r")
    p.core.set_spin_limit(0)
    p.reset(src, mask, tgt, (0, 0), (4, 7))
    with pytest.raises(_abi.FpieTimeoutError):
        p.step(64)
    np.testing.assert_array_equal(p.tgt, tgt)
