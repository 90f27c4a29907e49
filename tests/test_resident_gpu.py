"""The resident kernel (grid_res.cu) against the oracle, bit for bit.

Every shape, pinned, at the edges of its tiles: grids of exactly one tile, one
pixel more, a ragged last tile, and (from the rule, unpinned) sizes on both
sides of where the choice changes.  Inputs outside the range in which its
quartered sums are exact: values that decay through the subnormals, values
near overflow, infinities and NaNs, tiny gradients.  The tolerance is none:
states are compared for equality (NaN equal to NaN), since the kernel's
arithmetic is the oracle's.
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle import cjacobi, np_jacobi

pytestmark = pytest.mark.gpu

SHAPES = {  # name: (tile rows, tile columns)
    "p6w4x64k8r": (32, 48), "p8w4x64k8r": (48, 48), "p8w8x128k8r": (48, 112),
    "p6w4x64k16r": (16, 32), "p8w4x64k16r": (32, 32), "p8w8x64k16r": (96, 32),
    "p8w8x128k16r": (32, 96), "p12w8x128k16r": (64, 96), "p16w8x128k16r": (96, 96),
    "p16w8x128k4r": (120, 120),
}


def _inputs(n, m, seed, density=0.9):
    rng = np.random.default_rng(seed)
    mask = (rng.random((n, m)) < density).astype(np.int32)
    tgt = rng.uniform(0, 255, (n, m, 3)).astype(np.float32)
    grad = rng.uniform(-30, 30, (n, m, 3)).astype(np.float32)
    grad[mask == 0] = 0
    return mask, tgt, grad


def _compare(s, o, sweeps):
    for k in sweeps:
        img, err = s.step(k)
        o.sweep(k)
        np.testing.assert_array_equal(s.state(), o.x)
        np.testing.assert_array_equal(img, o.image())


@pytest.mark.parametrize("extra", [(0, 0), (1, 1), (37, 5)])
@pytest.mark.parametrize("kernel", sorted(SHAPES))
def test_tile_edges(kernel, extra):
    from fpie_gb300 import backend

    th, tw = SHAPES[kernel]
    for ty, tx in ((1, 1), (3, 2)):
        mask, tgt, grad = _inputs(ty * th + extra[0], tx * tw + extra[1], ty)
        mask[: th // 2, : tw // 2] = 0  # a corner without unknowns
        s = backend.GridSolver(8, 8)
        s.set_kernel(kernel)
        s.reset(mask.size, mask, tgt, grad)
        assert s.kernel == s.resident == kernel
        # one sweep, a whole exchange period, odd remainders, several periods
        _compare(s, cjacobi.CGrid(mask, tgt, grad), (1, 16, 7, 8, 100))


@pytest.mark.parametrize("kernel", sorted(SHAPES))
@pytest.mark.parametrize("less", [(0, 0), (1, 3), (0, -1), (-1, 0)])
def test_a_region_that_holds_the_grid(kernel, less):
    """Grids as large as a region (all its rows, its columns but a lane on each
    side), with masked pixels on their borders; and one row or column more."""
    from fpie_gb300 import backend

    th, tw = SHAPES[kernel]
    depth = int(kernel.split("k")[1][:-1])
    mask, tgt, grad = _inputs(th + 2 * depth - less[0], tw + 2 * depth - 8 - less[1], 9)
    mask[0, ::2] = mask[-1, 1::2] = 1
    mask[::3, 0] = mask[1::3, -1] = 1
    s = backend.GridSolver(8, 8)
    s.set_kernel(kernel)
    s.reset(mask.size, mask, tgt, grad)
    _compare(s, cjacobi.CGrid(mask, tgt, grad), (1, 16, 33, 64))


@pytest.mark.parametrize("size", [(32, 48), (33, 48), (48, 49), (160, 320), (161, 320), (672, 672)])
def test_rule_picks_a_resident_kernel(size):
    from fpie_gb300 import backend

    mask, tgt, grad = _inputs(*size, 3)
    s = backend.GridSolver(8, 8)
    s.reset(mask.size, mask, tgt, grad)
    assert s.resident in SHAPES
    _compare(s, cjacobi.CGrid(mask, tgt, grad), (33, 100))


@pytest.mark.parametrize("size,deep4", [((768, 768), False), ((769, 673), True), ((840, 840), True),
                                        ((841, 840), False), ((97, 2592), False), ((193, 2305), True)])
def test_depth_4_above_64_tiles_of_the_flow_kernel(size, deep4):
    from fpie_gb300 import backend

    mask, tgt, grad = _inputs(*size, 5)
    s = backend.GridSolver(8, 8)
    s.reset(mask.size, mask, tgt, grad)
    assert (s.resident == "p16w8x128k4r") == deep4
    _compare(s, cjacobi.CGrid(mask, tgt, grad), (33,))


def test_inactive_tiles_and_new_masks():
    """Tiles without unknowns neither send nor wait; a second reset of the
    same geometry with another mask and the state's other buffer."""
    from fpie_gb300 import backend

    s = backend.GridSolver(8, 8)
    s.set_kernel("p8w4x64k16r")
    for seed in (1, 2):
        mask, tgt, grad = _inputs(150, 200, seed, 0.5)
        mask[40:110] = 0
        mask[:, 90:130] = 0
        mask[75, 110] = seed - 1
        s.reset(mask.size, mask, tgt, grad)
        _compare(s, cjacobi.CGrid(mask, tgt, grad), (50, 51))


def _islands():
    """3x3 islands of unknowns on a black ground: values halve every two
    sweeps, through 2^-60 and the subnormals to 0; beside them a solid part
    whose values stay ordinary."""
    n, m = 100, 130
    mask = np.zeros((n, m), np.int32)
    for r in range(2, n - 5, 7):
        for c in range(2, 60, 7):
            mask[r:r + 3, c:c + 3] = 1
    mask[3:95, 64:128] = 1
    mask[50, 58:64] = 1  # a bridge, so that tiny and ordinary values meet
    rng = np.random.default_rng(4)
    tgt = np.where(mask[..., None] != 0, rng.uniform(0, 255, (n, m, 3)), 0).astype(np.float32)
    grad = np.zeros((n, m, 3), np.float32)
    grad[:, 64:] = rng.uniform(-30, 30, (n, m - 64, 3))
    grad[mask == 0] = 0
    return mask, tgt, grad


@pytest.mark.parametrize("kernel", ["auto", "p8w4x64k16r", "p16w8x128k16r"])
def test_values_decaying_through_the_subnormals(kernel):
    from fpie_gb300 import backend

    mask, tgt, grad = _islands()
    s = backend.GridSolver(8, 8)
    s.set_kernel(kernel)
    s.reset(mask.size, mask, tgt, grad)
    o = np_jacobi.GridJacobi(mask, tgt, grad)
    least = []
    for k in (150, 101, 37, 90):  # below 2^-60 from ~140 sweeps, subnormal from ~270
        s.step(k)
        o.sweep(k)
        np.testing.assert_array_equal(s.state(), o.x)
        least.append(float(np.abs(o.x[o.x != 0]).min()))
    assert min(least) < 2.0**-126


@pytest.mark.parametrize("kind", ["huge", "inf", "nan", "tiny gradient", "nan outside the mask"])
def test_inputs_out_of_range(kind):
    from fpie_gb300 import backend

    mask, tgt, grad = _inputs(70, 90, 6)
    mask[30:34, 40:50] = 0
    if kind == "huge":
        tgt *= np.float32(1e36)
        grad *= np.float32(1e35)
    elif kind == "inf":
        tgt[20, 30, 0] = np.inf
        tgt[32, 45, 1] = -np.inf
    elif kind == "nan":
        tgt[20, 30, 0] = np.nan
    elif kind == "tiny gradient":
        tgt[:] = 0
        grad *= np.float32(1e-43)
    else:
        grad[mask == 0] = np.nan  # never read: an unmasked pixel has no gradient
    s = backend.GridSolver(8, 8)
    s.reset(mask.size, mask, tgt, grad)
    assert s.resident
    o = np_jacobi.GridJacobi(mask, tgt, grad)
    with np.errstate(all="ignore"):
        for k in (1, 40, 21):
            s.step(k)
            o.sweep(k)
            np.testing.assert_array_equal(s.state(), o.x)
    # the next reset starts from ordinary inputs again
    mask, tgt, grad = _inputs(70, 90, 7)
    s.reset(mask.size, mask, tgt, grad)
    _compare(s, cjacobi.CGrid(mask, tgt, grad), (40,))


def test_wait_times_out_without_hanging():
    """Spin limit 0: an exchange gives up at its first unmet poll, the step
    raises, and the solver stays usable."""
    from fpie_gb300 import _abi, backend

    mask, tgt, grad = _inputs(300, 300, 8)
    s = backend.GridSolver(8, 8)
    s.set_kernel("p12w8x128k16r")
    s.set_spin_limit(0)
    s.reset(mask.size, mask, tgt, grad)
    with pytest.raises(_abi.FpieTimeoutError):
        s.step(5000)
    s.set_spin_limit(1 << 26)
    s.reset(mask.size, mask, tgt, grad)
    _compare(s, cjacobi.CGrid(mask, tgt, grad), (100,))


def test_tiles_that_do_not_fit_are_refused():
    from fpie_gb300 import _abi, backend

    mask, tgt, grad = _inputs(900, 900, 9)
    s = backend.GridSolver(8, 8)
    s.set_kernel("p8w4x64k16r")
    s.reset(mask.size, mask, tgt, grad)
    assert s.resident == ""
    with pytest.raises(_abi.FpieArgumentError):
        s.step(10)
    s.set_kernel("auto")
    _compare(s, cjacobi.CGrid(mask, tgt, grad), (20,))


@pytest.mark.parametrize("size", [(30, 40), (150, 200)])
@pytest.mark.parametrize("max_sweeps,every", [(0, 16), (100, 33), (4000, 64), (4000, 4000)])
def test_solve_stops_where_the_norms_do(size, max_sweeps, every):
    """The block queued ahead of a check that succeeds leaves no trace: the
    count, the state and what later steps make of it are those of a loop over
    step and residual_norms."""
    from fpie_gb300 import backend

    mask, tgt, grad = _inputs(*size, 11, 0.8)
    s, t = backend.GridSolver(8, 8), backend.GridSolver(8, 8)
    for tol in (1e9, 20.0, 0.5):
        for q in (s, t):
            q.reset(mask.size, mask, tgt, grad)
        assert s.resident
        done = 0
        while done < max_sweeps and t.residual_norms()[0].max() > tol:
            t.step(min(every, max_sweeps - done))
            done += min(every, max_sweeps - done)
        assert s.solve(tol, max_sweeps, every) == done
        np.testing.assert_array_equal(s.state(), t.state())
        for k in (5, 20):
            a, b = s.step(k), t.step(k)
            np.testing.assert_array_equal(a[0], b[0])
            np.testing.assert_array_equal(s.state(), t.state())
        assert s.solve(1e9, 100, 10) == 0  # nothing to do
        np.testing.assert_array_equal(s.state(), t.state())


@pytest.mark.parametrize("size", [(30, 40), (150, 200), (830, 300)])
def test_short_steps_between_long_ones(size):
    """Steps of a few sweeps run as launches after a reset's first one, long
    ones on the resident kernel, on the same state."""
    from fpie_gb300 import backend

    s = backend.GridSolver(8, 8)
    for seed in (1, 2):
        mask, tgt, grad = _inputs(*size, seed, 0.8)
        s.reset(mask.size, mask, tgt, grad)
        assert s.resident
        _compare(s, cjacobi.CGrid(mask, tgt, grad), (1, 1, 4, 5, 16, 17, 3, 40, 2, 16, 1, 64, 16))
