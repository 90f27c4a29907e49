"""The range in which quartered sums round as the reference's do.

On the CPU in exact integers: 16 sweeps of ((((g + up) + down) + left) + right)
/ 4 and of its quartered form, each operation rounded to float32 with
subnormals, agree for inputs that are 0 or at least 2^-94, and not for much
smaller ones.  On the GPU: pictures whose values pass through that limit, on
every resident shape, against the oracle.
"""

from __future__ import annotations

import random

import numpy as np
import pytest

from oracle import np_jacobi

S = 170  # values are integers in units of 2^-S


def _rn(n: int) -> int:
    """n to the nearest float32, ties to even."""
    a = abs(n)
    shift = max(a.bit_length() - 24, S - 149)
    q, r = a >> shift, a & ((1 << shift) - 1)
    half = 1 << (shift - 1)
    q += r > half or (r == half and q & 1)
    return (q << shift) if n >= 0 else -(q << shift)


def _sweep(x, g, quartered):
    n = len(x)

    def at(i, j):
        return x[i][j] if 0 <= i < n and 0 <= j < n else 0

    out = [[0] * n for _ in range(n)]
    for i in range(n):
        for j in range(n):
            t = g[i][j] // 4 if quartered else g[i][j]
            for v in (at(i - 1, j), at(i + 1, j), at(i, j - 1), at(i, j + 1)):
                t = _rn(t + v // 4) if quartered else _rn(t + v)
            out[i][j] = t if quartered else _rn(t // 4)
    return out


def _draw(rng, least, share, n=10):
    """Values of 24 bits with magnitudes from 2^least on, odd in their last."""
    def value():
        if rng.random() > share:
            return 0
        return rng.choice((-1, 1)) * ((rng.randrange(1 << 23, 1 << 24) | 1) << (S + least - 23 + rng.choice((0, 0, 1, 9))))
    return [[value() for _ in range(n)] for _ in range(n)]


def _differs(seed, least, share):
    rng = random.Random(seed)
    x = y = _draw(rng, least, share)
    g = _draw(rng, least, share if seed % 2 else 0.0)
    for _ in range(16):
        x, y = _sweep(x, g, False), _sweep(y, g, True)
    return x != y


@pytest.mark.parametrize("share", [0.02, 0.1, 1.0])
def test_16_sweeps_agree_from_the_limit_on(share):
    assert not any(_differs(seed, -94, share) for seed in range(8))


def test_much_smaller_values_do_not():
    assert any(_differs(seed, -116, 0.02) for seed in range(12))


SHAPES = {  # name: (tile rows, tile columns)
    "p6w4x64k8r": (32, 48), "p8w4x64k8r": (48, 48), "p8w8x128k8r": (48, 112),
    "p6w4x64k16r": (16, 32), "p8w4x64k16r": (32, 32), "p8w8x64k16r": (96, 32),
    "p8w8x128k16r": (32, 96), "p12w8x128k16r": (64, 96), "p16w8x128k16r": (96, 96),
    "p16w8x128k4r": (120, 120),
}


def _black(n, m, seed):
    """Black but for a bright strip and two faint spots, without a gradient on
    the black; values run through it ahead of what diffuses."""
    rng = np.random.default_rng(seed)
    mask = (rng.random((n, m)) < 0.98).astype(np.int32)
    mask[:, 0] = mask[:, -1] = mask[0] = mask[-1] = 0
    tgt = np.zeros((n, m, 3), np.float32)
    tgt[:, :9] = rng.uniform(0, 255, (n, 9, 3))
    tgt[n // 2, m - 9] = np.float32(2.0**-94 * (1 + 2.0**-23))
    tgt[n // 3, m - 19] = np.float32(2.0**-126 * (1 + 2.0**-23))
    grad = np.zeros((n, m, 3), np.float32)
    grad[:, 2:5] = rng.uniform(-30, 30, (n, 3, 3))
    grad[n // 4, m - 30] = np.float32(-(2.0**-94))
    grad[mask == 0] = 0
    return mask, tgt, grad


@pytest.mark.gpu
@pytest.mark.parametrize("tiles", [(1, 1), (2, 3)])
@pytest.mark.parametrize("kernel", sorted(SHAPES))
def test_black_pictures_on_every_shape(kernel, tiles):
    from fpie_gb300 import backend

    th, tw = SHAPES[kernel]
    depth = int(kernel.split("k")[1][:-1])
    n, m = ((th + 2 * depth, tw + 2 * depth - 8) if tiles == (1, 1)
            else (tiles[0] * th - 3, tiles[1] * tw + 2))
    mask, tgt, grad = _black(n, m, 1)
    s = backend.GridSolver(8, 8)
    s.set_kernel(kernel)
    s.reset(mask.size, mask, tgt, grad)
    o = np_jacobi.GridJacobi(mask, tgt, grad)
    for k in (16, 31, 4, 65, 34):
        s.step(k)
        o.sweep(k)
        np.testing.assert_array_equal(s.state(), o.x)


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", ["p8w8k16", "p16w8k16", "p16w8k8"])
def test_black_pictures_in_a_batch(kernel):
    from fpie_gb300.batch import BatchSolver

    b = BatchSolver(1e9)
    b.set_kernel(kernel)
    jobs = [_black(90, 150, 2), _black(33, 97, 3)]
    ids = [b.add(*j, 150) for j in jobs]
    oracles = [np_jacobi.GridJacobi(*j) for j in jobs]
    for k in (16, 31, 103):
        b.run(k)
        for i, o in zip(ids, oracles):
            o.sweep(k)
            np.testing.assert_array_equal(b.state(i), o.x)
