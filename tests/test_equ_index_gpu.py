"""The unknowns' coordinates are those of the system loaded, or an error."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call,dtype", [("fpie_equ_get_index", np.int32),
                                        ("fpie_equ_get_index64", np.int64)])
@pytest.mark.parametrize("side", [9, 20, 30])
def test_a_reset_from_arrays_has_no_index(call, dtype, side):
    from fpie_gb300 import _abi, backend

    rng = np.random.default_rng(side)
    src, tgt = (rng.integers(0, 256, (22, 22, 3), dtype=np.uint8) for _ in range(2))
    mask = np.full((22, 22), 255, np.uint8)  # its frame is cleared: 20 x 20 unknowns
    s = backend.EquSolver(256)

    def index():
        out = np.full((2, max(s.N - 1, 400)), -1, dtype)
        _abi.call(call, s._h, ctypes.c_void_p(out[0].ctypes.data), ctypes.c_void_p(out[1].ctypes.data))
        return out[:, : s.N - 1]

    for _ in range(2):
        s.reset_images(src, mask, tgt, (0, 0), (0, 0), "src")
        np.testing.assert_array_equal(index(), np.argwhere(np.pad(np.ones((20, 20)), 1)).T)
        ids = s.partition(np.pad(np.ones((side, side), np.int32), 1))
        N = side * side + 1
        A = np.zeros((N, 4), np.int32)
        A[1:] = np.stack([ids[:-2, 1:-1], ids[2:, 1:-1], ids[1:-1, :-2], ids[1:-1, 2:]], -1).reshape(-1, 4)
        s.reset(N, A, np.zeros((N, 3), np.float32), np.zeros((N, 3), np.float32))
        with pytest.raises(_abi.FpieError):
            index()
