"""The bench's apron factor of resident kernels, with one region and with tiles."""

from __future__ import annotations

import pathlib
import sys

import pytest

sys.path.insert(0, str(pathlib.Path(__file__).resolve().parent.parent))
import bench  # noqa: E402


@pytest.mark.parametrize("kernel,crop,factor", [
    ("p6w4x64k8r", (38, 38), 64 / 56), ("p6w4x64k8r", (48, 56), 64 / 56),
    ("p6w4x64k8r", (49, 56), 2.0), ("p6w4x64k8r", (48, 57), 2.0),
    ("p16w8x128k4r", (802, 802), 128 * 128 / (120 * 120)),
    ("p16w8k16d", (38, 38), 128 * 128 / (96 * 96))])
def test_apron_factor(kernel, crop, factor):
    assert abs(bench.apron_factor(kernel, crop) - factor) < 1e-12
