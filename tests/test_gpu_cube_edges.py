# SPDX-License-Identifier: Apache-2.0
"""The cube passes at the edges of their layouts, bit for bit against the oracle: block lengths and
tables of the max / min passes on both sides of their size rules, windows of one and several chunks,
several rungs of one staging in any order (with skipped and one-sample windows), rows and panels of
fewer than 8 lines, and 1-D lines on both sides of the tiled passes' rule and of their tiles."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_stages import check, dev  # noqa: F401

pytestmark = pytest.mark.gpu

# windows of every kind: direct, short blocks, the longest blocks, one and several chunks, clamped
WINS = [1, 3, 5, 7, 11, 13, 15, 17, 19, 27, 29, 31, 33, 55, 63, 65, 127, 641, 1281, 4001]
SHAPES = [(7, 640), (9, 641), (640, 9), (641, 34), (3, 2, 33), (2, 1100), (2300, 3), (17, 16, 40)]
LINES = [4096, 8800, 9100, 12289, 16384, 20481]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("op", ["max", "maxmin", "box"])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_windows_and_rungs(dev, shape, op, dtype):  # noqa: F811
    wins = np.asarray([[w, WINS[(i * 7 + 3) % len(WINS)]] for i, w in enumerate(WINS)], dtype=np.int32)
    wins[4, 1] = 0  # a rung that skips an element
    check(dev, shape, op, wins, dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("op", ["min", "maxmin", "box"])
@pytest.mark.parametrize("n", LINES)
def test_long_lines(dev, n, op, dtype):  # noqa: F811
    wins = np.asarray([[w] for w in (1, 3, 31, 33, 255, 257, 259, 1023, 1025, 1027, 2049, n - 1 + n % 2, 2 * n + 1)], dtype=np.int32)
    check(dev, (n,), op, wins, dtype)
