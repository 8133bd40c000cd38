# SPDX-License-Identifier: Apache-2.0
"""The tensor-core transforms' tiles of 256 columns (orient_tc.cu: passes of several waves of tiles) against
those of 128, which an element alone takes: the same bits. Rows and columns that end inside the first and the
second half of a tile, elements that begin inside one."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_stages import dev, gpu_transform, host_transform  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(60, 257, 300), (130, 149, 260), (160, 100, 513), (64, 24, 40, 130), (300, 128, 128)],
                         ids=lambda s: "x".join(map(str, s)))
def test_batches_equal_their_elements(dev, shape):  # noqa: F811
    rng = np.random.default_rng(sum(shape))
    x = rng.standard_normal(shape).astype(np.float32)
    kinds = [0, 2, 1][: len(shape) - 1]
    got = gpu_transform(dev, x, kinds)
    for b in range(0, shape[0], 7):
        alone = gpu_transform(dev, x[b : b + 1], kinds)[0]
        assert np.array_equal(got[b].view(np.uint32), alone.view(np.uint32)), b
    want = host_transform(x[:1], kinds)
    assert np.abs(got[:1] - want).max() <= 2e-5 * np.abs(want).max()  # (the bound of the stages' tests)
