# SPDX-License-Identifier: Apache-2.0
"""1-D lines that several CTAs share, bit for bit: significant extrema of lines cut
into parts (plateaus across the cuts, cuts at the lines' ends, batches that leave one part) against the
oracle, and the energies of rows that one warp folds in several steps or a whole CTA takes, at the
steps' edges, against their definition on the returned rows."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from test_gpu_stats import check_flags, dev  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("batch,n", [(1, 511), (1, 512), (1, 1024), (2, 1025), (3, 3000), (1, 8191), (50, 1600), (149, 1200)])
def test_extrema_of_lines_in_parts(dev, dtype, batch, n):  # noqa: F811
    rng = np.random.default_rng(n + batch)
    long = np.repeat(np.round(rng.standard_normal((batch, n // 300 + 2)) * 3), 300, axis=-1)[:, 7 : 7 + n]
    flat = np.zeros((batch, n))
    flat[:, 1:-1] = 1  # one plateau over every part
    for x in (long, flat, rng.standard_normal((batch, n)), long + (rng.random((batch, n)) < 0.01)):
        x = x.astype(dtype)
        for tau in (0.0, 0.75):
            check_flags(dev, x, np.full(x.shape, tau, dtype))


def canonical_energy(row):
    """sum v^2 in float64 over 32-sample chunks, then the pairwise tree over the chunks."""
    d = np.zeros((row.size + 31) // 32 * 32)
    d[: row.size] = row
    d = d.reshape(-1, 32)
    acc = np.zeros(len(d))
    for e in range(32):
        acc = acc + d[:, e] * d[:, e]
    s = np.zeros(1 << (len(acc) - 1).bit_length())
    s[: len(acc)] = acc
    while s.size > 1:
        s = s[0::2] + s[1::2]
    return s[0]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("batch,n", [(1, 31), (40, 33), (9, 1023), (1, 1024), (300, 1025), (2, 2049), (1, 9217), (3, 33000)])
def test_energies_at_the_steps_edges(dev, dtype, batch, n):  # noqa: F811
    import eda

    rng = np.random.default_rng(n)
    t = np.arange(n)
    x = (np.sin(2 * np.pi * t / 7) + 3 * np.sin(2 * np.pi * t / 61) + rng.standard_normal((batch, n))).astype(dtype)
    y, info = eda.decompose(x, axes=1, max_imf=2, return_info=True)
    for b in range(batch):
        for k in range(int(info.n_imfs[b])):
            assert info.energy[b, k] == canonical_energy(y[b, k]), (b, k)
