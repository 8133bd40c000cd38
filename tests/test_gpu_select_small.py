# SPDX-License-Identifier: Apache-2.0
"""The small form of the exact selections (stats.cu: elements whose keys fit one CTA's shared memory), bit
for bit against the oracle: the edges of its thread counts and of its size rule, ties, one value, two far
values (the ranks part), narrow and full ranges of keys, masks, differences and centres."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from test_gpu_stats import dev, gpu_select, items  # noqa: F401

pytestmark = pytest.mark.gpu

SIZES = [(3, 2), (3, 33), (5, 127), (2, 129), (2, 513), (2, 2049), (70, 4096), (2, 4097), (1, 8192), (2, 19999), (1, 26600),
         (1, 26700), (1, 32768), (1, 32800), (3, 90, 101), (3, 14, 15, 44)]


def field(shape, dtype, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "normal":
        x = rng.standard_normal(shape)
    elif kind == "ties":
        x = rng.integers(-2, 3, shape).astype(np.float64)
    elif kind == "constant":
        x = np.full(shape, -2.5)
    elif kind == "parted":  # half of the samples each around two far values
        x = np.where(rng.random(shape) < 0.5, -1e30, 1e-30) * (1 + 1e-3 * rng.random(shape))
    elif kind == "narrow":  # neighbouring floats, most of them in a few values
        x = 1 + np.finfo(dtype).eps * rng.integers(0, 5000, shape)
    else:  # every magnitude, with zeros of both signs and infinities
        x = rng.standard_normal(shape) * 10.0 ** rng.uniform(-44 if dtype == np.float32 else -320, 38, shape)
        x.reshape(-1)[::5] = -0.0
        x.reshape(-1)[::7] = 0.0
        x.reshape(-1)[:2] = [np.inf, -np.inf][: x.size]
    return x.astype(dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SIZES, ids=["x".join(map(str, s)) for s in SIZES])
@pytest.mark.parametrize("kind", ["normal", "ties", "constant", "parted", "narrow", "all"])
def test_small(dev, shape, dtype, kind):  # noqa: F811
    x = field(shape, dtype, kind, sum(shape))
    rng = np.random.default_rng(1)
    mask = rng.integers(0, 4, shape).astype(np.uint8)
    mask[0] = 0
    center = rng.standard_normal(shape[0])
    cases = [({"q": q}, 0, 0, None, None) for q in (-1.0, 0.0, 0.3, 0.5, 1.0)]
    cases += [({"mask": mask}, 0, 0, mask, None), ({"mask": mask, "center": center}, 0, 0, mask, center)]
    if kind != "all" and shape[-1] > 1:
        cases += [({"src": 1, "axes": 1, "center": c}, 1, 1, None, c) for c in (None, center)]
    for kw, src, axes, m, c in cases:
        out, cnt = gpu_select(dev, x, **kw)
        for b in range(0, shape[0], 9 if shape[0] > 9 else 1):
            v = items(x[b], src, axes, None if m is None else m[b], 1 if m is not None else 0, None if c is None else c[b])
            assert cnt[b] == v.size
            want = oracle.select(v, kw.get("q", -1.0)) if v.size else np.nan
            assert (np.isnan(out[b]) and np.isnan(want)) or out[b] == want, (kw, b)
