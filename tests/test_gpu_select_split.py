# SPDX-License-Identifier: Apache-2.0
"""The split form of the exact selections (stats.cu: large elements in batches of 16 or more), bit for bit
against the oracle: brackets that hold the ranks, ties that fill the list (handed on to the other
forms), one value everywhere, ranks at both ends, masks, differences and centres, rows with padding;
both sides of the size rule, and the launches of each."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

import oracle
from test_gpu_stats import dev, gpu_select, items  # noqa: F401

pytestmark = pytest.mark.gpu

# 16 elements, 65 536 padded items each and 2^21 in all are the split's; three shapes lie just below
SPLIT = [(32, 256, 256), (17, 500, 523), (33, 65535), (16, 97, 88, 101), (40, 300, 311)]
BELOW = [(31, 256, 256), (15, 500, 523), (40, 256, 223)]
SHAPES = SPLIT + BELOW


def fields(shape, dtype, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "normal":
        x = rng.standard_normal(shape)
    elif kind == "ties":  # a few values: more ties at the median than the list holds
        x = rng.integers(-2, 3, shape).astype(np.float64)
    elif kind == "constant":
        x = np.full(shape, 2.5)
    else:  # half of the samples one value, the rest spread
        x = np.where(rng.random(shape) < 0.5, -0.0, rng.standard_normal(shape))
    x[0].reshape(-1)[:3] = [np.inf, -np.inf, 1e-40]
    return x.astype(dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
@pytest.mark.parametrize("kind", ["normal", "ties", "constant", "half"])
def test_split_samples(dev, shape, dtype, kind):  # noqa: F811
    x = fields(shape, dtype, kind, sum(shape))
    for q in (-1.0, 0.0, 0.25, 1.0):
        out, cnt = gpu_select(dev, x, q=q)
        for b in range(0, shape[0], 7):
            v = items(x[b], 0, 0, None, 0, None)
            want = oracle.select(v, q)  # NaN between -inf and inf, in both
            assert (np.isnan(out[b]) and np.isnan(want)) or out[b] == want, (q, b)
            assert cnt[b] == v.size


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(17, 500, 523), (16, 97, 88, 101)], ids=["2d", "3d"])
def test_split_masks_differences_and_centres(dev, shape, dtype):  # noqa: F811
    rng = np.random.default_rng(2)
    x = fields(shape, dtype, "normal", 9)
    x[0] = np.nan_to_num(x[0], posinf=3, neginf=-3)
    mask = rng.integers(0, 4, shape).astype(np.uint8)
    mask[1] = 0  # no item: NaN
    mask[2] = 0
    mask[2].reshape(-1)[:5] = 1  # fewer items than the sample can find
    center = rng.standard_normal(shape[0])
    for c in (None, center):
        out, cnt = gpu_select(dev, x, mask=mask, bits=1, center=c, q=0.3)
        for b in range(3):
            v = items(x[b], 0, 0, mask[b], 1, None if c is None else c[b])
            want = oracle.select(v, 0.3)
            assert (np.isnan(out[b]) and np.isnan(want)) or out[b] == want, b
            assert cnt[b] == v.size
        for axes in range(1, 1 << (len(shape) - 1)):
            out, cnt = gpu_select(dev, x, src=1, axes=axes, center=c)
            for b in (0, shape[0] - 1):
                v = items(x[b], 1, axes, None, 0, None if c is None else c[b])
                assert out[b] == oracle.select(v), (axes, b)
                assert cnt[b] == v.size


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_size_rule(dev, dtype):  # noqa: F811
    """The split form's three launches come before those of the other forms."""
    _, lib = dev
    n, rest = ctypes.c_int64(), (ctypes.c_int64(), ctypes.c_double(), ctypes.c_double())

    def launches(shape, **kw):
        x = fields(shape, dtype, "normal", 1)
        lib.eda_profile(0)
        gpu_select(dev, x, **kw)
        lib.eda_profile_read(ctypes.byref(n), *(ctypes.byref(v) for v in rest))
        return n.value

    for kw in ({}, {"src": 1, "axes": 3}):
        assert launches((16, 500, 523), **kw) - launches((15, 500, 523), **kw) == 3
        assert launches((32, 256, 256), **kw) - launches((31, 256, 256), **kw) == (3 if not kw else 0)
    assert launches((40, 256, 256)) - launches((40, 255, 256)) == 3
