# SPDX-License-Identifier: Apache-2.0
"""Replayed launch sequences (replay.hpp) give what the same launches issued one by one give, bit for
bit: the first, second and later calls of a geometry, on other data each time; geometries in turn,
more of them than the cache keeps; another constant of the call; fields that fail; other streams and
threads; both sides of the size rule; settings and instrumentation changed, and the device synchronised, by
another thread meanwhile; the launches counted. Calls that are instrumented (eda_profile) issue every one."""

from __future__ import annotations

import ctypes
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from eda import _native

    return ctypes.CDLL(str(_native.LIB))


def field(shape, dtype, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal(shape)
    for a in range(1, len(shape)):
        t = np.arange(shape[a]).reshape([-1 if k == a else 1 for k in range(len(shape))])
        x = x + np.sin(2 * np.pi * t / rng.uniform(9, 30)) + 2 * np.sin(2 * np.pi * t / rng.uniform(50, 90))
    return x.astype(dtype)


def results(x, **kw):
    import eda

    y, info = eda.decompose(x, axes=tuple(range(1, x.ndim)), return_info=True, errors="status", **kw)
    y = y.cpu().numpy() if hasattr(y, "cpu") else np.asarray(y)
    return [y] + [np.asarray(getattr(info, k)) for k in ("n_imfs", "error", "windows", "sifts", "spacing", "energy")]


def issued(lib, x, **kw):
    lib.eda_profile(1)
    try:
        return results(x, **kw)
    finally:
        lib.eda_profile(0)


def check(lib, x, **kw):
    got, want = results(x, **kw), issued(lib, x, **kw)
    for a, b in zip(got, want):
        assert a.shape == b.shape and a.tobytes() == b.tobytes()


SHAPES = [(1, 2048), (3, 300), (2, 41, 67), (3, 9, 14, 33), (1, 2), (70, 513), (1, 20011)]


def replays(lib):
    """Graphs built, launches of them, sequences refused, graphs evicted so far."""
    out = [ctypes.c_int64() for _ in range(4)]
    assert lib.eda_testing_replays(*(ctypes.byref(c) for c in out)) == 0
    return np.array([c.value for c in out])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_calls_of_one_geometry(lib, shape, dtype):
    before = replays(lib)
    for seed in range(4):
        x = field(shape, dtype, seed)
        if seed == 1:
            x[-1] = 0.5  # a field without modes beside the others
        if seed == 2:
            x[0].reshape(-1)[1] = np.nan  # one that fails
        check(lib, x)
    built, launched, refused, _ = replays(lib) - before
    assert built > 0 and launched >= built and refused == 0


def test_geometries_and_constants_in_turn(lib):
    for shape in SHAPES:  # (the first graphs, which the others push out)
        for seed in range(3):
            check(lib, field(shape, np.float32, seed))
    before = replays(lib)
    for seed in range(2):
        for shape in SHAPES:  # (each has several sequences: more than the cache keeps)
            for kw in ({}, {"max_imf": 2}, {"tie_tolerance": 0.01}, {"check_finite": False}):
                check(lib, field(shape, np.float32, seed), **kw)
    _, _, refused, evicted = replays(lib) - before
    assert evicted > 0 and refused == 0


@pytest.mark.parametrize("shape", [(4, 512, 512), (5, 512, 512)], ids=["at the limit", "above"])
def test_size_rule(lib, shape):
    before = replays(lib)
    for seed in range(3):
        check(lib, field(shape, np.float32, seed), max_imf=2)
    built, launched, refused, _ = replays(lib) - before
    assert refused == 0
    assert (built > 0 and launched > 0) if shape[0] == 4 else (built == 0 and launched == 0)


def test_streams_and_threads(lib):
    import torch

    xs = [field((2, 700), np.float32, s) for s in range(6)]
    want = [issued(lib, x) for x in xs]
    wrong = []

    def work(k):
        stream = torch.cuda.Stream()
        for rep in range(3):
            for i in range(len(xs)):
                j = (i + k) % len(xs)
                with torch.cuda.stream(stream if rep else torch.cuda.current_stream()):
                    got = results(torch.from_numpy(xs[j]).cuda())
                if any(a.tobytes() != b.tobytes() for a, b in zip(got, want[j])):
                    wrong.append((k, rep, j))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_the_product_of_the_transforms_changed_during_calls(lib):
    """A call takes the product that is set when it begins, all of its transforms the same one: what calls
    beside a thread that keeps changing it have left in the cache is what a later call issues."""
    import eda

    try:
        for i in range(5):
            x, ends = field((1, 60 + 8 * i, 70), np.float32, i), threading.Event()

            def change():
                while not ends.is_set():
                    eda.set_transform_precision("bf16x3")
                    eda.set_transform_precision("tf32x3")

            t = threading.Thread(target=change)
            t.start()
            for _ in range(4):
                results(x)
            ends.set()
            t.join()
            for name in ("tf32x3", "bf16x3"):
                eda.set_transform_precision(name)
                check(lib, x)
    finally:
        eda.set_transform_precision("tf32x3")


def test_another_thread_synchronises_the_device(lib):
    """The sequences are built without a capture, during which no thread may synchronise the device."""
    import torch

    torch.cuda.synchronize()
    ends, errors, rounds = threading.Event(), [], [0]

    def synchronise():
        while not ends.is_set():
            try:
                torch.cuda.synchronize()
                rounds[0] += 1
            except RuntimeError as e:
                errors.append(str(e))
                return

    t = threading.Thread(target=synchronise)
    t.start()
    try:
        for i in range(8):
            for shape in ((1, 900 + 2 * i), (1, 24 + i, 33)):
                for seed in range(4):
                    check(lib, field(shape, np.float32, seed))
    finally:
        ends.set()
        t.join()
    assert rounds[0] > 0 and not errors


def counts(lib):
    n, passes, moved, ms = ctypes.c_int64(), ctypes.c_int64(), ctypes.c_double(), ctypes.c_double()
    assert lib.eda_profile_read(ctypes.byref(n), ctypes.byref(passes), ctypes.byref(moved), ctypes.byref(ms)) == 0
    return n.value, passes.value, moved.value


def test_instrumentation_switched_during_calls(lib):
    """Sequences hold no instrumentation: with it off again, replays count no bytes and no passes."""
    ends = threading.Event()

    def switch():
        while not ends.is_set():
            lib.eda_profile(1)
            time.sleep(1e-3)
            lib.eda_profile(0)
            time.sleep(1e-3)

    xs = [field((1, 1300 + 2 * i), np.float32, i) for i in range(6)]
    t = threading.Thread(target=switch)
    t.start()
    for x in xs[::-1]:
        for _ in range(6):
            results(x)
    ends.set()
    t.join()
    for x in xs:
        lib.eda_profile(0)
        results(x)
        assert counts(lib)[1:] == (0, 0.0)
        check(lib, x)


@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_replayed_launches_are_counted(lib, shape):
    x = field(shape, np.float32, 5)
    launches = []
    for on in (1, 0, 0, 0):
        lib.eda_profile(on)
        results(x)
        launches.append(counts(lib)[0])
    lib.eda_profile(0)
    assert launches[0] > 20 and len(set(launches)) == 1, launches


def test_sequences_are_built_in_a_second_call(lib):
    """The modes of one call share their sequences: a geometry that is met once builds no graph."""
    before = replays(lib)
    for n in range(5000, 5040, 4):
        results(field((1, n), np.float32, n))
    assert not (replays(lib) - before)[:3].any()
    results(field((1, 5036), np.float32, 5036))
    assert (replays(lib) - before)[0] > 0


@pytest.mark.parametrize("workers", [1, 4])
def test_ragged_batches_issue_every_launch(lib, workers):
    import eda

    rng = np.random.default_rng(workers)
    batches = [[rng.standard_normal(600).astype(np.float32) for _ in range(3)],  # one group of one length
               [rng.standard_normal((20 + k, 30)).astype(np.float32) for k in range(3)],
               [rng.standard_normal(s).astype(np.float32) for s in (100, 90, 2000, 2100, 77)]]
    before = replays(lib)
    for _ in range(3):
        for xs in batches:
            eda.decompose_ragged(xs, workers=workers)
    assert not (replays(lib) - before).any()
