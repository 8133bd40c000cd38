# SPDX-License-Identifier: Apache-2.0
"""The work that users of this framework have it do, as cases to time: decompositions of 1-D, 2-D and
3-D fields in the sizes of the repository's benchmark configurations and tests (one short signal up
to batches of images and volumes), uniform and ragged batches, device and host input, float32 and
float64, with and without the orientation, and the monogenic signal. Inputs follow the benchmark's
recipes (tones, chirps, rings, wavy stripes, blobs, shells, noise), made on the GPU from the seed."""

from __future__ import annotations

import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "eda-cuda_b200"))

import eda  # noqa: E402

TAU = 2 * math.pi
#: The rows that results are stored with, by the spatial dimensions (the mode bound at the largest sizes).
ROWS = {1: 20, 2: 14, 3: 12}


def listed():
    return [
        # one recorded signal decomposed on its own: the smallest call, all latency (the 1-D configuration)
        {"name": "signal", "kind": "uniform", "batch": 1, "d0": 2048, "d1": 0, "d2": 0, "dtype": "float32",
         "host": False, "max_imf": -1, "orientation": False},
        # one long float64 record (odd length) in host memory, its first four modes returned there
        {"name": "record_f64", "kind": "uniform", "batch": 1, "d0": 20011, "d1": 0, "d2": 0, "dtype": "float64",
         "host": True, "max_imf": 4, "orientation": False},
        # channels of one recording: a uniform batch of signals
        {"name": "channels", "kind": "uniform", "batch": 64, "d0": 4096, "d1": 0, "d2": 0, "dtype": "float32",
         "host": False, "max_imf": -1, "orientation": False},
        # a corpus of short recordings of different lengths (the short ragged configuration)
        {"name": "ragged_short", "kind": "ragged", "batch": 1024, "lo": 256, "hi": 8192, "dims": 1,
         "dtype": "float32"},
        # a corpus of recordings over the whole range of lengths (the ragged configuration)
        {"name": "ragged_long", "kind": "ragged", "batch": 1024, "lo": 256, "hi": 65536, "dims": 1,
         "dtype": "float32"},
        # one odd-sized image, as an interactive user decomposes it
        {"name": "image", "kind": "uniform", "batch": 1, "d0": 301, "d1": 443, "d2": 0, "dtype": "float32",
         "host": False, "max_imf": -1, "orientation": False},
        # the headline: a batch of images resident on the GPU
        {"name": "images", "kind": "uniform", "batch": 64, "d0": 512, "d1": 512, "d2": 0, "dtype": "float32",
         "host": False, "max_imf": -1, "orientation": False},
        # images from pinned host memory, their first three modes back in host memory
        {"name": "images_host", "kind": "uniform", "batch": 16, "d0": 512, "d1": 512, "d2": 0, "dtype": "float32",
         "host": True, "max_imf": 3, "orientation": False},
        # float64 images with every mode's orientation
        {"name": "images_f64", "kind": "uniform", "batch": 4, "d0": 333, "d1": 500, "d2": 0, "dtype": "float64",
         "host": False, "max_imf": -1, "orientation": True},
        # volumes (the 3-D configuration), the largest call
        {"name": "volumes", "kind": "uniform", "batch": 4, "d0": 256, "d1": 256, "d2": 256, "dtype": "float32",
         "host": False, "max_imf": -1, "orientation": False},
        # a folder of images of different sizes
        {"name": "ragged_images", "kind": "ragged", "batch": 32, "lo": 64, "hi": 1536, "dims": 2,
         "dtype": "float32"},
        # the monogenic signal of a batch of images
        {"name": "monogenic", "kind": "monogenic", "batch": 16, "d0": 1000, "d1": 768, "d2": 0, "dtype": "float32"},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng: random.Random):
    kind = rng.choice(["signals", "signals", "images", "images", "volumes", "ragged1", "ragged2", "monogenic"])
    dtype = "float64" if rng.random() < 0.25 else "float32"
    host = rng.random() < 0.25
    if kind == "signals":
        n = _log_int(rng, 256, 65536)
        return {"kind": "uniform", "batch": _log_int(rng, 1, max(1, min(256, (1 << 20) // n))), "d0": n, "d1": 0,
                "d2": 0, "dtype": dtype, "host": host,
                "max_imf": 3 if host else -1, "orientation": False}
    if kind == "images":
        h, w = _log_int(rng, 64, 1536), _log_int(rng, 64, 1536)
        most = (1 << 23) // (h * w)  # samples of a call
        return {"kind": "uniform", "batch": _log_int(rng, 1, max(1, min(64, most))), "d0": h, "d1": w, "d2": 0,
                "dtype": dtype, "host": host, "max_imf": 2 if host else -1,
                "orientation": not host and rng.random() < 0.25}
    if kind == "volumes":
        a, b, c = (_log_int(rng, 24, 192) for _ in range(3))
        return {"kind": "uniform", "batch": _log_int(rng, 1, max(1, min(4, (1 << 22) // (a * b * c)))), "d0": a,
                "d1": b, "d2": c, "dtype": "float32", "host": False, "max_imf": -1, "orientation": False}
    if kind == "ragged1":
        return {"kind": "ragged", "batch": _log_int(rng, 16, 1024), "lo": 256, "hi": _log_int(rng, 1024, 65536),
                "dims": 1, "dtype": "float32"}
    if kind == "ragged2":
        return {"kind": "ragged", "batch": _log_int(rng, 4, 24), "lo": 64, "hi": _log_int(rng, 128, 1024), "dims": 2,
                "dtype": "float32"}
    return {"kind": "monogenic", "batch": _log_int(rng, 1, 16), "d0": _log_int(rng, 64, 1024),
            "d1": _log_int(rng, 64, 1024), "d2": 0, "dtype": dtype}


# ---------------------------------------------------------------------------------------------
# inputs

def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _u(g, shape, lo, hi):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _noise(g, shape):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).double()


def _chirps(g, lengths):
    """One signal per length (rows of the longest): a linear chirp from 0.002 to 0.2 cycles per sample, an
    FM tone, a slope, noise."""
    n = torch.tensor(lengths, device="cuda", dtype=torch.float64)[:, None]
    t = torch.arange(max(lengths), device="cuda", dtype=torch.float64)[None]
    w = _u(g, n.shape, 0.05, 0.3)
    f = torch.cos(TAU * (0.002 * t + 0.5 * 0.198 / n * t * t)) + 0.8 * torch.cos(w * t + 0.8 * torch.sin(w * t))
    f += _u(g, n.shape, -1e-3, 1e-3) * t
    return f + 0.01 * _noise(g, f.shape)


def _tones(g, batch, n):
    t = torch.arange(n, device="cuda", dtype=torch.float64)[None]
    f = 0.01 * _noise(g, (batch, n))
    for amp, period in ((1, 8), (2, 64), (3, 512)):
        f += amp * torch.sin(TAU * t / period + _u(g, (batch, 1), 0, TAU))
    return f


def _images(g, batch, h, w):
    """Rings, wavy stripes, two blobs and noise, their scales following the image's side."""
    s = math.sqrt(h * w) / 512
    y = torch.arange(h, device="cuda", dtype=torch.float64)[None, :, None]
    x = torch.arange(w, device="cuda", dtype=torch.float64)[None, None, :]
    one = (batch, 1, 1)
    f = torch.cos(TAU * torch.hypot(y - _u(g, one, 0, h), x - _u(g, one, 0, w)) / (6 * s if s > 1 else 6))
    f += 1.5 * torch.cos(TAU * (x + 4 * s * torch.sin(TAU * y / (128 * s))) / (24 * s))
    for _ in range(2):
        f += 3 * torch.exp(-((y - _u(g, one, 0, h)) ** 2 + (x - _u(g, one, 0, w)) ** 2) / (2 * (80 * s) ** 2))
    return f + 0.02 * _noise(g, f.shape)


def _volume(g, a, b, c):
    """Spherical shells, a plane wave of rising period, a wide blob and noise."""
    z = torch.arange(a, device="cuda", dtype=torch.float64)[:, None, None]
    y = torch.arange(b, device="cuda", dtype=torch.float64)[None, :, None]
    x = torch.arange(c, device="cuda", dtype=torch.float64)[None, None, :]
    at = lambda n: float(_u(g, (1,), 0, n))  # noqa: E731
    f = torch.cos(TAU * torch.sqrt((z - at(a)) ** 2 + (y - at(b)) ** 2 + (x - at(c)) ** 2) / 8)
    f = f + torch.cos(TAU * z / (32 + 32 * z / max(a - 1, 1)))
    sigma = 90 * max(a, b, c) / 256
    f += 3 * torch.exp(-((z - at(a)) ** 2 + (y - at(b)) ** 2 + (x - at(c)) ** 2) / (2 * sigma ** 2))
    return f + 0.01 * _noise(g, f.shape)


def _fields(case, g):
    spatial = [case[k] for k in ("d0", "d1", "d2") if case[k]]
    if len(spatial) == 1:
        return _tones(g, case["batch"], spatial[0])
    if len(spatial) == 2:
        return _images(g, case["batch"], *spatial)
    return torch.stack([_volume(g, *spatial) for _ in range(case["batch"])])


def prepare(case, seed):
    g = _gen(seed)
    dtype = getattr(torch, case["dtype"])
    if case["kind"] == "ragged":
        # the sizes follow the case, the samples the seed
        r = random.Random(case["batch"] * 131071 + case["hi"])
        if case["dims"] == 1:
            lengths = [_log_int(r, case["lo"], case["hi"]) for _ in range(case["batch"])]
            rows = _chirps(g, lengths).to(dtype)
            xs = [rows[i, :n].clone() for i, n in enumerate(lengths)]
            return {"case": case, "dims": 1, "xs": xs, "samples": sum(lengths)}
        sides = [(r.randint(case["lo"], case["hi"]), r.randint(case["lo"], case["hi"])) for _ in range(case["batch"])]
        xs = [_images(g, 1, h, w)[0].to(dtype) for h, w in sides]
        return {"case": case, "dims": 2, "xs": xs, "samples": sum(h * w for h, w in sides)}
    x = _fields(case, g).to(dtype)
    if case.get("host"):
        x = x.cpu().pin_memory().numpy()
    return {"case": case, "dims": x.ndim - 1, "x": x, "axes": tuple(range(1, x.ndim))}


def _stored(t, dim, size):
    """t in storage of `size` entries along `dim` (a program that archives results lays them out by the most
    modes that a field can have, zero beyond its own)."""
    shape = list(t.shape)
    shape[dim] = size - shape[dim]
    if isinstance(t, np.ndarray):
        return np.concatenate([t, np.zeros(shape, t.dtype)], dim)
    return torch.cat([t, t.new_zeros(shape)], dim)


def run(state):
    case = state["case"]
    if case["kind"] == "monogenic":
        m = eda.monogenic(state["x"], state["axes"])
        return {k: getattr(m, k).torch() for k in ("amplitude", "phase", "frequency", "direction", "coherence")}
    most = ROWS[state["dims"]]
    if case["kind"] == "ragged":
        rows, infos = eda.decompose_ragged(state["xs"], return_info=True)
        flat = torch.cat([r.torch().reshape(-1) for r in rows])
        windows = np.zeros((len(infos), most), np.int32)
        for w, i in zip(windows, infos):
            w[:i.windows.size] = i.windows
        return {"rows": _stored(flat, 0, most * state["samples"]), "n_imfs": np.array([int(i.n_imfs) for i in infos]),
                "windows": windows}
    got = eda.decompose(state["x"], state["axes"], case["max_imf"], return_info=True,
                        return_orientation=case["orientation"])
    rows, info = got[:2]
    # host rows are returned as they are: max_imf says how many there are
    out = {"rows": rows if case["host"] else _stored(rows.torch(), 1, most), "n_imfs": info.n_imfs,
           "windows": _stored(info.windows, 1, most), "sifts": _stored(info.sifts, 1, most),
           "energy": _stored(info.energy, 1, most)}
    if case["orientation"]:
        out["direction"] = _stored(got[2].direction.torch(), 1, most)
        out["coherence"] = _stored(got[2].coherence.torch(), 1, most)
    return out


def work(case):
    """Bytes: the input once and the rows once (4 modes' worth of rows, as the recipes' fields have; the
    monogenic signal's planes). Flops: the fast transforms of the orientation (2-D and 3-D; per mode or
    call the forward one and those of the Riesz components)."""
    item = 8 if case["dtype"] == "float64" else 4
    if case["kind"] == "ragged":
        dims = case["dims"]
        # the mean of exp(U[ln lo, ln hi]) lengths, of the product of two U[lo, hi] sides
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"]) if dims == 1 else ((case["lo"] + case["hi"]) / 2) ** 2
        samples = case["batch"] * mean
        side = mean
    else:
        spatial = [case[k] for k in ("d0", "d1", "d2") if case[k]]
        dims = len(spatial)
        side = math.prod(spatial)
        samples = case["batch"] * side
    transforms = 1 + dims + dims * (dims + 1) // 2
    if case["kind"] == "monogenic":
        return {"bytes": item * samples * (1 + 4 + dims), "flops": 5 * samples * math.log2(side) * (2 * transforms)}
    planes = 1 + 4 + (3 * (dims + 1) if case.get("orientation") else 0)
    return {"bytes": item * samples * planes,
            "flops": 5 * samples * math.log2(side) * transforms * 3 if dims >= 2 else samples}


def exact(case, seed):
    """The monogenic signal in float64 by dense transforms. A decomposition has no value of this kind: its
    rows follow from order statistics, extremum counts and odd windows of the data in its own dtype, and a
    restatement of the whole method in plain torch takes minutes."""
    if case["kind"] != "monogenic":
        return None
    f = prepare(case, seed)["x"].double()
    n = f.shape[1:]

    def basis(size):  # rows: frequencies; the orthonormal cosine basis and its sine partner
        k = torch.arange(size, device="cuda", dtype=torch.float64)[:, None]
        x = torch.arange(size, device="cuda", dtype=torch.float64)[None]
        scale = torch.where(k > 0, 2.0, 1.0).div(size).sqrt()
        angle = math.pi * torch.remainder(k * (2 * x + 1), 4 * size) / (2 * size)
        return scale * torch.cos(angle), scale * torch.sin(angle)

    (c0, s0), (c1, s1) = basis(n[0]), basis(n[1])
    spec = c0 @ (f - f.mean((1, 2), keepdim=True)) @ c1.T
    u = [torch.arange(n[0], device="cuda", dtype=torch.float64)[:, None] / (2 * n[0]) + 0 * spec[0],
         torch.arange(n[1], device="cuda", dtype=torch.float64)[None] / (2 * n[1]) + 0 * spec[0]]
    rad = torch.hypot(u[0], u[1])
    inv = torch.where(rad > 0, 1 / rad, 0.0)
    back = lambda m, odd0, odd1: (s0 if odd0 else c0).T @ (m * spec) @ (s1 if odd1 else c1)  # noqa: E731
    p, q = back(u[0] * inv, 1, 0), back(u[1] * inv, 0, 1)
    r00, r11 = back(-(u[0] * inv) ** 2, 0, 0), back(-(u[1] * inv) ** 2, 0, 0)
    r01 = back(u[0] * u[1] * inv ** 2, 1, 1)
    t00, t01, t11 = p * p + r00 * r00 + r01 * r01, p * q + r00 * r01 + r01 * r11, q * q + r01 * r01 + r11 * r11
    gap = torch.hypot(t00 - t11, 2 * t01)
    angle = 0.5 * torch.atan2(2 * t01, t00 - t11)
    n0, n1 = torch.cos(angle), torch.sin(angle)
    tie = 2.0 ** -14 if case["dtype"] == "float32" else 2.0 ** -30
    lead = torch.where(n0.abs() > tie, n0, n1)
    n0, n1 = torch.where(lead < 0, -n0, n0), torch.where(lead < 0, -n1, n1)
    quad = n0 * p + n1 * q
    a2 = f * f + p * p + q * q
    dnf = n0 * back(-u[0], 1, 0) + n1 * back(-u[1], 0, 1)
    dnq = (n0 * n0 * back(u[0] * u[0] * inv, 0, 0) + n1 * n1 * back(u[1] * u[1] * inv, 0, 0)
           + 2 * n0 * n1 * back(-u[0] * u[1] * inv, 1, 1))
    return {"amplitude": a2.sqrt(), "phase": torch.atan2(quad, f), "frequency": (f * dnq - quad * dnf) / a2,
            "direction": torch.stack([n0, n1], 1), "coherence": gap / (t00 + t11)}
