"""What the speed of this framework is measured on: transforms through the
flagfft.h plans of the Python binding, over the sizes, types, directions and
batch shapes that programs call them with.

A case is a dict of plain values:

* ``kind`` "plan": one plan of ``type`` (C2C, Z2Z, R2C, D2Z), a 1-D transform
  of ``n`` points (``n0`` = 0) or a 2-D one of ``n0`` x ``n``, ``batch`` of them.
  ``mode`` "f" is one forward call, "i" one inverse call (complex types), "fi"
  the forward call and the inverse of its result (R2C then C2R, D2Z then Z2D).
* ``kind`` "uneven": one batch plan of ``count`` complex transforms whose
  lengths are log-uniform in [16, ``n``] (40% powers of two, 30% 7-smooth,
  30% primes), ``salt`` choosing the set.

Every call is out of place on device buffers.  Inputs are uniform in [-1, 1),
or normal for the long real and the 2-D transforms, seeded.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import flagfft_b200 as ffb
from flagfft_b200.workloads import length_groups, uneven_lengths

_REAL_INVERSE = {"R2C": "C2R", "D2Z": "Z2D"}
_SINGLE = ("C2C", "R2C")
_REAL = ("R2C", "D2Z")


def _plan(name, type_, n, batch, mode, n0=0, normal=False):
    return {"name": name, "kind": "plan", "type": type_, "n0": n0, "n": n, "batch": batch, "mode": mode,
            "normal": normal, "salt": 0}


def _uneven(name, count, n, salt, mode="f"):
    return {"name": name, "kind": "uneven", "type": "C2C", "n0": 0, "n": n, "batch": count, "mode": mode,
            "normal": False, "salt": salt}


def listed():
    return [
        # a few short rows there and back: two launches, latency
        _plan("c2c_1024x8_both_ways", "C2C", 1024, 8, "fi"),
        # the plain power-of-two batch of the benchmark (configuration 1)
        _plan("c2c_4096x256_both_ways", "C2C", 4096, 256, "fi"),
        # a smooth length that is not a power of two (sample rates, image widths), inverse
        _plan("c2c_1200x4096_inverse", "C2C", 1200, 4096, "i"),
        # a prime length whose convolution fits on chip (configuration 2)
        _plan("c2c_1009x1024", "C2C", 1009, 1024, "f"),
        # a prime length whose convolution is long, in both precisions (configuration 2)
        _plan("c2c_10007x1024", "C2C", 10007, 1024, "f"),
        _plan("z2z_10007x256", "Z2Z", 10007, 256, "f"),
        # frames of a real signal to spectra and back: the commonest use of a real transform
        _plan("r2c_c2r_2048x8192", "R2C", 2048, 8192, "fi"),
        # the same in double precision at a length that is not a power of two
        _plan("d2z_z2d_1500x1024", "D2Z", 1500, 1024, "fi"),
        # long real signals (configuration 3)
        _plan("r2c_c2r_2^24x4", "R2C", 1 << 24, 4, "fi", normal=True),
        _plan("d2z_3*2^20x2", "D2Z", 3 << 20, 2, "f", normal=True),
        # a large image (configuration 3)
        _plan("c2c_2d_4096x4096", "C2C", 4096, 1, "f", n0=4096, normal=True),
        # many transforms of uneven lengths in one batch plan (configuration 4, fewer of them)
        _uneven("uneven_600_to_16384", 600, 16384, 0),
    ]


# 1-D calls hold at most this many points over the batch, 2-D calls as many per call
_MOST_POINTS = 1 << 24


def _is_prime(n):
    return n > 1 and all(n % d for d in range(2, math.isqrt(n) + 1))


def _smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def _length(rng, lo, hi):
    """Log-uniform in [lo, hi]: a power of two, a 7-smooth number, or up to
    2^17 also a prime or any number (the long primes and the numbers with a
    long prime factor among them take a convolution)."""
    x = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.random() * (0.65 if x > 1 << 17 else 1.0)
    if kind < 0.35:
        return min(hi, max(lo, 1 << round(math.log2(x))))
    if kind < 0.65:
        while not _smooth(x):
            x -= 1
        return max(lo, x)
    if kind < 0.85:
        while not _is_prime(x):
            x -= 1
        return max(lo, x)
    return x


def draw(rng):
    family = rng.random()
    mode = rng.choice(["f", "i", "fi"])
    points = int(math.exp(rng.uniform(math.log(1 << 13), math.log(_MOST_POINTS))))
    if family < 0.12:  # uneven lengths in one plan
        case = _uneven("", rng.randint(50, 600), rng.choice([2048, 4096, 16384]), rng.randint(1, 1 << 20),
                       rng.choice(["f", "i"]))
    elif family < 0.27:  # 2-D, complex and real
        n0, n = _length(rng, 32, 4096), _length(rng, 32, 4096)
        type_ = rng.choice(["C2C", "C2C", "R2C", "Z2Z"])
        cap = _MOST_POINTS // (2 if type_ == "Z2Z" else 1)
        while n0 * n > cap:
            n0 //= 2
        case = _plan("", type_, n, 1, mode, n0=n0, normal=True)
    else:  # 1-D, from one long transform to many short ones
        type_ = rng.choice(["C2C", "C2C", "Z2Z", "R2C", "R2C", "D2Z"])
        if type_ in ("Z2Z", "D2Z"):
            points //= 2
        n = _length(rng, 16, 1 << (24 if type_ == "R2C" else 22))
        if type_ in _REAL and n % 2 and rng.random() < 0.75:
            n += 1
        case = _plan("", type_, n, max(1, min(32768, points // n)), mode)
    if case["type"] in _REAL and case["mode"] == "i":
        case["mode"] = "fi"
    del case["name"]
    return case


def _lengths(case):
    return length_groups(uneven_lengths(case["batch"], 0x55AB + case["salt"], 16, case["n"]))


def _input(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    real = torch.float32 if case["type"] in _SINGLE else torch.float64
    if case["kind"] == "uneven":
        lengths, counts = _lengths(case)
        shape = (sum(a * b for a, b in zip(lengths, counts)),)
    else:
        shape = (case["batch"],) + ((case["n0"],) if case["n0"] else ()) + (case["n"],)
    full = shape if case["type"] in _REAL else shape + (2,)
    if case["normal"]:
        x = torch.randn(full, generator=gen, device="cuda", dtype=real)
    else:
        x = torch.rand(full, generator=gen, device="cuda", dtype=real) * 2 - 1
    return x if case["type"] in _REAL else torch.view_as_complex(x)


def prepare(case, seed):
    x = _input(case, seed)
    state = {"x": x, "mode": case["mode"]}
    if case["kind"] == "uneven":
        state["plan"] = ffb.plan_batch(*_lengths(case), ffb.C2C)
        state["y"] = torch.empty_like(x)
        return state
    n0, n, batch = case["n0"], case["n"], case["batch"]

    def plan(type_):
        t = getattr(ffb, type_)
        return ffb.plan2d(n0, n, t) if n0 else ffb.plan1d(n, t, batch)

    state["plan"] = plan(case["type"])
    if case["type"] in _REAL:
        state["y"] = torch.empty(x.shape[:-1] + (n // 2 + 1,), device="cuda",
                                 dtype=torch.complex64 if x.dtype == torch.float32 else torch.complex128)
        if case["mode"] == "fi":
            state["inverse"] = plan(_REAL_INVERSE[case["type"]])
    else:
        state["y"] = torch.empty_like(x)
        state["inverse"] = state["plan"]
    if case["mode"] == "fi":
        state["z"] = torch.empty_like(x)
    return state


def run(state):
    if state["mode"] == "i":
        state["plan"].execute(state["x"], state["y"], ffb.INVERSE)
        return state["y"]
    state["plan"].execute(state["x"], state["y"], ffb.FORWARD)
    if state["mode"] == "f":
        return state["y"]
    state["inverse"].execute(state["y"], state["z"], ffb.INVERSE)
    return state["y"], state["z"]


def work(case):
    """Input read once and output written once per call; 5 N log2 N flops per
    complex transform, half of it per real one."""
    size = 8 if case["type"] in _SINGLE else 16
    calls = 2 if case["mode"] == "fi" else 1
    if case["kind"] == "uneven":
        lengths, counts = _lengths(case)
        return {"bytes": sum(2.0 * size * n * c for n, c in zip(lengths, counts)),
                "flops": sum(5.0 * n * math.log2(n) * c for n, c in zip(lengths, counts))}
    rows = case["batch"] * max(case["n0"], 1)
    points = case["n"] * max(case["n0"], 1)
    flops = 5.0 * points * math.log2(points) * case["batch"]
    if case["type"] in _REAL:
        one = rows * (case["n"] * size / 2 + (case["n"] // 2 + 1) * size)
        flops /= 2
    else:
        one = 2.0 * rows * case["n"] * size
    return {"bytes": float(one * calls), "flops": flops * calls}


def tolerance(case):
    """About four times the difference from the 64-bit (single precision) or
    extended (double precision) transform that the paths show: 1e-7 to 2.5e-7
    without and 2e-7 to 4e-7 with a convolution in single precision, 2e-16 to
    1e-15 in double."""
    return {"rel": 1.5e-6 if case["type"] in _SINGLE else 4e-15}


def exact(case, seed):
    x = _input(case, seed)
    single = case["type"] in _SINGLE
    if case["kind"] == "uneven":
        x = x.to(torch.complex128)
        lengths, counts = _lengths(case)
        fft = torch.fft.fft if case["mode"] == "f" else torch.fft.ifft
        norm = "backward" if case["mode"] == "f" else "forward"
        out, at = [], 0
        for n, c in zip(lengths, counts):
            out.append(fft(x[at:at + n * c].reshape(c, n), norm=norm).reshape(-1))
            at += n * c
        return torch.cat(out)
    real = case["type"] in _REAL
    axes = (-2, -1) if case["n0"] else (-1,)
    points = case["n"] * max(case["n0"], 1)
    if single:
        x = x.to(torch.float64 if real else torch.complex128)
        if case["mode"] == "i":
            return torch.fft.ifftn(x, dim=axes, norm="forward")
        y = torch.fft.rfftn(x, dim=axes) if real else torch.fft.fftn(x, dim=axes)
    else:
        # double precision is held against extended precision, rounded once
        if points * case["batch"] > 1 << 23:
            return None
        h = x.cpu().numpy().astype(np.longdouble if real else np.clongdouble)
        if case["mode"] == "i":
            y = np.fft.ifftn(h, axes=axes, norm="forward")
        else:
            y = np.fft.rfftn(h, axes=axes) if real else np.fft.fftn(h, axes=axes)
        y = torch.from_numpy(y.astype(np.complex128))
        if case["mode"] == "i":
            return y
    return y if case["mode"] == "f" else (y, x * points)
