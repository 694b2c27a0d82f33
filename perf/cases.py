"""The work whose speed is followed from one version to the next.

Every case calls the library the way a program does: a plan made once
(`aclfft.Plan`, `aclfft.RaggedPlan`), device buffers, and one or more exec
calls per pass.  `listed()` names twelve fixed cases, `draw(rng)` gives more
of the same ranges, `prepare(case, seed)` makes a program's buffers and
plans, `run(state)` is one pass, `work(case)` the bytes and operations that
no implementation can do without, and `exact(case, seed)` the same outputs
from torch.fft in double precision.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "ops-fft_gb300"))

import aclfft as A  # noqa: E402

MAX_ODD_REAL = 6561      # odd real lengths run in one on-chip transform
# real lengths whose R2C adjoint takes per-bin loss weights
WEIGHTED = (256, 512, 1024, 2048, 3000, 4096, 8192)


def listed():
    return [
        # one short real signal, as a control loop calls it: spectrum, signal
        # back and the adjoint, three calls whose latency is what counts
        {"name": "real_step_2100x1", "kind": "real", "n": 2100, "batch": 1, "weighted": False},
        # the plain batched transform: N = 4096, batch 256, forward
        {"name": "c2c_4096x256", "kind": "c2c", "n": 4096, "batch": 256, "inverse": False},
        # a spectral loss step: R2C, C2R of the spectrum and the R2C adjoint of
        # the loss gradient w * X, mixed-radix N = 3000, batch 4096
        {"name": "real_step_3000x4096", "kind": "real", "n": 3000, "batch": 4096, "weighted": True},
        # a length with four prime factors, batched, backward direction
        {"name": "c2c_2310x4096_inv", "kind": "c2c", "n": 2310, "batch": 4096, "inverse": True},
        # long batched transforms, one transform larger than one SM holds
        {"name": "c2c_65536x64", "kind": "c2c", "n": 65536, "batch": 64, "inverse": False},
        # many real signals of 16384 samples, forward and adjoint
        {"name": "real_step_16384x4096", "kind": "real", "n": 16384, "batch": 4096, "weighted": False},
        # long real signals (a quarter million samples), forward, backward and adjoint
        {"name": "real_step_262144x128", "kind": "real", "n": 262144, "batch": 128, "weighted": False},
        # 2D images, forward and normalised inverse
        {"name": "fft2_8x2048x2048", "kind": "nd", "dims": "2048,2048", "batch": 8},
        # one 3D volume, forward and normalised inverse
        {"name": "fft3_512x512x512", "kind": "nd", "dims": "512,512,512", "batch": 1},
        # strided transforms down the columns of a [256][263168] array
        {"name": "vertical_256x263168", "kind": "vertical", "n": 256, "batch": 263168, "inverse": False},
        # real data in double precision, forward and backward
        {"name": "double_step_3000x2048", "kind": "double", "n": 3000, "batch": 2048},
        # 10000 transforms of mixed lengths and kinds in one launch
        {"name": "ragged_10000", "kind": "ragged", "count": 10000, "lo": 16, "hi": 32768, "set": 12345},
    ]


def _smooth(n):
    for p in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47):
        while n % p == 0:
            n //= p
    return n == 1


def _length(rng, lo, hi, odd=None):
    """A length the planner takes, log-uniform over [lo, hi]: half of them
    powers of two or small multiples of one, the others any product of primes
    up to 47 (odd=True / False restricts the parity)."""
    while True:
        x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        if odd is not True and rng.random() < 0.5:
            m = rng.choice([1, 1, 1, 3, 5, 7, 9, 15])
            n = m << max(0, round(math.log2(x / m)))
        else:
            n = round(x)
            while not _smooth(n):
                n += 1
        if lo <= n <= hi and (odd is None or n % 2 == int(odd)):
            return n


def _batch(rng, per, lo_points, hi_points):
    pts = math.exp(rng.uniform(math.log(max(lo_points, per)), math.log(max(hi_points, per))))
    return max(1, round(pts / per))


def draw(rng: random.Random):
    kind = rng.choice(["c2c", "c2c", "c2c", "real", "real", "real", "nd", "nd", "vertical", "double", "ragged"])
    if kind == "c2c":
        n = _length(rng, 16, 1 << 20)
        return {"kind": kind, "n": n, "batch": _batch(rng, n, 1 << 10, 1 << 25), "inverse": rng.random() < 0.5}
    if kind == "real":
        if rng.random() < 0.2:
            n = rng.choice(WEIGHTED)
            return {"kind": kind, "n": n, "batch": _batch(rng, n, 1 << 10, 1 << 26), "weighted": True}
        odd = rng.random() < 0.2
        n = _length(rng, 16, MAX_ODD_REAL if odd else 1 << 20, odd)
        return {"kind": kind, "n": n, "batch": _batch(rng, n, 1 << 10, 1 << 26), "weighted": False}
    if kind == "nd":
        if rng.random() < 0.5:
            a, b = _length(rng, 32, 4096), _length(rng, 32, 4096)
            return {"kind": kind, "dims": f"{a},{b}", "batch": _batch(rng, a * b, 1 << 14, 1 << 25)}
        d = [_length(rng, 24, 480) for _ in range(3)]
        return {"kind": kind, "dims": ",".join(map(str, d)), "batch": 1}
    if kind == "vertical":
        n = 1 << rng.randint(8, 15)  # vertical plans take powers of two from 256
        return {"kind": kind, "n": n, "batch": _batch(rng, n, 1 << 14, 1 << 26), "inverse": rng.random() < 0.5}
    if kind == "double":
        n = _length(rng, 16, 1 << 16)
        return {"kind": kind, "n": n, "batch": _batch(rng, n, 1 << 10, 1 << 23)}
    hi = 1 << rng.randint(10, 15)
    return {"kind": kind, "count": round(math.exp(rng.uniform(math.log(100), math.log(10000)))), "lo": 16, "hi": hi,
            "set": rng.randint(0, 1 << 30)}


def _dims(case):
    return tuple(int(v) for v in case["dims"].split(","))


def _inputs(case, seed):
    """The input tensors of a case, from the seed alone."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def real(*shape, dtype=torch.float32):
        return torch.randn(shape, generator=g, device="cuda", dtype=dtype)

    def cplx(*shape):
        return torch.view_as_complex(real(*shape, 2))

    kind = case["kind"]
    if kind == "c2c":
        return (cplx(case["batch"], case["n"]),)
    if kind == "vertical":
        return (cplx(case["n"], case["batch"]),)
    if kind == "nd":
        return (cplx(case["batch"], *_dims(case)),)
    n, b = case.get("n"), case.get("batch")
    if kind == "real":
        x = real(b, n)
        if not case["weighted"]:
            return (x,)
        return x, torch.rand((b, n // 2 + 1), generator=g, device="cuda")
    if kind == "double":
        return (real(b, n, dtype=torch.float64),)
    _, _, ino, _, ci, _ = _ragged(case)
    return (real(ci // 4),)


def _ragged(case):
    lens, kinds = A.ragged_lengths(case["count"], case["lo"], case["hi"], 0.7, case["set"])
    return (lens, kinds) + A.ragged_layout(lens, kinds)


def prepare(case, seed):
    kind = case["kind"]
    x = _inputs(case, seed)
    stream = torch.cuda.current_stream()
    n, b = case.get("n"), case.get("batch")
    st = {"kind": kind, "x": x}

    def plan(make, *args):
        p = make(*args)
        p.set_stream(stream)
        return p

    if kind in ("c2c", "vertical"):
        dim = A.VERTICAL if kind == "vertical" else A.HORIZONTAL
        st["plan"] = plan(A.Plan.plan1d, n, A.C2C, b, dim)
        st["dir"] = A.BACKWARD if case["inverse"] else A.FORWARD
        st["y"] = torch.empty_like(x[0])
    elif kind == "nd":
        d = _dims(case)
        st["plan"] = plan(A.Plan.plan2d, b, *d) if len(d) == 2 else plan(A.Plan.plan3d, *d)
        st["plan"].set_norm(A.NORM_BACKWARD)
        st["y"], st["z"] = torch.empty_like(x[0]), torch.empty_like(x[0])
    elif kind == "real":
        st["r2c"] = plan(A.Plan.plan1d, n, A.R2C, b)
        st["c2r"] = plan(A.Plan.plan1d, n, A.C2R, b)
        st["X"] = torch.empty((b, n // 2 + 1), dtype=torch.complex64, device="cuda")
        st["y"], st["dx"] = torch.empty_like(x[0]), torch.empty_like(x[0])
    elif kind == "double":
        st["d2z"] = plan(A.Plan.plan1d, n, A.D2Z, b)
        st["z2d"] = plan(A.Plan.plan1d, n, A.Z2D, b)
        st["X"] = torch.empty((b, n // 2 + 1), dtype=torch.complex128, device="cuda")
        st["y"] = torch.empty_like(x[0])
    else:
        lens, kinds, ino, outo, _, co = _ragged(case)
        p = A.RaggedPlan(lens, kinds, ino, outo)
        p.set_stream(stream)
        p.autotune()
        st["plan"] = p
        st["y"] = torch.zeros(co // 4, dtype=torch.float32, device="cuda")
    return st


def run(st):
    kind, x = st["kind"], st["x"]
    if kind in ("c2c", "vertical"):
        st["plan"].exec_c2c(x[0], st["y"], st["dir"])
        return st["y"]
    if kind == "nd":
        st["plan"].exec_c2c(x[0], st["y"], A.FORWARD)
        st["plan"].exec_c2c(st["y"], st["z"], A.BACKWARD)
        return st["y"], st["z"]
    if kind == "real":
        st["r2c"].exec_r2c(x[0], st["X"])
        st["c2r"].exec_c2r(st["X"], st["y"])
        if len(x) == 2:
            st["r2c"].exec_r2c_adjoint_weighted(st["X"], x[1], st["dx"])
        else:
            st["r2c"].exec_r2c_adjoint(st["X"], st["dx"])
        return st["X"], st["y"], st["dx"]
    if kind == "double":
        st["d2z"].exec_d2z(x[0], st["X"])
        st["z2d"].exec_z2d(st["X"], st["y"])
        return st["X"], st["y"]
    st["plan"].exec(x[0], st["y"], A.FORWARD)
    return st["y"]


def _flops(n, count):
    return 5.0 * n * math.log2(max(n, 2)) * count


def work(case):
    """Each input read once and each output written once; 5 N log2 N
    operations per complex transform, half of them for real data."""
    kind = case["kind"]
    n, b = case.get("n"), case.get("batch")
    if kind in ("c2c", "vertical"):
        return {"bytes": 16 * n * b, "flops": _flops(n, b)}
    if kind == "nd":
        p = math.prod(_dims(case))
        return {"bytes": 2 * 16 * p * b, "flops": 2 * _flops(p, b)}
    if kind in ("real", "double"):
        e = 4 if kind == "real" else 8
        one = e * n + 2 * e * (n // 2 + 1)
        if kind == "double":
            return {"bytes": 2 * one * b, "flops": _flops(n, b)}
        extra = 4 * (n // 2 + 1) if case["weighted"] else 0
        return {"bytes": (3 * one + extra) * b, "flops": 1.5 * _flops(n, b)}
    lens, kinds = A.ragged_lengths(case["count"], case["lo"], case["hi"], 0.7, case["set"])
    by = fl = 0
    for m, t in zip(lens.tolist(), kinds.tolist()):
        by += 16 * m if t == A.C2C else 4 * m + 8 * (m // 2 + 1)
        fl += _flops(m, 1 if t == A.C2C else 0.5)
    return {"bytes": by, "flops": fl}


def exact(case, seed):
    kind = case["kind"]
    x = _inputs(case, seed)
    n = case.get("n")
    if kind == "c2c":
        z = x[0].to(torch.complex128)
        return torch.fft.ifft(z, norm="forward") if case["inverse"] else torch.fft.fft(z)
    if kind == "vertical":
        z = x[0].to(torch.complex128)
        return torch.fft.ifft(z, dim=0, norm="forward") if case["inverse"] else torch.fft.fft(z, dim=0)
    if kind == "nd":
        z = x[0].to(torch.complex128)
        return torch.fft.fftn(z, dim=tuple(range(1, z.dim()))), z
    if kind == "real":
        r = x[0].double()
        X = torch.fft.rfft(r)
        y = n * r
        # the adjoint of R2C: Re of the transposed transform of (w *) X over the kept bins
        G = X * x[1].double() if len(x) == 2 else X.clone()
        G[:, 1:(n + 1) // 2] *= 0.5
        return X, y, torch.fft.irfft(G, n, norm="forward")
    if kind == "double":
        return torch.fft.rfft(x[0]), n * x[0]
    lens, kinds, ino, outo, _, co = _ragged(case)
    src, out = x[0].double(), torch.zeros(co // 4, dtype=torch.float64, device="cuda")
    groups = {}
    for i, (m, t) in enumerate(zip(lens.tolist(), kinds.tolist())):
        groups.setdefault((m, t), []).append(i)
    for (m, t), ids in groups.items():
        c2c = t == A.C2C
        m_in, m_out = (2 * m, 2 * m) if c2c else (m, 2 * (m // 2 + 1))
        at = torch.from_numpy(ino[ids] // 4).cuda()[:, None] + torch.arange(m_in, device="cuda")
        rows = src[at]
        y = torch.fft.fft(torch.view_as_complex(rows.view(len(ids), m, 2))) if c2c else torch.fft.rfft(rows)
        to = torch.from_numpy(np.asarray(outo)[ids] // 4).cuda()[:, None] + torch.arange(m_out, device="cuda")
        out[to] = torch.view_as_real(y).reshape(len(ids), m_out)
    return out
