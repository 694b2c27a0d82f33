"""The tiles that are compiled with their length, threads and radices
(csrc/tile_list.h): every shape is one that the kernel can run, and the planner
arrives at each of them, so that none is compiled in vain."""
import os
import re

import numpy as np
import pytest

import aclfft as A

_LIST = os.path.join(os.path.dirname(A.__file__), "csrc", "tile_list.h")


def _shapes():
    rows, out = True, []
    for line in open(_LIST):
        if line.startswith("#define GFFT_TILE_COLS"):
            rows = False
        m = re.match(r"\s+X\(([\d, ]+)\)", line)
        if m:
            v = [int(t) for t in m.group(1).split(",")]
            out.append((v[0], rows, v[1], v[2], v[3], v[4:]))
    return out


SHAPES = _shapes()


@pytest.mark.parametrize("ident,rows,L,T,W,rad", SHAPES)
def test_shape_fits_the_kernel(ident, rows, L, T, W, rad):
    assert int(np.prod(rad)) == L and all(2 <= r <= 16 for r in rad)
    assert T * W <= 512 and (rows or W & (W - 1) == 0)
    for r in rad:
        nb = -(-(L // r) // T)             # butterflies a thread holds in this pass
        assert nb * r <= 16 and nb * T >= L // r
    # the padding of the first radix, and that of every later pass' strides
    shift = rad[0].bit_length() - 1 if rad[0] & (rad[0] - 1) == 0 else 30
    pad = lambda i: i + (i >> shift)
    ns = 1
    for p, r in enumerate(rad):
        nbf = L // r
        for j in range(nbf):
            i0 = j // ns * ns * r + j % ns
            for q in range(r):
                if p:
                    assert pad(j) + q * (nbf + (nbf >> shift)) == pad(j + q * nbf)
                assert pad(i0) + q * (1 if ns == 1 else ns + (ns >> shift)) == pad(i0 + q * ns)
        ns *= r


def test_identities_are_the_translation_units():
    ids = sorted(s[0] for s in SHAPES)
    assert ids == list(range(len(ids)))
    csrc = os.path.dirname(_LIST)
    assert sorted(f for f in os.listdir(csrc) if re.match(r"tile_s\d+\.cu", f)) == sorted(f"tile_s{i}.cu" for i in ids)


@pytest.mark.parametrize("ident,rows,L,T,W,rad", [s for s in SHAPES if s[1] or s[2] >= 256])
def test_planner_arrives_at_the_shape(ident, rows, L, T, W, rad):
    """Rows of few and many; strided axes (from 256 points) and the first passes
    of long rows, whose tiles are narrower."""
    if rows:
        plans = [(L, b, A.HORIZONTAL) for b in (64, 1024, 70000)]
    else:
        plans = [(L, b, A.VERTICAL) for b in (64, 600, 4096, 70000)]
        plans += [(n, 64, A.HORIZONTAL) for n in (L * L, L * L // 2, L * L * 2)]
    found = []
    for n, b, dim in plans:
        with A.Plan.plan1d(n, A.C2C, b, dim) as p:
            assert p.check() == "ok"
            i = p.info()
            if i.onchip_length == L:
                found.append((i.threads_per_transform, i.transforms_per_cta, [i.radix[k] for k in range(i.nradix)]))
    assert (T, W, rad) in found, found
