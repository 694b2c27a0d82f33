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


@pytest.mark.parametrize("n,typ,rad,T,W", [(256, A.R2C, [16, 8], 16, 4), (128, A.C2C, [16, 8], 16, 4),
                                           (256, A.C2C, [16, 16], 16, 4), (512, A.C2C, [8, 8, 8], 64, 1)])
@pytest.mark.parametrize("b", [1, 2, 3, 5])
def test_few_rows_take_a_compiled_tile(n, typ, rad, T, W, b):
    with A.Plan.plan1d(n, typ, b) as p:
        assert p.check() == "ok"
        i = p.info()
        assert ([i.radix[k] for k in range(i.nradix)], i.threads_per_transform, i.transforms_per_cta) == (rad, T, W)
    L = int(np.prod(rad))
    assert any(s[1] and (s[2], s[3], s[4], s[5]) == (L, T, W, rad) for s in SHAPES)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 3, 15, 64, 128, 256, 300, 512, 1024])
@pytest.mark.parametrize("b", [1, 3])
def test_rows_that_leave_most_of_a_tile_idle(n, b):
    """Tolerance: twice 2^-24 per radix-2 level, one product and one sum each."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    x = (rng.standard_normal((b, n)) + 1j * rng.standard_normal((b, n))).astype(np.complex64)
    bound = 2.0 * 2.0 ** -24 * max(np.log2(n), 2.0)
    st = torch.cuda.current_stream()
    with A.Plan.plan1d(n, A.C2C, b) as p, A.Plan.plan1d(n, A.R2C, b) as q, A.Plan.plan1d(n, A.C2R, b) as c:
        for plan in (p, q, c):
            plan.set_stream(st)
        xd, rd = torch.from_numpy(x).cuda(), torch.from_numpy(x.real.copy()).cuda()
        hd, bd = torch.empty((b, n // 2 + 1), dtype=torch.complex64, device="cuda"), torch.empty_like(rd)
        p.exec_c2c(xd, xd, A.FORWARD)  # in place
        q.exec_r2c(rd, hd)
        c.exec_c2r(hd, bd)
    h = np.fft.rfft(x.real.astype(np.float64))
    for out, exact in ((xd, np.fft.fft(x.astype(np.complex128))), (hd, h), (bd, x.real.astype(np.float64) * n)):
        assert np.linalg.norm(out.cpu().numpy() - exact) <= 2 * bound * np.linalg.norm(exact)


@pytest.mark.parametrize("n", [13, 14, 15, 16])
def test_one_thread_rows_up_to_12_mb(n):
    line = (3 << 19) // n
    for b, stages in ((1, 1), (line, 1), (line + 1, 2)):  # tiles have one stage, the row kernel prefetches
        with A.Plan.plan1d(n, A.C2C, b) as p:
            assert p.check() == "ok"
            assert min(p.info().stages, 2) == stages


@pytest.mark.gpu
@pytest.mark.parametrize("n", [13, 14, 15, 16])
def test_one_thread_rows(n):
    """One row, a tile that is not full, and both sides of the kernels' line.
    Tolerance: twice 2^-24 per radix-2 level."""
    torch = pytest.importorskip("torch")
    for b in (1, 65, (3 << 19) // n, (3 << 19) // n + 1):
        g = torch.Generator(device="cuda")
        g.manual_seed(n + b)
        x = torch.randn((b, n), dtype=torch.complex64, generator=g, device="cuda")
        exact = torch.fft.fft(x.to(torch.complex128))
        y = torch.empty_like(x)
        with A.Plan.plan1d(n, A.C2C, b) as p:
            p.set_stream(torch.cuda.current_stream())
            p.exec_c2c(x, y, A.FORWARD)
            p.exec_c2c(x, x, A.FORWARD)  # in place
        assert ((y - exact).norm() / exact.norm()).item() <= 2.0 * 2.0 ** -24 * np.log2(n)
        assert torch.equal(x, y)


@pytest.mark.parametrize("n,width", [(256, 8), (512, 8), (1024, 8), (2048, 4)])
def test_few_columns_keep_a_compiled_tile(n, width):
    for b in (2, 3, 17, 257):  # (one column is one row)
        with A.Plan.plan1d(n, A.C2C, b, A.VERTICAL) as p:
            assert p.check() == "ok"
            i = p.info()
            key = (n, i.threads_per_transform, i.transforms_per_cta, [i.radix[k] for k in range(i.nradix)])
            assert i.transforms_per_cta == width and key in [s[2:] for s in SHAPES if not s[1]]


@pytest.mark.gpu
@pytest.mark.parametrize("n,b", [(256, 1), (256, 17), (512, 3), (512, 129), (1024, 1), (1024, 51), (2048, 2), (2048, 65)])
def test_few_columns(n, b):
    """Tolerance: twice 2^-24 per radix-2 level."""
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda")
    g.manual_seed(n + b)
    x = torch.randn((n, b), dtype=torch.complex64, generator=g, device="cuda")
    exact = torch.fft.fft(x.to(torch.complex128), dim=0)
    y = torch.empty_like(x)
    with A.Plan.plan1d(n, A.C2C, b, A.VERTICAL) as p:
        p.set_stream(torch.cuda.current_stream())
        p.exec_c2c(x, y, A.FORWARD)
        p.exec_c2c(x, x, A.FORWARD)  # in place
    assert ((y - exact).norm() / exact.norm()).item() <= 2.0 * 2.0 ** -24 * np.log2(n)
    assert torch.equal(x, y)
