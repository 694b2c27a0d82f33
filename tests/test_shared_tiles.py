"""Plans whose argument-driven tiles differ in mode run them on one kernel:
rows and columns of real 2D and 3D transforms, and the two passes of long even
real rows with the packing on paired columns.  Lengths of one, two and three
passes on either axis, radices of every kind, one row and many, in place.

Tolerance: twice 2^-24 per radix-2 level of the transform."""
import numpy as np
import pytest

import aclfft as A

torch = pytest.importorskip("torch")

VOLUMES = [(1, 7, 14), (1, 16, 32), (3, 13, 30), (2, 45, 28), (115, 21, 120), (1, 875, 750), (5, 100, 96), (1, 20, 2310),
           (2, 1000, 8), (64, 30, 64)]
CUBES = [(3, 5, 12), (32, 30, 40), (48, 11, 26), (20, 125, 56), (128, 15, 10)]
LONG = [(17150, 4), (17820, 1), (30000, 20), (30250, 3), (36000, 2), (40000, 1), (98304, 2), (17820, 950), (100000, 90)]


def _ok(out, exact, n, what):
    err = ((out - exact).norm() / exact.norm()).item()
    assert err <= 2.0 * 2.0 ** -24 * max(np.log2(n), 2.0), (what, err)


@pytest.mark.parametrize("n,b", LONG)
def test_long_rows_stay_in_bounds(n, b):
    for typ in (A.R2C, A.C2R):
        with A.Plan.plan1d(n, typ, b) as p:
            assert p.check() == "ok" and p.work_size() == n // 2 * b * 8


@pytest.mark.gpu
@pytest.mark.parametrize("dims", VOLUMES + CUBES)
def test_real_2d_and_3d(dims):
    g = torch.Generator(device="cuda")
    g.manual_seed(sum(dims))
    flat = dims in VOLUMES
    axes = (1, 2) if flat else (0, 1, 2)
    pts = int(np.prod(dims[1:] if flat else dims))
    x = torch.randn(dims, generator=g, device="cuda")
    exact = torch.fft.rfftn(x.double(), dim=axes)
    make = A.Plan.plan2d if flat else A.Plan.plan3d
    st = torch.cuda.current_stream()
    with make(*dims, A.R2C) as p, make(*dims, A.C2R) as q:
        assert p.check() == "ok" and q.check() == "ok"
        p.set_stream(st)
        q.set_stream(st)
        X = torch.empty(exact.shape, dtype=torch.complex64, device="cuda")
        y, a, B = torch.empty_like(x), torch.empty_like(x), torch.empty_like(X)
        p.exec_r2c(x, X)
        kept = X.clone()
        q.exec_c2r(X, y)
        assert torch.equal(X, kept)
        p.exec_r2c_adjoint(X, a)
        q.exec_c2r_adjoint(x, B)
        buf = torch.zeros(2 * X.numel(), device="cuda")
        buf[:x.numel()] = x.flatten()
        p.exec_r2c(buf, buf)  # in place
        assert torch.equal(buf, torch.view_as_real(X).flatten())
        q.exec_c2r(buf, buf)
        assert torch.equal(buf[:x.numel()], y.flatten())
    n = dims[2]
    w = torch.full((n // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
    w[0] = w[-1] = 1.0
    _ok(X, exact, pts, "r2c")
    _ok(y, x.double() * pts, pts * pts, "c2r")
    _ok(B, exact * w, pts, "c2r adjoint")
    _ok(a, torch.fft.irfftn(exact / w, s=[dims[k] for k in axes], dim=axes, norm="forward"), pts * pts, "r2c adjoint")


@pytest.mark.gpu
@pytest.mark.parametrize("n,b", LONG)
def test_long_real_rows(n, b):
    g = torch.Generator(device="cuda")
    g.manual_seed(n + b)
    x = torch.randn((b, n), generator=g, device="cuda")
    X = torch.randn((b, n // 2 + 1), dtype=torch.complex64, generator=g, device="cuda")
    X[:, 0].imag.zero_()
    X[:, -1].imag.zero_()
    w = torch.full((n // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
    w[0] = w[-1] = 1.0
    st = torch.cuda.current_stream()
    with A.Plan.plan1d(n, A.R2C, b) as p, A.Plan.plan1d(n, A.C2R, b) as q:
        p.set_stream(st)
        q.set_stream(st)
        Y, y, a, B = torch.empty_like(X), torch.empty_like(x), torch.empty_like(x), torch.empty_like(X)
        p.exec_r2c(x, Y)
        q.exec_c2r(X, y)
        p.exec_r2c_adjoint(X, a)
        q.exec_c2r_adjoint(x, B)
        buf = torch.zeros(2 * X.numel(), device="cuda")
        buf[:b * n] = x.flatten()
        p.exec_r2c(buf, buf)  # in place
        assert torch.equal(buf, torch.view_as_real(Y).flatten())
        buf.copy_(torch.view_as_real(X).flatten())
        q.exec_c2r(buf, buf)
        assert torch.equal(buf[:b * n].view(b, n), y)
    F = torch.fft.rfft(x.double())
    _ok(Y, F, n, "r2c")
    _ok(B, F * w, n, "c2r adjoint")
    Xd = X.to(torch.complex128)
    _ok(y, torch.fft.irfft(Xd, n, norm="forward"), n, "c2r")
    _ok(a, torch.fft.irfft(Xd / w, n, norm="forward"), n, "r2c adjoint")
