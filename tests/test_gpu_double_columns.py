"""Strided double-precision axes on tiles of 8, 16 and 32 columns (short axes
take wider tiles): one column, columns that do not fill the last tile, every
width, and the widest tile's largest exchange buffer.  Tolerance: as in the
other double-precision tests, 1e-12 (the errors seen are about 1e-15)."""
import numpy as np
import pytest

import aclfft as A
import oracle as O

torch = pytest.importorskip("torch")

SHAPES = [(1, 2, 1), (1, 9, 5), (500, 16, 64), (311, 9, 33), (37, 24, 287), (19, 30, 555), (333, 13, 31), (5, 48, 2009),
          (11, 100, 301), (2, 225, 1209)]


@pytest.mark.parametrize("b,nx,ny", SHAPES)
def test_launches_stay_in_bounds(b, nx, ny):
    for typ in (A.Z2Z, A.D2Z, A.Z2D):
        with A.Plan.plan2d(b, nx, ny, typ) as p:
            assert p.check() == "ok"


@pytest.mark.gpu
@pytest.mark.parametrize("b,nx,ny", SHAPES)
def test_columns(b, nx, ny):
    rng = np.random.default_rng(b + nx + ny)
    x = rng.standard_normal((b, nx, ny)) + 1j * rng.standard_normal((b, nx, ny))
    st = torch.cuda.current_stream()
    xd = torch.from_numpy(x).cuda()
    yd = torch.empty_like(xd)
    with A.Plan.plan2d(b, nx, ny, A.Z2Z) as p:
        p.set_stream(st)
        p.exec_z2z(xd, yd, A.FORWARD)
        zd = xd.clone()
        p.exec_z2z(zd, zd, A.BACKWARD)  # in place
    assert O.errors(yd.cpu().numpy(), np.fft.fft2(x))["rel_l2"] <= 1e-12
    assert O.errors(zd.cpu().numpy(), np.fft.ifft2(x, norm="forward"))["rel_l2"] <= 1e-12
    r = x.real.copy()
    rd, hd, bd = torch.from_numpy(r).cuda(), torch.empty((b, nx, ny // 2 + 1), dtype=torch.complex128, device="cuda"), None
    with A.Plan.plan2d(b, nx, ny, A.D2Z) as p, A.Plan.plan2d(b, nx, ny, A.Z2D) as q:
        p.set_stream(st)
        q.set_stream(st)
        p.exec_d2z(rd, hd)
        bd = torch.empty_like(rd)
        q.exec_z2d(hd.clone(), bd)
    assert O.errors(hd.cpu().numpy(), np.fft.rfft2(r))["rel_l2"] <= 1e-12
    assert O.errors(bd.cpu().numpy(), r * nx * ny)["rel_l2"] <= 1e-12
