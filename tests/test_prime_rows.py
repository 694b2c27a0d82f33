"""2D and 3D transforms whose rows have a prime above 16: strided axes on the
column kernel (few points) and on tiles (many points, compiled lengths), and
both sides of the line of 2^18 column points between them.

Tolerance: a prime-p butterfly sums p products, so an output's relative error
stays below 2^-24 * (2 log2 N + p)."""
import numpy as np
import pytest

import aclfft as A

CASES = [(1, 32, 41), (14, 20, 86), (2, 90, 34), (3, 91, 34), (1, 16, 205), (5, 256, 23), (455, 24, 47),
         (60, 21, 19), (32, 30, 41), (21, 125, 82), (75, 96, 38), (64, 128, 17)]


@pytest.mark.parametrize("dims", CASES)
def test_launches_stay_in_bounds(dims):
    for typ in (A.C2C, A.R2C, A.C2R):
        for make in (A.Plan.plan2d, A.Plan.plan3d):
            with make(*dims, typ) as p:
                assert p.check() == "ok"


@pytest.mark.gpu
@pytest.mark.parametrize("flat", [True, False])
@pytest.mark.parametrize("dims", CASES)
def test_complex_and_real(dims, flat):
    torch = pytest.importorskip("torch")
    axes, make = ((1, 2), A.Plan.plan2d) if flat else ((0, 1, 2), A.Plan.plan3d)
    pts = int(np.prod(dims[1:] if flat else dims))
    tol = 2.0 ** -24 * (2 * np.log2(pts) + 47)
    g = torch.Generator(device="cuda")
    g.manual_seed(pts)
    st = torch.cuda.current_stream()
    z = torch.randn(dims, dtype=torch.complex64, generator=g, device="cuda")
    x = z.real.contiguous()
    X = torch.empty(dims[:2] + (dims[2] // 2 + 1,), dtype=torch.complex64, device="cuda")
    Z, y = torch.empty_like(z), torch.empty_like(x)
    with make(*dims, A.C2C) as c, make(*dims, A.R2C) as p, make(*dims, A.C2R) as q:
        for plan in (c, p, q):
            plan.set_stream(st)
        c.exec_c2c(z, Z, A.FORWARD)
        p.exec_r2c(x, X)
        q.exec_c2r(X, y)
        ref = z.to(torch.complex128)
        c.exec_c2c(z, z, A.FORWARD)  # in place
    assert torch.equal(z, Z)
    for out, exact, f in ((Z, torch.fft.fftn(ref, dim=axes), 1), (X, torch.fft.rfftn(x.double(), dim=axes), 1),
                          (y, x.double() * pts, 2)):
        assert ((out - exact).norm() / exact.norm()).item() <= f * tol
