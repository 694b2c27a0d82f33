"""The register-to-register tile kernel (csrc/tile_fft.cuh) at the sizes where
it can go wrong: every radix alone and as first, inner and last radix, odd and
power-of-two paddings, rows and columns that do not fill a tile, one thread
per row, staged outputs and the outer-twiddle table of long transforms.

Tolerance: a radix-2 level rounds each output twice (one product, one sum), so
the relative L2 error of log2 N levels stays below 2 * 2^-24 * log2 N."""
import math

import numpy as np
import pytest

import aclfft as A
import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _bound(n):
    return 2.0 * 2.0 ** -24 * max(math.log2(n), 2.0)


def _ok(out, exact, n, what):
    e = O.errors(out, exact)
    assert e["rel_l2"] <= _bound(n), (what, e)


def _cplx(rng, *shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


# (length, rows): single radices, two radices of every kind in both places,
# three and four passes, the longest row of 512 threads; 1 row, a partly
# filled tile, more rows than one wave
ROWS = [(r, 5) for r in range(2, 17)] + [
    (18, 33), (20, 64), (22, 67), (26, 3), (28, 31), (30, 100), (32, 40000), (36, 7), (60, 1), (64, 1), (64, 70),
    (105, 9), (143, 4), (154, 300), (180, 2), (210, 1), (224, 17), (420, 50), (1000, 3), (1001, 2), (1155, 2),
    (1536, 4), (1859, 3), (2310, 301), (3000, 5), (3375, 2), (5040, 2), (6000, 3), (7680, 2)]


@pytest.mark.parametrize("n,b", ROWS)
def test_rows(n, b):
    rng = np.random.default_rng(n)
    x = _cplx(rng, b, n)
    xd = torch.from_numpy(x).cuda()
    with A.Plan.plan1d(n, A.C2C, b) as p:
        assert p.check() == "ok"
        p.set_stream(torch.cuda.current_stream())
        yd = torch.empty_like(xd)
        p.exec_c2c(xd, yd, A.FORWARD)
        zd = xd.clone()
        p.exec_c2c(zd, zd, A.BACKWARD)  # in place
    _ok(yd.cpu().numpy(), O.c2c(x, -1), n, ("fwd", n, b))
    _ok(zd.cpu().numpy(), O.c2c(x, 1), n, ("bwd", n, b))


@pytest.mark.parametrize("n,b", [(6, 5), (15, 9), (26, 33), (64, 70), (100, 31), (105, 9), (210, 1), (256 * 7, 3),
                                 (448, 5), (999, 3), (1001, 2), (2100, 1), (2310, 7), (4620, 3), (6720, 2), (12000, 2)])
def test_real_rows_and_adjoints(n, b):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((b, n)).astype(np.float32)
    X = _cplx(rng, b, n // 2 + 1)
    st = torch.cuda.current_stream()
    with A.Plan.plan1d(n, A.R2C, b) as p, A.Plan.plan1d(n, A.C2R, b) as q:
        assert p.check() == "ok" and q.check() == "ok"
        p.set_stream(st)
        q.set_stream(st)
        xd, Xd = torch.from_numpy(x).cuda(), torch.from_numpy(X).cuda()
        Yd, yd = torch.empty_like(Xd), torch.empty_like(xd)
        ad, bd = torch.empty_like(xd), torch.empty_like(Xd)
        p.exec_r2c(xd, Yd)
        q.exec_c2r(Xd, yd)
        p.exec_r2c_adjoint(Xd, ad)
        q.exec_c2r_adjoint(xd, bd)
    _ok(Yd.cpu().numpy(), O.r2c(x), n, ("r2c", n))
    _ok(yd.cpu().numpy(), O.c2r(X, n), n, ("c2r", n))
    w = np.full(n // 2 + 1, 2.0)
    w[0] = 1
    if n % 2 == 0:
        w[-1] = 1
    _ok(ad.cpu().numpy(), O.c2r((X / w).astype(np.complex128), n), n, ("r2c adjoint", n))
    _ok(bd.cpu().numpy(), O.r2c(x) * w, n, ("c2r adjoint", n))


@pytest.mark.parametrize("b,nx,ny", [(1, 30, 7), (3, 77, 33), (2, 143, 50), (1, 512, 19), (1, 1024, 130), (1, 2048, 66),
                                     (2, 169, 21), (5, 15, 100), (1, 1859, 12), (1, 16, 5000)])
def test_columns(b, nx, ny):
    rng = np.random.default_rng(nx)
    x = _cplx(rng, b, nx, ny)
    with A.Plan.plan2d(b, nx, ny) as p:
        assert p.check() == "ok"
        p.set_stream(torch.cuda.current_stream())
        xd = torch.from_numpy(x).cuda()
        yd = torch.empty_like(xd)
        p.exec_c2c(xd, yd, A.FORWARD)
    _ok(yd.cpu().numpy(), np.fft.fft2(x.astype(np.complex128)), nx * ny, (b, nx, ny))


# staged first passes (even and odd pass lengths), the outer-twiddle table and,
# above 2^20 points, the product of two tables
@pytest.mark.parametrize("n,b", [(14641, 3), (18432, 2), (46200, 5), (45045, 1), (131072, 3), (262144, 1), (1 << 21, 1)])
def test_long_rows(n, b):
    rng = np.random.default_rng(n)
    x = _cplx(rng, b, n)
    with A.Plan.plan1d(n, A.C2C, b) as p:
        assert p.check() == "ok"
        p.set_stream(torch.cuda.current_stream())
        xd = torch.from_numpy(x).cuda()
        yd = torch.empty_like(xd)
        p.exec_c2c(xd, yd, A.BACKWARD)
    _ok(yd.cpu().numpy(), np.fft.ifft(x.astype(np.complex128), norm="forward"), n, (n, b))


def test_columns_longer_than_4_gb():
    """256 strided samples whose span needs 64-bit offsets; sampled columns."""
    n, b = 256, (1 << 21) + 3
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    xd = torch.view_as_complex(torch.randn((n, b, 2), generator=g, device="cuda"))
    cols = torch.tensor([0, 1, 15, 16, 12345, b // 2, b - 17, b - 2, b - 1], device="cuda")
    want = np.fft.fft(xd[:, cols].cpu().numpy().astype(np.complex128), axis=0)
    with A.Plan.plan1d(n, A.C2C, b, A.VERTICAL) as p:
        assert p.check() == "ok"
        p.set_stream(torch.cuda.current_stream())
        p.exec_c2c(xd, xd, A.FORWARD)
    _ok(xd[:, cols].cpu().numpy(), want, n, "wide")


# ragged tiles: awkward radix sets (four passes, 11 and 13), tiles that do not
# divide a factor, outer twiddles as one table (to 2^16) and as a product
@pytest.mark.parametrize("kind", [A.C2C, A.R2C])
@pytest.mark.parametrize("lens", [[2, 2, 4, 6, 26, 3146, 4050, 4004, 4095], [4394, 4375, 5005, 8190, 30030, 32760],
                                  [131072, 148176, 155925, 13 ** 5]])
def test_ragged_tiles(lens, kind):
    rng = np.random.default_rng(len(lens))
    kinds = np.full(len(lens), kind, np.int32)
    ino, outo, ci, co = A.ragged_layout(lens, kinds)
    hin = rng.standard_normal(ci // 4).astype(np.float32)
    din, dout = torch.from_numpy(hin).cuda(), torch.zeros(co // 4, device="cuda")
    with A.RaggedPlan(np.array(lens, np.int32), kinds, ino, outo) as p:
        assert p.check() == "ok"
        p.set_options(autotune=False, graph=False)
        p.set_stream(torch.cuda.current_stream())
        p.exec(din, dout, A.FORWARD)
        assert p.error_flags() == 0
    hout = dout.cpu().numpy()
    for n, i, o in zip(lens, ino // 4, outo // 4):
        if kind == A.C2C:
            x, y = hin[i:i + 2 * n].view(np.complex64), hout[o:o + 2 * n].view(np.complex64)
            _ok(y, np.fft.fft(x.astype(np.complex128)), n, ("ragged c2c", n))
        else:
            y = hout[o:o + 2 * (n // 2 + 1)].view(np.complex64)
            _ok(y, np.fft.rfft(hin[i:i + n].astype(np.float64)), n, ("ragged r2c", n))


# the three ways items are claimed (none: at most one a CTA and no long
# transform; one by one; ahead), launched again on the queue the last left
@pytest.mark.parametrize("count,hi", [(40, 4096), (200, 16384), (3000, 32768)])
def test_ragged_claims(count, hi):
    lens, kinds = A.ragged_lengths(count, 16, hi, 0.7, 7)
    ino, outo, ci, co = A.ragged_layout(lens, kinds)
    g = torch.Generator(device="cuda")
    g.manual_seed(count)
    x = torch.randn(ci // 4, generator=g, device="cuda")
    ys = [torch.zeros(co // 4, device="cuda") for _ in range(3)]
    with A.RaggedPlan(lens, kinds, ino, outo) as p:
        p.set_stream(torch.cuda.current_stream())
        p.set_options(autotune=False, graph=False)
        assert p.check() == "ok"
        for y in ys:
            p.exec(x, y, A.FORWARD)
        assert p.error_flags() == 0
    assert torch.equal(ys[0], ys[1]) and torch.equal(ys[0], ys[2])
    h, o = x.cpu().numpy(), ys[0].cpu().numpy()
    for k in list(range(0, count, max(1, count // 60))) + [int(np.argmax(lens))]:
        n, a, b = int(lens[k]), int(ino[k]) // 4, int(outo[k]) // 4
        if int(kinds[k]) == int(A.C2C):
            want = np.fft.fft(h[a:a + 2 * n].view(np.complex64).astype(np.complex128))
            _ok(o[b:b + 2 * n].view(np.complex64), want, n, (count, k, n))
        else:
            want = np.fft.rfft(h[a:a + n].astype(np.float64))
            _ok(o[b:b + 2 * (n // 2 + 1)].view(np.complex64), want, n, (count, k, n))


# lengths with a codelet, whose rows in device memory run on the tile kernel
@pytest.mark.parametrize("n,b", [(128, 16383), (128, 16384), (256, 8192), (512, 16384), (1024, 8192), (2048, 4096),
                                 (4096, 2048), (8192, 63), (8192, 64)])
def test_rows_of_built_lengths(n, b):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    xd = torch.view_as_complex(torch.randn((b, n, 2), generator=g, device="cuda"))
    rows = [0, 1, b // 2, b - 2, b - 1]
    want = np.fft.ifft(xd[rows].cpu().numpy().astype(np.complex128), norm="forward")
    with A.Plan.plan1d(n, A.C2C, b) as p:
        assert p.check() == "ok"
        p.set_stream(torch.cuda.current_stream())
        p.exec_c2c(xd, xd, A.BACKWARD)
    _ok(xd[rows].cpu().numpy(), want, n, (n, b))


@pytest.mark.parametrize("n,b", [(256, 16384), (512, 8192), (8192, 512)])
def test_real_rows_of_built_lengths(n, b):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    xd = torch.randn((b, n), generator=g, device="cuda")
    Xd = torch.empty((b, n // 2 + 1), dtype=torch.complex64, device="cuda")
    yd = torch.empty_like(xd)
    rows = [0, 1, b // 2, b - 1]
    with A.Plan.plan1d(n, A.R2C, b) as p, A.Plan.plan1d(n, A.C2R, b) as q:
        assert p.check() == "ok" and q.check() == "ok"
        p.set_stream(torch.cuda.current_stream())
        q.set_stream(torch.cuda.current_stream())
        p.exec_r2c(xd, Xd)
        q.exec_c2r(Xd, yd)
        p.exec_r2c_adjoint_weighted(Xd, torch.ones((b, n // 2 + 1), device="cuda"), torch.empty_like(xd))
    _ok(Xd[rows].cpu().numpy(), np.fft.rfft(xd[rows].cpu().numpy().astype(np.float64)), n, (n, b))
    _ok(yd[rows].cpu().numpy(), n * xd[rows].cpu().numpy().astype(np.float64), n * n, (n, b))


# tiles compiled with their length: one row, a partial tile, both thread
# counts and the batches between which they change; weights on the adjoint
@pytest.mark.parametrize("L", [128, 256, 512, 1024, 1500, 2048, 4096])
def test_compiled_row_tiles(L):
    few = 152 * 256 // (L // (10 if L == 1500 else 16 if L in (256, 4096) else 8))
    for b in (1, 3, 9, few, few + 1):
        rng = np.random.default_rng(L + b)
        z = (rng.standard_normal((b, L)) + 1j * rng.standard_normal((b, L))).astype(np.complex64)
        x = rng.standard_normal((b, 2 * L)).astype(np.float32)
        w = rng.standard_normal((b, L + 1)).astype(np.float32)
        zd, xd, wd = (torch.from_numpy(v).cuda() for v in (z, x, w))
        Zd, Xd, yd, g1, g2 = (torch.empty_like(v) for v in (zd, torch.empty((b, L + 1), dtype=torch.complex64,
                                                                            device="cuda"), xd, xd, xd))
        with A.Plan.plan1d(L, A.C2C, b) as p, A.Plan.plan1d(2 * L, A.R2C, b) as r, A.Plan.plan1d(2 * L, A.C2R, b) as c:
            for q in (p, r, c):
                assert q.check() == "ok"
                q.set_stream(torch.cuda.current_stream())
            p.exec_c2c(zd, Zd, A.FORWARD)
            r.exec_r2c(xd, Xd)
            c.exec_c2r(Xd, yd)
            r.exec_r2c_adjoint_weighted(Xd, wd, g1)
            r.exec_r2c_adjoint(Xd * wd, g2)
            p.exec_c2c(zd, zd, A.FORWARD)
        assert torch.equal(zd, Zd) and torch.equal(g1, g2)
        X = np.fft.rfft(x.astype(np.float64))
        _ok(Zd.cpu().numpy(), np.fft.fft(z.astype(np.complex128)), L, ("c2c", L, b))
        _ok(Xd.cpu().numpy(), X, 2 * L, ("r2c", L, b))
        _ok(yd.cpu().numpy(), 2 * L * x.astype(np.float64), 4 * L * L, ("c2r", L, b))
        h = X * w * 0.5
        h[:, 0] *= 2
        h[:, -1] *= 2
        _ok(g1.cpu().numpy(), np.fft.irfft(h, 2 * L, norm="forward"), 4 * L * L, ("adjoint", L, b))


# columns of the compiled lengths and tile widths, as strided axes and as the
# passes of long rows (staged, with outer twiddles, paired real columns)
@pytest.mark.parametrize("nx,ny,b", [(128, 125, 40), (256, 72, 70), (256, 9, 2), (512, 80, 64), (512, 24, 128),
                                     (1024, 40, 64), (2048, 24, 64), (32, 30, 1), (512, 60, 1), (1024, 37, 1), (30, 1, 3)])
def test_compiled_column_tiles(nx, ny, b):
    rng = np.random.default_rng(nx)
    x = (rng.standard_normal((b, nx, ny)) + 1j * rng.standard_normal((b, nx, ny))).astype(np.complex64)
    xd = torch.from_numpy(x).cuda()
    with A.Plan.plan2d(b, nx, ny, A.C2C) as p:
        assert p.check() == "ok"
        p.set_stream(torch.cuda.current_stream())
        p.exec_c2c(xd, xd, A.BACKWARD)
    _ok(xd.cpu().numpy(), np.fft.ifft2(x.astype(np.complex128), norm="forward"), nx * ny, (nx, ny, b))


@pytest.mark.parametrize("n,b", [(1 << 17, 64), (1 << 18, 33), (1 << 20, 9), (1 << 22, 3)])
def test_compiled_long_tiles(n, b):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    z = torch.view_as_complex(torch.randn((b, n, 2), generator=g, device="cuda"))
    x = torch.randn((b, 2 * n), generator=g, device="cuda")
    Z, X, y = torch.empty_like(z), torch.empty((b, n + 1), dtype=torch.complex64, device="cuda"), torch.empty_like(x)
    with A.Plan.plan1d(n, A.C2C, b) as p, A.Plan.plan1d(2 * n, A.R2C, b) as r, A.Plan.plan1d(2 * n, A.C2R, b) as c:
        for q in (p, r, c):
            assert q.check() == "ok"
            q.set_stream(torch.cuda.current_stream())
        p.exec_c2c(z, Z, A.FORWARD)
        r.exec_r2c(x, X)
        c.exec_c2r(X, y)
    rows = [0, b // 2, b - 1]
    _ok(Z[rows].cpu().numpy(), np.fft.fft(z[rows].cpu().numpy().astype(np.complex128)), n, ("c2c", n, b))
    _ok(X[rows].cpu().numpy(), np.fft.rfft(x[rows].cpu().numpy().astype(np.float64)), 2 * n, ("r2c", n, b))
    _ok(y[rows].cpu().numpy(), 2 * n * x[rows].cpu().numpy().astype(np.float64), 4 * n * n, ("c2r", n, b))


# real rows of 16384: clusters below 64 (R2C) and 1024 (C2R) rows, rows in one
# CTA from there; of 131072: clusters below 8 rows, two passes from there; in
# place, and no weighted adjoint on any
@pytest.mark.parametrize("n,b", [(16384, 63), (16384, 64), (16384, 1023), (16384, 1024), (131072, 7), (131072, 8),
                                 (131072, 33)])
def test_real_rows_beside_clusters(n, b):
    nb, least = n // 2 + 1, (64, 1024) if n == 16384 else (8, 8)
    g = torch.Generator(device="cuda")
    g.manual_seed(b)
    x = torch.randn((b, n), generator=g, device="cuda")
    X = torch.empty((b, nb), dtype=torch.complex64, device="cuda")
    y, gd = torch.empty_like(x), torch.empty_like(x)
    io = torch.empty(b * nb * 2, device="cuda")
    with A.Plan.plan1d(n, A.R2C, b) as r, A.Plan.plan1d(n, A.C2R, b) as c:
        for q in (r, c):
            assert q.check() == "ok"
            q.set_stream(torch.cuda.current_stream())
        assert (r.info().cluster_ctas > 0) == (b < least[0]) and (c.info().cluster_ctas > 0) == (b < least[1])
        r.exec_r2c(x, X)
        c.exec_c2r(X, y)
        r.exec_r2c_adjoint(X, gd)
        with pytest.raises(A.AclfftError):
            r.exec_r2c_adjoint_weighted(X, torch.ones((b, nb), device="cuda"), gd)
        io[:b * n] = x.reshape(-1)
        r.exec_r2c(io, io)
        assert torch.equal(io, torch.view_as_real(X).reshape(-1))
        c.exec_c2r(io, io)
        assert torch.equal(io[:b * n], y.reshape(-1))
    rows = [0, b // 2, b - 1]
    xs = x[rows].cpu().numpy().astype(np.float64)
    h = np.fft.rfft(xs) * 0.5
    h[:, 0] *= 2
    h[:, -1] *= 2
    _ok(X[rows].cpu().numpy(), np.fft.rfft(xs), n, ("r2c", b))
    _ok(y[rows].cpu().numpy(), n * xs, n * n, ("c2r", b))
    _ok(gd[rows].cpu().numpy(), np.fft.irfft(h, n, norm="forward"), n * n, ("adjoint", b))


# paired columns: odd and even pass lengths and column counts on both sides,
# one item and several, adjoint weights, in place (through the workspace)
@pytest.mark.parametrize("n,b", [(2 * 14641, 2), (60060, 3), (90090, 1), (92400, 5), (98304, 2), (262144, 3),
                                 (2 * 15625, 4), (1 << 21, 1)])
def test_long_real_rows(n, b):
    rng = np.random.default_rng(n)
    nb = n // 2 + 1
    x = rng.standard_normal((b, n)).astype(np.float32)
    X = _cplx(rng, b, nb)
    st = torch.cuda.current_stream()
    w = np.full(nb, 2.0)
    w[0] = w[-1] = 1
    xd, Xd = torch.from_numpy(x).cuda(), torch.from_numpy(X).cuda()
    with A.Plan.plan1d(n, A.R2C, b) as p, A.Plan.plan1d(n, A.C2R, b) as q:
        assert p.check() == "ok" and q.check() == "ok" and p.info().nsteps == 2
        p.set_stream(st)
        q.set_stream(st)
        Yd, yd, ad, bd = torch.empty_like(Xd), torch.empty_like(xd), torch.empty_like(xd), torch.empty_like(Xd)
        p.exec_r2c(xd, Yd)
        q.exec_c2r(Xd, yd)
        p.exec_r2c_adjoint(Xd, ad)
        q.exec_c2r_adjoint(xd, bd)
        ip = torch.zeros(2 * nb * b, device="cuda")
        ip[:n * b] = xd.reshape(-1)
        p.exec_r2c(ip, ip)
        q.set_norm(A.NORM_BACKWARD)
        p.exec_r2c(xd, Yd)
        iq = torch.view_as_real(Yd).reshape(-1).clone()
        q.exec_c2r(iq, iq)
    assert torch.equal(torch.from_numpy(X).cuda(), Xd)
    _ok(Yd.cpu().numpy(), np.fft.rfft(x.astype(np.float64)), n, ("r2c", n))
    assert torch.equal(ip, torch.view_as_real(Yd).reshape(-1))
    assert torch.all(Yd[:, 0].imag == 0) and torch.all(Yd[:, -1].imag == 0)
    Xe = X.astype(np.complex128)
    _ok(yd.cpu().numpy(), n * np.fft.irfft(Xe, n), n, ("c2r", n))
    _ok(ad.cpu().numpy(), n * np.fft.irfft(Xe / w, n), n, ("r2c adjoint", n))
    _ok(bd.cpu().numpy(), np.fft.rfft(x.astype(np.float64)) * w, n, ("c2r adjoint", n))
    _ok(iq[:n * b].cpu().numpy().reshape(b, n), x.astype(np.float64), n * n, ("round trip", n))


# double precision: every radix, one and several passes, rows that do not fill
# a CTA, the longest rows of one launch, columns, even and odd real lengths,
# in place.  FP64 rounding is 2^-53: the same bound with that unit.
@pytest.mark.parametrize("n,b", [(r, 7) for r in range(2, 17)] + [(30, 33), (96, 5), (143, 2), (210, 70), (1000, 3), (1500, 2),
                                                                 (2310, 5), (3375, 1), (4096, 2), (7680, 1), (8192, 1)])
def test_double_rows(n, b):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((b, n)) + 1j * rng.standard_normal((b, n))
    r = rng.standard_normal((b, n))
    X = rng.standard_normal((b, n // 2 + 1)) + 1j * rng.standard_normal((b, n // 2 + 1))
    st = torch.cuda.current_stream()
    bound = 4.0 * 2.0 ** -53 * max(math.log2(n), 2.0)  # both sides round
    with A.Plan.plan1d(n, A.Z2Z, b) as p, A.Plan.plan1d(n, A.D2Z, b) as q, A.Plan.plan1d(n, A.Z2D, b) as s:
        assert p.check() == "ok" and q.check() == "ok" and s.check() == "ok"
        for h in (p, q, s):
            h.set_stream(st)
        xd, rd, Xd = torch.from_numpy(x).cuda(), torch.from_numpy(r).cuda(), torch.from_numpy(X).cuda()
        yd, zd, Rd, sd = torch.empty_like(xd), xd.clone(), torch.empty_like(Xd), torch.empty_like(rd)
        p.exec_z2z(xd, yd, A.FORWARD)
        p.exec_z2z(zd, zd, A.BACKWARD)
        q.exec_d2z(rd, Rd)
        s.exec_z2d(Xd, sd)
        ip = torch.zeros(2 * (n // 2 + 1) * b, dtype=torch.float64, device="cuda")
        ip[:n * b] = rd.reshape(-1)
        q.exec_d2z(ip, ip)
    for got, want in ((yd, np.fft.fft(x)), (zd, np.fft.ifft(x, norm="forward")), (Rd, np.fft.rfft(r)),
                      (sd, n * np.fft.irfft(X, n))):
        e = O.errors(got.cpu().numpy(), want)
        assert e["rel_l2"] <= bound, (n, b, e)
    e = O.errors(ip.cpu().numpy().view(np.complex128).reshape(b, -1), np.fft.rfft(r))
    assert e["rel_l2"] <= bound, (n, b, e)


@pytest.mark.parametrize("b,nx,ny", [(2, 33, 10), (1, 512, 7), (3, 60, 64), (1, 2048, 5), (1, 6000, 3)])
def test_double_columns(b, nx, ny):
    rng = np.random.default_rng(nx)
    x = rng.standard_normal((b, nx, ny)) + 1j * rng.standard_normal((b, nx, ny))
    xd = torch.from_numpy(x).cuda()
    with A.Plan.plan2d(b, nx, ny, A.Z2Z) as p:
        assert p.check() == "ok"
        p.set_stream(torch.cuda.current_stream())
        p.exec_z2z(xd, xd, A.FORWARD)
    e = O.errors(xd.cpu().numpy(), np.fft.fft2(x))
    assert e["rel_l2"] <= 4.0 * 2.0 ** -53 * math.log2(nx * ny), e
