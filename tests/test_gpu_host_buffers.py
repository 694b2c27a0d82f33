"""Host buffers of every kind (pageable or pinned, either side), at sizes around
the lines between one copy each way and chunks: 8 MB in and out, and 64 MB for a
pinned input with a pageable output.  In place too, where rows change pitch.

Tolerance: twice 2^-24 per radix-2 level."""
import numpy as np
import pytest

import aclfft as A

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _host(shape, dtype, pinned):
    t = torch.empty(shape, dtype=dtype)
    return t.pin_memory() if pinned else t


@pytest.mark.parametrize("pin_in,pin_out", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("n,b", [(8192, 8), (8192, 64), (8192, 512), (4096, 1024), (1500, 701), (2310, 333)])
def test_complex_rows(n, b, pin_in, pin_out):
    g = torch.Generator()
    g.manual_seed(n + b)
    x = _host((b, n), torch.complex64, pin_in)
    torch.view_as_real(x).normal_(generator=g)
    kept = x.clone()
    y = _host((b, n), torch.complex64, pin_out)
    with A.Plan.plan1d(n, A.C2C, b) as p:
        p.exec_c2c(x, y, A.FORWARD)
        assert torch.equal(x, kept)
        p.exec_c2c(x, x, A.FORWARD)  # in place
    exact = torch.fft.fft(kept.cuda().to(torch.complex128)).cpu()
    for out in (y, x):
        assert ((out - exact).norm() / exact.norm()).item() <= 2.0 * 2.0 ** -24 * np.log2(n)


@pytest.mark.parametrize("pin_in,pin_out", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("n,b", [(16384, 64), (16384, 600), (3000, 700), (2100, 1000)])
def test_real_rows(n, b, pin_in, pin_out):
    g = torch.Generator()
    g.manual_seed(n + b)
    x = _host((b, n), torch.float32, pin_in)
    x.normal_(generator=g)
    X = _host((b, n // 2 + 1), torch.complex64, pin_out)
    y = _host((b, n), torch.float32, pin_out)
    buf = _host(2 * X.numel(), torch.float32, pin_in)
    buf[:x.numel()] = x.flatten()
    with A.Plan.plan1d(n, A.R2C, b) as p, A.Plan.plan1d(n, A.C2R, b) as q:
        p.exec_r2c(x, X)
        q.exec_c2r(X, y)
        p.exec_r2c(buf, buf)  # in place
    exact = torch.fft.rfft(x.cuda().double()).cpu()
    tol = 2.0 * 2.0 ** -24 * np.log2(n)
    for out in (X, torch.view_as_complex(buf.view(b, n // 2 + 1, 2))):
        assert ((out - exact).norm() / exact.norm()).item() <= tol
    assert ((y - x.double() * n).norm() / (x.double() * n).norm()).item() <= 2 * tol
