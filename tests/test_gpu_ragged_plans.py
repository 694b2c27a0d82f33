"""Several ragged plans alive at once: what one plan sets up for its own
launches leaves the other plans' launches as they were."""
import numpy as np
import pytest

import aclfft as A
import oracle as O

torch = pytest.importorskip("torch")


def _plan(lengths):
    lens = np.array(lengths, np.int32)
    kinds = np.full(len(lens), A.C2C, np.int32)
    ino, outo, ci, _ = A.ragged_layout(lens, kinds)
    x = np.random.default_rng(len(lens)).standard_normal(ci // 4).astype(np.float32)
    p = A.RaggedPlan(lens, kinds, ino, outo)
    p.set_options(autotune=False, graph=False)
    p.set_stream(torch.cuda.current_stream())
    return p, lens, ino, x


def _check(p, lens, ino, x):
    xd = torch.from_numpy(x).cuda()
    yd = torch.zeros_like(xd)
    p.exec(xd, yd, A.FORWARD)
    assert p.error_flags() == 0
    y = yd.cpu().numpy()
    for n, o in zip(lens.tolist(), (ino // 4).tolist()):
        row = x[o:o + 2 * n].view(np.complex64)[None, :]
        e = O.errors(y[o:o + 2 * n].view(np.complex64), O.c2c(row, -1)[0])
        assert e["rel_l2"] <= 2.0 * 2.0 ** -24 * np.log2(n), (n, e)


@pytest.mark.gpu
def test_a_small_plan_does_not_shrink_the_limits_of_a_large_one():
    """Direct launches (no graph) of a plan with 48 KB or more of shared memory
    a CTA, before and after a plan with a few KB has been set up and run."""
    large, small = _plan([32768] * 4 + [4096] * 300), _plan([16] * 5)
    assert large[0].info().smem_bytes > 48 * 1024 > small[0].info().smem_bytes
    for p in (large, small, large, small):
        _check(*p)


@pytest.mark.parametrize("count,steps", [(1, 4), (10, 4), (38, 4), (39, 2), (76, 2), (77, 1), (1000, 1)])
def test_steps_of_few_long_transforms_are_cut(count, steps):
    """8192 points are two steps; a step is one item, or is cut into two or four
    while every item has a CTA of its own (304 of them)."""
    lens, kinds = np.full(count, 8192, np.int32), np.full(count, A.C2C, np.int32)
    ino, outo, _, _ = A.ragged_layout(lens, kinds)
    with A.RaggedPlan(lens, kinds, ino, outo) as p:
        assert p.check() == "ok" and p.info().items == 2 * steps * count


@pytest.mark.gpu
@pytest.mark.parametrize("lengths", [[8192], [8192] * 39, [4125, 5000, 8190, 9009], [16384, 7776, 100, 4096, 30, 2],
                                     [65536, 8748], [6561, 14641, 28561, 16807]])
@pytest.mark.parametrize("r2c", [False, True])
def test_few_long_transforms(lengths, r2c):
    """Tolerance: twice 2^-24 per radix-2 level."""
    lens = np.array(lengths, np.int32)
    kinds = np.full(len(lens), A.R2C if r2c else A.C2C, np.int32)
    ino, outo, ci, co = A.ragged_layout(lens, kinds)
    x = np.random.default_rng(len(lens)).standard_normal(ci // 4).astype(np.float32)
    xd, yd = torch.from_numpy(x).cuda(), torch.zeros(co // 4, device="cuda")
    with A.RaggedPlan(lens, kinds, ino, outo) as p:
        assert p.check() == "ok"
        p.set_options(autotune=False, graph=True)
        p.set_stream(torch.cuda.current_stream())
        for _ in range(2):  # the queue is left clear for the next launch
            yd.zero_()
            p.exec(xd, yd, A.FORWARD)
            assert p.error_flags() == 0
    y = yd.cpu().numpy()
    for n, i, o in zip(lens.tolist(), (ino // 4).tolist(), (outo // 4).tolist()):
        if r2c:
            out, exact = y[o:o + 2 * (n // 2 + 1)].view(np.complex64), np.fft.rfft(x[i:i + n].astype(np.float64))
        else:
            out = y[o:o + 2 * n].view(np.complex64)
            exact = np.fft.fft(x[i:i + 2 * n].view(np.complex64).astype(np.complex128))
        assert np.linalg.norm(out - exact) <= 2.0 * 2.0 ** -24 * np.log2(n) * np.linalg.norm(exact), n
