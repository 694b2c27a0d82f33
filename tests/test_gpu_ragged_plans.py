"""Several ragged plans alive at once: what one plan sets up for its own
launches leaves the other plans' launches as they were."""
import numpy as np
import pytest

import aclfft as A
import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


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


def test_a_small_plan_does_not_shrink_the_limits_of_a_large_one():
    """Direct launches (no graph) of a plan with 48 KB or more of shared memory
    a CTA, before and after a plan with a few KB has been set up and run."""
    large, small = _plan([32768] * 4 + [4096] * 300), _plan([16] * 5)
    assert large[0].info().smem_bytes > 48 * 1024 > small[0].info().smem_bytes
    for p in (large, small, large, small):
        _check(*p)
