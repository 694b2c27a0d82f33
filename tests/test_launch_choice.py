"""Which launch a plan makes, as aclfftGetPlanInfo reports it: lengths with a
specialised codelet run on compiled tiles in device memory unless a switch or
a tuned choice asks for the codelet."""
import numpy as np
import pytest

import aclfft as A


def _info(n, typ=A.C2C, b=4096):
    with A.Plan.plan1d(n, typ, b) as p:
        assert p.check() == "ok"
        return p.info()


@pytest.mark.parametrize("n,typ,rad,threads,rows", [
    (4096, A.C2C, [16, 16, 16], 256, 1), (512, A.C2C, [8, 8, 8], 32, 2), (1024, A.R2C, [8, 8, 8], 32, 2),
    (3000, A.C2R, [15, 10, 10], 150, 1)])
def test_info_describes_the_launch_of_device_buffers(n, typ, rad, threads, rows):
    """The radices, threads, rows and shared memory of the tile, not those of
    the codelet that pinned host buffers use; the codelet stays named."""
    i = _info(n, typ)
    L = int(np.prod(rad))
    assert i.kernel >= 0 and i.groups_per_cta == 0 and i.stages == 1
    assert [i.radix[k] for k in range(i.nradix)] == rad and i.onchip_length == L
    assert i.threads_per_transform == threads and i.transforms_per_cta == rows
    # at most one element of padding in eight, and two to a row
    assert rows * L * 8 <= i.smem_bytes <= rows * (L + L // 8 + 2) * 8
