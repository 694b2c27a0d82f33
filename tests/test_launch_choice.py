"""Which launch a plan makes, as aclfftGetPlanInfo reports it: lengths with a
specialised codelet run on compiled tiles in device memory unless a switch or
a tuned choice asks for the codelet."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

import aclfft as A

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


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


@pytest.mark.parametrize("name,value,field,want", [
    ("OPS_FFT_CODELET_VARIANT", "0", "groups_per_cta", None), ("OPS_FFT_CODELET_NG", "2", "groups_per_cta", 2),
    ("OPS_FFT_CODELET_NST", "3", "stages", 3), ("OPS_FFT_CODELET_PP", "1", "groups_per_cta", None),
    ("OPS_FFT_FUSE_R2C", "0", "groups_per_cta", None)])
def test_codelet_switches_act_on_device_buffers(name, value, field, want, monkeypatch):
    monkeypatch.setenv(name, value)
    i = _info(2048, A.R2C)
    assert i.kernel >= 0 and i.groups_per_cta >= 1
    assert want is None or getattr(i, field) == want


_NO_CODELETS = r"""
import json, sys
sys.path[:0] = [sys.argv[1] + "/ops-fft_gb300"]
import aclfft as A
out = []
for n in (4096, 2310):
    with A.Plan.plan1d(n, A.C2C, 4096) as p:
        i = p.info()
        out.append([p.check(), i.kernel, i.groups_per_cta, i.smem_bytes, i.transforms_per_cta * i.onchip_length * 8])
print(json.dumps(out))
"""


def test_no_codelets_means_the_generic_row_kernel():
    """OPS_FFT_CODELETS=0 (read once per process): prefetch slots and ping-pong
    buffers in shared memory, at least twice a tile's one exchange buffer."""
    env = dict(os.environ, OPS_FFT_CODELETS="0")
    r = subprocess.run([sys.executable, "-c", _NO_CODELETS, ROOT], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    for check, kernel, groups, smem, rows in json.loads(r.stdout.strip().splitlines()[-1]):
        assert check == "ok" and kernel == -1 and groups == 0 and smem >= 2 * rows


_WEIGHTED = r"""
import sys
sys.path[:0] = [sys.argv[1] + "/ops-fft_gb300", sys.argv[1] + "/oracle"]
import numpy as np, torch, aclfft as A, oracle as O
n, b = 1024, 64
rng = np.random.default_rng(n)
X = (rng.standard_normal((b, n // 2 + 1)) + 1j * rng.standard_normal((b, n // 2 + 1))).astype(np.complex64)
w = rng.random((b, n // 2 + 1), dtype=np.float32)
with A.Plan.plan1d(n, A.R2C, b) as p:
    p.set_autotune(True)
    assert p.info().tuned == 1 and p.check() == "ok"
    print("candidates", p.info().tune_candidates)
    Xd, wd, gd = torch.from_numpy(X).cuda(), torch.from_numpy(w).cuda(), torch.empty((b, n), device="cuda")
    torch.cuda.synchronize()
    p.exec_r2c_adjoint_weighted(Xd, wd, gd)
    torch.cuda.synchronize()
half = np.full(n // 2 + 1, 0.5)
half[0] = half[-1] = 1.0
e = O.errors(gd.cpu().numpy(), O.c2r((X * w * half).astype(np.complex128), n))
assert e["rel_l2"] <= 1e-6, e
"""


@pytest.mark.gpu
@pytest.mark.parametrize("choice", ["-1 0 0 0 -1 0 -1", "-1 15 4 -1 -1 0 1"])
def test_weighted_adjoint_of_a_tuned_plan(choice, tmp_path):
    """Whatever tuning chose for the R2C itself, its weighted adjoint runs as it
    did before tuning: after a tuning of its own, and with cached choices of no
    codelets and of a codelet shape that does not fit shared memory."""
    pytest.importorskip("torch")
    path = tmp_path / "plan_tune.txt"
    env = dict(os.environ, OPS_FFT_PLAN_TUNE_CACHE=str(path))

    def child():
        r = subprocess.run([sys.executable, "-c", _WEIGHTED, ROOT], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        return r.stdout

    child()
    key = path.read_text().splitlines()[-1].split()[0]
    path.write_text(f"{key} {choice}\n")
    assert "candidates 0" in child()


_TUNE_PLAN = r"""
import sys
sys.path[:0] = [sys.argv[1] + "/ops-fft_gb300"]
import aclfft as A
with A.Plan.plan1d(1024, A.R2C, 512) as p:
    p.set_autotune(True)
    print("candidates", p.info().tune_candidates)
"""

_TUNE_RAGGED = r"""
import sys
sys.path[:0] = [sys.argv[1] + "/ops-fft_gb300", sys.argv[1] + "/oracle"]
import numpy as np, torch, aclfft as A, oracle as O
lens = np.array([1500, 1500, 18000], np.int32)
kinds = np.full(3, A.C2C, np.int32)
ino, outo, ci, co = A.ragged_layout(lens, kinds)
x = np.random.default_rng(1).standard_normal(ci // 4).astype(np.float32)
xd, yd = torch.from_numpy(x).cuda(), torch.zeros(co // 4, device="cuda")
with A.RaggedPlan(lens, kinds, ino, outo) as p:
    p.set_stream(torch.cuda.current_stream())
    p.exec(xd, yd, A.FORWARD)
    assert p.error_flags() == 0 and p.info().tuned_classes == 2
y = yd.cpu().numpy()
for n, i, o in zip(lens.tolist(), (ino // 4).tolist(), (outo // 4).tolist()):
    e = O.errors(y[o:o + 2 * n].view(np.complex64), O.c2c(x[i:i + 2 * n].view(np.complex64)[None], -1)[0])
    assert e["rel_l2"] <= 1e-6, (n, e)
"""


def _run_child(code, **env):
    r = subprocess.run([sys.executable, "-c", code, ROOT], env=dict(os.environ, **env), capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout


@pytest.mark.gpu
def test_plan_choices_of_other_kernels_are_not_used(tmp_path):
    """A tune file written before the launches changed has no version: it is
    tuned again, and the file then holds lines that are used."""
    pytest.importorskip("torch")
    path = tmp_path / "plan_tune.txt"
    env = {"OPS_FFT_PLAN_TUNE_CACHE": str(path)}
    _run_child(_TUNE_PLAN, **env)
    line = path.read_text().splitlines()[-1]
    path.write_text(line.split(":", 1)[1] + "\n" if line.startswith("v") else line + "\n")
    assert "candidates 0" not in _run_child(_TUNE_PLAN, **env)
    assert "candidates 0" in _run_child(_TUNE_PLAN, **env)


@pytest.mark.gpu
def test_ragged_choices_name_their_radices(tmp_path):
    """A ragged tune file of candidate indices (as written before), one with
    radices that the length does not have, and one of this version."""
    pytest.importorskip("torch")
    path = tmp_path / "ragged_tune.txt"
    for old in ("0 1500 1 0\n0 18000 1 1\n", "r 0 1500 15.10.9\nr 0 18000 150.120\n"):
        path.write_text(old)
        for _ in range(2):  # tuned again, then read back
            _run_child(_TUNE_RAGGED, OPS_FFT_TUNE_CACHE=str(path))
            lines = [line.split() for line in path.read_text().splitlines()]
            assert [line[:3] for line in lines] == [["r", "0", "1500"], ["r", "0", "18000"]], lines
            for _, _, n, radices in lines:
                product = 1
                for r in radices.replace("+", ".").split("."):
                    product *= int(r)
                assert product == int(n) and radices.count("+") == int(int(n) > 4096)
