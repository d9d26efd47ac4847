"""The tile form of the acoustic kernel at the edges of its variants (7, 10 and
16 explicit warps; the last level of each; blocks of 1, 31, 32 and 33 columns)
against the column sweep.  Both evaluate every point with the same binary32
operations in the same order, so the results must agree bit for bit."""
import os
import subprocess
import sys

import numpy as np
import pytest

from cm1_b200.cases import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nj,nk,bc", [
    (33, 6, 6, 1),        # few tiles: 16 explicit warps, fewer levels than warps
    (31, 5, 128, 2),      # 16 warps, the most levels
    (32, 150, 7, 2),      # 7 warps, one round of levels
    (33, 80, 84, 1),      # 7 warps, the most levels
    (64, 75, 85, 2),      # 10 warps, the fewest levels
    (33, 76, 128, 1),     # 10 warps, the most levels
])
@pytest.mark.parametrize("nrk", [1, 3])
def test_tile_equals_column_sweep(ni, nj, nk, bc, nrk, cm1g, monkeypatch):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    case = make_case("dry_bubble", ni=ni, nj=nj, nk=nk, bc=bc)
    lay, st, gr = case.lay, case.state, case.grid
    rng = np.random.default_rng(ni + nk)

    def noise(amp, stag):
        a = rng.normal(0, amp, lay.shape(stag)).astype(np.float32)
        if stag == 4:
            a[lay.kx(1)] = a[lay.kx(nk + 1)] = 0.0
        return a

    A = {n: noise(a, q) for n, a, q in (("ua", 1.0, 2), ("va", 1.0, 3), ("wa", 0.2, 4), ("uten", 1e-3, 2), ("vten", 1e-3, 3),
                                        ("wten", 1e-2, 4), ("ppi", 1e-4, 1), ("ppx", 1e-5, 1), ("ppten", 1e-9, 1))}
    A.update(u3d=A["ua"] + noise(0.1, 2), v3d=A["va"] + noise(0.1, 3), w3d=A["wa"].copy(), pp3d=A["ppi"].copy())
    A["piadv"] = (gr["pi0"] + A["ppi"]).astype(np.float32)
    A["thv"] = (gr["th0"] + noise(0.5, 1)).astype(np.float32)
    A["ppterm"] = (A["piadv"] * np.float32(0.4)).astype(np.float32)
    A.update(rru=np.zeros_like(A["ua"]), rrv=np.zeros_like(A["va"]), rrw=np.zeros_like(A["wa"]))
    for n in ("radbcw", "radbce", "radbcs", "radbcn"):
        A[n] = st[n]
    ctx = cm1g.Context(case.cfg, case.grid)
    got = {}
    for form in ("tile", "col"):
        monkeypatch.setenv("CM1G_SOUND_FORM", form)
        d = cm1g.to_device(A)
        ctx.sound(nrk, case.dt, case.dt, **d)
        got[form] = cm1g.to_host(d)
    ctx.close()
    for n in ("u3d", "v3d", "w3d", "pp3d", "ppx", "rru", "rrv", "rrw"):
        assert np.isfinite(got["col"][n][lay.interior({"u3d": 2, "rru": 2, "v3d": 3, "rrv": 3, "w3d": 4}.get(n, 1))]).all(), n
        assert np.array_equal(got["tile"][n], got["col"][n]), n


TWO_CONTEXTS = """
import ctypes as C
import numpy as np
from cm1_b200 import binding
from cm1_b200.cases import make_case

case = make_case("dry_bubble", ni=40, nj=8, nk=100)     # over 48 KB of shared memory a block
cuda, ctx = C.CDLL("libcuda.so.1"), C.c_void_p()

def step():
    c = binding.Context(case.cfg, case.grid)
    st = {k: v.copy() for k, v in case.state.items()}
    c.step(st, case.dt, case.mass1)
    c.close()
    return st

first = step()
assert cuda.cuCtxCreate_v2(C.byref(ctx), 0, 0) == 0      # current from here on
second = step()
assert cuda.cuCtxDestroy_v2(ctx) == 0
assert all(np.array_equal(first[k], second[k], equal_nan=True) for k in first)
assert not np.array_equal(first["w3d"], case.state["w3d"])
print("same step")
"""


def test_every_cuda_context_gets_the_kernels_limits(cm1g):
    """A second CUDA context of a process (as a second device has one) launches
    tiles that take more shared memory than the default limit."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", TWO_CONTEXTS], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same step" in r.stdout, r.stdout + r.stderr
