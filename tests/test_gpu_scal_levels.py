"""The scalar tile chooses the levels of a block by the grid's size, and the
positive-definite pass names its levels in words of at most 32: grids whose choice
is the smallest (4), a middle and the largest number of levels, with level counts
that end a chunk and one past it, columns one past a word and rows one past a
tile.  The advs entry and a step's tracers are the oracle's bit for bit (binary32
in the reference's order on both sides)."""
import ctypes as C

import numpy as np
import pytest

from cm1_b200.cases import make_case
from test_gpu_weno_values import _field

pytestmark = pytest.mark.gpu


def _torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("ni,nj,nk,bc", [(4, 4, 6, 1), (33, 8, 8, 2), (65, 15, 9, 1), (161, 113, 33, 2), (352, 240, 65, 1)])
def test_step_tracer_bitwise(ni, nj, nk, bc, cm1g, oracle_lib):
    torch = _torch()
    case = make_case("supercell", ni=ni, nj=nj, nk=nk, bc=bc, npt=2)
    rng = np.random.default_rng(ni)
    for n, kind in enumerate(("sparse", "smooth")):
        case.state["pta"][n] = case.state["pt3d"][n] = _field(kind, case.lay.shape(1), rng)
    ref, _, _ = oracle_lib.step(case)
    ctx = cm1g.Context(case.cfg, case.grid)
    dev = cm1g.to_device(case.state)
    ctx.step(dev, case.dt, case.mass1)
    torch.cuda.synchronize()
    sel = case.lay.interior(1)
    for n in range(2):
        assert np.array_equal(dev["pt3d"][n].cpu().numpy()[sel], ref["pt3d"][n][sel], equal_nan=True)
    ctx.close()


@pytest.mark.parametrize("pdef", [0, 1])
@pytest.mark.parametrize("ni,nj,nk,bc", [(4, 5, 6, 2), (32, 7, 8, 1), (33, 8, 17, 2), (225, 190, 33, 1)])
def test_advs_bitwise(ni, nj, nk, bc, pdef, cm1g, oracle_lib):
    _torch()
    case = make_case("dry_bubble", ni=ni, nj=nj, nk=nk, bc=bc, advwenos=1)
    lay = case.lay
    rng = np.random.default_rng(nk)
    # the caller's own fluxes: w's need not vanish at the bottom and top
    rru, rrv, rrw = (rng.normal(0, 8, lay.shape(s)).astype(np.float32) for s in (2, 3, 4))
    divx, sten = (rng.normal(0, 1e-3, lay.shape(1)).astype(np.float32) for _ in range(2))
    s = _field("sparse", lay.shape(1), rng)
    s0, weps, dt, ref = s.copy(), 1e-18, np.float32(0.5), sten.copy()
    g = case.grid_struct()
    fp = lambda a: a.ctypes.data_as(C.POINTER(C.c_float))       # noqa: E731
    assert oracle_lib.lib().oracle_advs(C.byref(case.cfg), C.byref(g), 1, 1, fp(rru), fp(rrv), fp(rrw), fp(divx), fp(s0),
                                        fp(s), fp(ref), pdef, pdef, dt, weps) == 0
    ctx = cm1g.Context(case.cfg, case.grid)
    d = cm1g.to_device(dict(rru=rru, rrv=rrv, rrw=rrw, divx=divx, s0=s0, s=s, sten=sten))
    ctx.advs(1, 1, d["divx"], d["rru"], d["rrv"], d["rrw"], d["s0"], d["s"], d["sten"], pdef, pdef, dt, weps)
    sel = lay.interior(1)
    assert np.array_equal(d["sten"].cpu().numpy()[sel], ref[sel], equal_nan=True)
    ctx.close()
