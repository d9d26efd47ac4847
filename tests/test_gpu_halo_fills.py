"""The halo fills on the smallest grid, at odd sizes and one point past a block
of 128 rows or columns, with periodic, open, wall and mixed sides: every halo
point, the corners that keep or copy an older value included, is the reference's
bit for bit.  And a large step with walls and mixed sides, whose
positive-definite masses beyond the domain are read from the points that the
fills copy there."""
import ctypes as C

import numpy as np
import pytest

from cm1_b200.cases import Layout, make_case
from test_gpu_parity import TOL_RANGE, field_errors

pytestmark = pytest.mark.gpu

STAG = {"s": 1, "p": 1, "u": 2, "v": 3, "w": 4}
SIDES = [(1, 1, 1, 1), (2, 2, 2, 2), (1, 1, 2, 2), (2, 2, 1, 1), (3, 3, 1, 1), (2, 3, 3, 2)]


def _torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _case(sides, **over):
    case = make_case("dry_bubble", bc=sides[0], **over)
    c = case.cfg
    c.wbc, c.ebc, c.sbc, c.nbc = sides
    return case


@pytest.mark.parametrize("sides", SIDES)
@pytest.mark.parametrize("ni,nj,nk", [(4, 4, 6), (4, 129, 7), (123, 5, 6), (17, 30, 9)])
def test_fills_bitwise(ni, nj, nk, sides, cm1g, oracle_lib):
    _torch()
    case = _case(sides, ni=ni, nj=nj, nk=nk)
    ctx = cm1g.Context(case.cfg, case.grid)
    rng = np.random.default_rng(ni + nj)
    for code, which in enumerate("spuvw", 1):
        for flag in ((0, 1) if which == "w" else (0,)):
            a = rng.normal(size=case.lay.shape(STAG[which])).astype(np.float32)
            ref = a.copy()
            assert oracle_lib.lib().oracle_bc(C.byref(case.cfg), code, ref.ctypes.data_as(C.POINTER(C.c_float)), flag) == 0
            d = cm1g.to_device({"a": a})["a"]
            ctx.bc(which, d, flag)
            assert np.array_equal(d.cpu().numpy(), ref), (which, flag)
    ctx.close()


@pytest.mark.parametrize("sides", [(1, 1, 1, 1), (2, 2, 2, 2)])
@pytest.mark.parametrize("ni,nj,ngxy", [(4, 9, 5), (9, 4, 5), (4, 4, 4), (4, 5, 7)])
def test_wide_halos_bitwise(ni, nj, ngxy, sides, cm1g, oracle_lib):
    """Halos as wide as the domain, and wider: periodic points then copy halo points."""
    _torch()
    case = _case(sides, ni=ni, nj=nj, nk=6)
    case.cfg.ngxy, w = ngxy, ngxy - 3
    grid = {k: np.ascontiguousarray(np.pad(a, [(0, 0)] * max(0, a.ndim - 2) + [(w, w)] * min(2, a.ndim), mode="edge"))
            for k, a in case.grid.items()}
    lay = Layout(ni, nj, 6, ngxy)
    ctx = cm1g.Context(case.cfg, grid)
    rng = np.random.default_rng(ni + nj)
    for code, which in enumerate("spuvw", 1):
        a = rng.normal(size=lay.shape(STAG[which])).astype(np.float32)
        ref = a.copy()
        assert oracle_lib.lib().oracle_bc(C.byref(case.cfg), code, ref.ctypes.data_as(C.POINTER(C.c_float)), 1) == 0
        d = cm1g.to_device({"a": a})["a"]
        ctx.bc(which, d, 1)
        assert np.array_equal(d.cpu().numpy(), ref), which
    ctx.close()


@pytest.mark.parametrize("sides", [(3, 3, 3, 3), (2, 3, 4, 2)])
def test_step_with_walls(sides, cm1g, oracle_lib):
    torch = _torch()
    case = make_case("supercell", ni=33, nj=25, nk=20)
    c = case.cfg
    c.wbc, c.ebc, c.sbc, c.nbc = sides
    ref, _, _ = oracle_lib.step(case)
    ctx = cm1g.Context(case.cfg, case.grid)
    dev = cm1g.to_device(case.state)
    ctx.step(dev, case.dt, case.mass1)
    torch.cuda.synchronize()
    for f, e in field_errors(case, cm1g.to_host(dev), ref).items():
        assert e <= TOL_RANGE, (f, e)
    ctx.close()
