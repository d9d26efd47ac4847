"""The scalar tile chooses the levels of a block by the grid's size, and the
positive-definite pass names its levels in words of at most 32: grids whose choice
is the smallest (4; 1 for the advs entry without the positive-definite pass), some
between and the largest that the entry takes (16), with level counts that end a
chunk and one past it, columns one past a word and rows one past a tile; and words
of 16 and 32 levels that are named by the next chunk's alone.
The advs entry and a step's tracers are the oracle's bit for bit (binary32 in the
reference's order on both sides)."""
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


def _levels(cm1g, ni, nj, nk, most, fewest=4):
    """The library's own choice for 32 x 7 cells a block, three blocks an SM."""
    f = cm1g.lib()._ZN4cm1g11tile_levelsEliiiii
    f.argtypes, f.restype = [C.c_long] + [C.c_int] * 5, C.c_int
    return f(-(-ni // 32) * -(-nj // 7), nk, 3 * 148, 2, fewest, most)


@pytest.mark.parametrize("ni,nj,nk,bc,kc", [(4, 4, 6, 1, 4), (33, 8, 8, 2, 4), (65, 15, 9, 1, 4), (161, 113, 33, 2, 8),
                                            (352, 240, 65, 1, 30)])
def test_step_tracer_bitwise(ni, nj, nk, bc, kc, cm1g, oracle_lib):
    torch = _torch()
    assert _levels(cm1g, ni, nj, nk, 32) == kc
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


def _beside(q, k, up):
    """Tracer profiles whose only negative provisional mass lies at level k where
    air rises (up) through its upper face, or at k + 1 where it sinks through its
    lower one, and takes from the level across that face."""
    q[...] = 1e-6 * (1.0 + 0.01 * np.arange(q.shape[0], dtype=np.float32))[:, None, None]
    q[k if up else k + 1] = 0.0


@pytest.mark.parametrize("nk,k,bc", [(33, 32, 1), (65, 32, 2), (65, 64, 2)])
def test_step_across_words_of_32_levels(nk, k, bc, cm1g, oracle_lib):
    """Level k is bit 31 of a word, level k + 1 bit 0 of the next chunk's: each has
    to be named by the other's word alone."""
    torch = _torch()
    case = make_case("supercell", ni=45, nj=17, nk=nk, bc=bc, npt=2)
    case.dt = 0.5
    lay, st = case.lay, case.state
    for n in ("ua", "u3d", "va", "v3d", "wa", "w3d"):
        st[n][...] = 0.0
    for n in ("wa", "w3d"):
        st[n][lay.kx(k + 1), lay.jx(5):lay.jx(8), lay.ix(10):lay.ix(12)] = 10.0
        st[n][lay.kx(k + 1), lay.jx(12):lay.jx(14), lay.ix(38):lay.ix(41)] = -10.0
    for n, up in enumerate((True, False)):
        _beside(st["pta"][n], lay.kx(k), up)
        st["pt3d"][n] = st["pta"][n]
    sel = lay.interior(1)
    ref, _, _ = oracle_lib.step(case)
    case.cfg.pdtra = 0
    plain, _, _ = oracle_lib.step(case)
    case.cfg.pdtra = 1
    for n, level in enumerate((k + 1, k)):
        assert (ref["pt3d"][n] != plain["pt3d"][n])[sel][level - 1].any()      # the second pass has work there
        assert (plain["pt3d"][n][sel][level - 1] > 0).all()                    # and no mass of its own to name it
    ctx = cm1g.Context(case.cfg, case.grid)
    ctx.set_tune(adv_shape=4)
    dev = cm1g.to_device(st)
    ctx.step(dev, case.dt, case.mass1)
    torch.cuda.synchronize()
    for n in range(2):
        assert np.array_equal(dev["pt3d"][n].cpu().numpy()[sel], ref["pt3d"][n][sel], equal_nan=True)
    ctx.close()


@pytest.mark.parametrize("up", [True, False])
def test_advs_across_words_of_16_levels(up, cm1g, oracle_lib):
    _torch()
    ni, nj, nk, k = 225, 163, 33, 16
    assert _levels(cm1g, ni, nj, nk, 16) == k
    case = make_case("dry_bubble", ni=ni, nj=nj, nk=nk, bc=1, advwenos=1)
    lay = case.lay
    rru, rrv, rrw = (np.zeros(lay.shape(q), np.float32) for q in (2, 3, 4))
    rrw[lay.kx(k + 1), lay.jx(30):lay.jx(33), lay.ix(100):lay.ix(102)] = 10.0 if up else -10.0
    divx, sten, s = (np.zeros(lay.shape(1), np.float32) for _ in range(3))
    _beside(s, lay.kx(k), up)
    s0, weps, dt = s.copy(), 1e-18, np.float32(0.5)
    g = case.grid_struct()
    fp = lambda a: a.ctypes.data_as(C.POINTER(C.c_float))       # noqa: E731
    ref = {}
    for pdef in (0, 1):
        ref[pdef] = sten.copy()
        assert oracle_lib.lib().oracle_advs(C.byref(case.cfg), C.byref(g), 1, 1, fp(rru), fp(rrv), fp(rrw), fp(divx),
                                            fp(s0), fp(s), fp(ref[pdef]), pdef, 1, dt, weps) == 0
    sel = lay.interior(1)
    assert (ref[0] != ref[1])[sel][(k + 1 if up else k) - 1].sum() == 6
    ctx = cm1g.Context(case.cfg, case.grid)
    d = cm1g.to_device(dict(rru=rru, rrv=rrv, rrw=rrw, divx=divx, s0=s0, s=s, sten=sten))
    ctx.advs(1, 1, d["divx"], d["rru"], d["rrv"], d["rrw"], d["s0"], d["s"], d["sten"], 1, 1, dt, weps)
    assert np.array_equal(d["sten"].cpu().numpy()[sel], ref[1][sel], equal_nan=True)
    ctx.close()


@pytest.mark.parametrize("pdef", [0, 1])
@pytest.mark.parametrize("ni,nj,nk,bc,kc", [(4, 5, 6, 2, 4), (32, 7, 8, 1, 4), (33, 8, 17, 2, 4), (225, 190, 33, 1, 10),
                                            (225, 163, 33, 2, 16)])
def test_advs_bitwise(ni, nj, nk, bc, kc, pdef, cm1g, oracle_lib):
    _torch()
    assert _levels(cm1g, ni, nj, nk, 16) == kc and _levels(cm1g, ni, nj, nk, 16, 1) == (1 if kc == 4 else kc)
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
