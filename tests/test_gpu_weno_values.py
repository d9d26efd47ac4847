"""WENO5 values where the folded evaluation cannot decide the reference's last
bit by itself: uniform and nearly uniform stencils (candidate values a few units
of the last place apart, whose nominal weights sum to ties), fields that reach
from normal to subnormal numbers, isolated points in a field of zeros, and
values whose smoothness indicators exceed every bound.  The scalar pass and the
per-routine entry must return the oracle's binary32 numbers."""
import ctypes as C

import numpy as np
import pytest

from cm1_b200.cases import make_case
from test_gpu_routines import _adv_inputs

pytestmark = pytest.mark.gpu
f32 = np.float32


def _torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _field(kind, shape, rng):
    if kind == "ties":      # a few units of the last place around levels of a constant
        a = np.broadcast_to(f32(2.77e-5) * (1 + np.arange(shape[0])[:, None, None]), shape).astype(f32)
        return (a.view(np.int32) + rng.integers(0, 3, shape, dtype=np.int32)).view(f32)
    if kind == "tiny":      # 1e-3 down through the subnormal range to 0
        return (10.0 ** rng.uniform(-47, -3, shape)).astype(f32)
    if kind == "sparse":    # isolated values in zeros
        return np.where(rng.random(shape) < 0.03, rng.lognormal(-7, 1, shape), 0.0).astype(f32)
    if kind == "huge":      # smoothness up to 1e20 over neighbours of 0
        return (rng.lognormal(20, 3, shape) * (rng.random(shape) < 0.7)).astype(f32)
    x = np.linspace(0, 9, shape[2])     # smooth: candidate values agree to few digits more than binary32's
    return (1e-4 * (1.5 + np.sin(x))[None, None, :] * np.cos(np.linspace(0, 1, shape[1]))[None, :, None]
            * np.linspace(1, 2, shape[0])[:, None, None]).astype(f32)


KINDS = ["ties", "tiny", "sparse", "huge", "smooth"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("pdef", [0, 1])
def test_advs_bitwise(kind, pdef, cm1g, oracle_lib):
    _torch()
    case = make_case("dry_bubble", ni=61, nj=23, nk=17, bc=1, advwenos=1)
    rng = np.random.default_rng(5)
    rru, rrv, rrw, divx, _, _, sten = _adv_inputs(case, rng, positive=True)
    s = _field(kind, case.lay.shape(1), rng)
    s0, weps, dt, ref = s.copy(), 1e-18, f32(0.5), sten.copy()
    g = case.grid_struct()
    fp = lambda a: a.ctypes.data_as(C.POINTER(C.c_float))       # noqa: E731
    assert oracle_lib.lib().oracle_advs(C.byref(case.cfg), C.byref(g), 1, 1, fp(rru), fp(rrv), fp(rrw), fp(divx), fp(s0),
                                        fp(s), fp(ref), pdef, pdef, dt, weps) == 0
    ctx = cm1g.Context(case.cfg, case.grid)
    d = cm1g.to_device(dict(rru=rru, rrv=rrv, rrw=rrw, divx=divx, s0=s0, s=s, sten=sten))
    ctx.advs(1, 1, d["divx"], d["rru"], d["rrv"], d["rrw"], d["s0"], d["s"], d["sten"], pdef, pdef, dt, weps)
    sel = case.lay.interior(1)
    assert np.array_equal(d["sten"].cpu().numpy()[sel], ref[sel], equal_nan=True)
    ctx.close()


@pytest.mark.parametrize("bc", [1, 2])
def test_step_tracers_bitwise(bc, cm1g, oracle_lib):
    torch = _torch()
    case = make_case("supercell", ni=61, nj=23, nk=17, bc=bc, npt=len(KINDS))
    rng = np.random.default_rng(6)
    for n, kind in enumerate(KINDS):
        case.state["pta"][n] = case.state["pt3d"][n] = _field(kind, case.lay.shape(1), rng)
    ref, _, _ = oracle_lib.step(case)
    ctx = cm1g.Context(case.cfg, case.grid)
    dev = cm1g.to_device(case.state)
    ctx.step(dev, case.dt, case.mass1)
    torch.cuda.synchronize()
    sel = case.lay.interior(1)
    for n, kind in enumerate(KINDS):
        assert np.array_equal(dev["pt3d"][n].cpu().numpy()[sel], ref["pt3d"][n][sel], equal_nan=True), kind
    ctx.close()


@pytest.mark.parametrize("weps", [0.0, 5e-52, 1e-45, 1e-36, 1e-28])
@pytest.mark.parametrize("kind,scale", [("tiny", 1e-12), ("ties", 1e-12), ("sparse", 1e-18), ("smooth", 1e-16)])
def test_advs_small_weps(kind, scale, weps, cm1g, oracle_lib):
    """Values and denominators so small that the squares and sixth powers of the
    folded evaluation, or the smoothness indicators, leave the normal range."""
    _torch()
    case = make_case("dry_bubble", ni=61, nj=23, nk=17, bc=1, advwenos=1)
    rng = np.random.default_rng(11)
    rru, rrv, rrw, divx, _, _, sten = _adv_inputs(case, rng, positive=True)
    s = (_field(kind, case.lay.shape(1), rng) * f32(scale)).astype(f32)
    sten[...] = 0.0
    s0, dt, ref = s.copy(), f32(0.5), sten.copy()
    g = case.grid_struct()
    fp = lambda a: a.ctypes.data_as(C.POINTER(C.c_float))       # noqa: E731
    assert oracle_lib.lib().oracle_advs(C.byref(case.cfg), C.byref(g), 1, 1, fp(rru), fp(rrv), fp(rrw), fp(divx), fp(s0),
                                        fp(s), fp(ref), 0, 0, dt, weps) == 0
    ctx = cm1g.Context(case.cfg, case.grid)
    d = cm1g.to_device(dict(rru=rru, rrv=rrv, rrw=rrw, divx=divx, s0=s0, s=s, sten=sten))
    ctx.advs(1, 1, d["divx"], d["rru"], d["rrv"], d["rrw"], d["s0"], d["s"], d["sten"], 0, 0, dt, weps)
    sel = case.lay.interior(1)
    assert np.array_equal(d["sten"].cpu().numpy()[sel], ref[sel], equal_nan=True)
    ctx.close()


def _infinite(shape, rng):
    """A smooth field with isolated infinities of both signs, points that are not
    a number, and values near binary32's largest."""
    a = _field("smooth", shape, rng)
    p = rng.random(shape)
    for q, x in enumerate((np.inf, -np.inf, np.nan, 3e38)):
        a[(p >= 0.004 * q) & (p < 0.004 * (q + 1))] = x
    return a


@pytest.mark.parametrize("pdef", [0, 1])
def test_advs_infinite(pdef, cm1g, oracle_lib):
    """The divisions' infinities and not-a-numbers are those of the operator."""
    _torch()
    case = make_case("dry_bubble", ni=61, nj=23, nk=17, bc=1, advwenos=1)
    rng = np.random.default_rng(7)
    rru, rrv, rrw, divx, _, _, sten = _adv_inputs(case, rng, positive=True)
    s = _infinite(case.lay.shape(1), rng)
    s0, weps, dt, ref = s.copy(), 1e-18, f32(0.5), sten.copy()
    g = case.grid_struct()
    fp = lambda a: a.ctypes.data_as(C.POINTER(C.c_float))       # noqa: E731
    assert oracle_lib.lib().oracle_advs(C.byref(case.cfg), C.byref(g), 1, 1, fp(rru), fp(rrv), fp(rrw), fp(divx), fp(s0),
                                        fp(s), fp(ref), pdef, pdef, dt, weps) == 0
    sel = case.lay.interior(1)
    assert np.isinf(ref[sel]).sum() > 100 and np.isfinite(ref[sel]).sum() > 100
    ctx = cm1g.Context(case.cfg, case.grid)
    d = cm1g.to_device(dict(rru=rru, rrv=rrv, rrw=rrw, divx=divx, s0=s0, s=s, sten=sten))
    ctx.advs(1, 1, d["divx"], d["rru"], d["rrv"], d["rrw"], d["s0"], d["s"], d["sten"], pdef, pdef, dt, weps)
    assert np.array_equal(d["sten"].cpu().numpy()[sel], ref[sel], equal_nan=True)
    ctx.close()
