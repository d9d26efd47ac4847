"""The marching tile kernels (momentum, Smagorinsky tendencies, 2nd-order
diffusion), the statistics' chunks and the closure's backward pass at the edges
of their tiles: one point less than, exactly and one point more than the points
a block owns in x (30 or 31) and y (8, 10 or 15), the fewest levels, a level
count that ends a chunk and one past it, and more scalars than one launch
carries."""
import ctypes as C

import numpy as np
import pytest

import test_gpu_diff2 as diff2
import test_gpu_statpack as statpack
import test_gpu_turb as turb
from cm1_b200.cases import make_case
from oracle import mlp_ref

pytestmark = pytest.mark.gpu


def _torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("ni,nj,nk,bc", [(30, 7, 6, 1), (31, 8, 8, 2), (32, 9, 65, 1), (61, 15, 33, 2), (62, 16, 7, 1)])
def test_momentum_matches_oracle(ni, nj, nk, bc, cm1g, oracle_lib):
    """Binary32 in the reference's order on both sides: bit for bit."""
    _torch()
    case = make_case("dry_bubble", ni=ni, nj=nj, nk=nk, bc=bc)
    lay = case.lay
    rng = np.random.default_rng(ni)
    u, v, w = (rng.normal(0, 3, lay.shape(s)).astype(np.float32) for s in (2, 3, 4))
    w[lay.kx(1)] = w[lay.kx(nk + 1)] = 0.0
    ten = [rng.normal(0, 1e-3, lay.shape(s)).astype(np.float32) for s in (2, 3, 4)]
    ref = [t.copy() for t in ten]
    g = case.grid_struct()
    fp = lambda a: a.ctypes.data_as(C.POINTER(C.c_float))       # noqa: E731
    assert oracle_lib.lib().oracle_advuvw(C.byref(case.cfg), C.byref(g), fp(u), fp(v), fp(w), *[fp(r) for r in ref]) == 0
    ctx = cm1g.Context(case.cfg, case.grid)
    d = cm1g.to_device(dict(u=u, v=v, w=w, ut=ten[0], vt=ten[1], wt=ten[2]))
    ctx.advuvw(1, d["u"], d["v"], d["w"], d["ut"], d["vt"], d["wt"])
    op = int(bc != 1)
    K, J, I = slice(1, nk + 1), slice(3, 3 + nj), slice(3, 3 + ni)
    got = [d[n].cpu().numpy() for n in ("ut", "vt", "wt")]
    assert np.array_equal(got[0][K, J, 3 + op:4 + ni - op], ref[0][K, J, 3 + op:4 + ni - op])
    assert np.array_equal(got[1][K, 3 + op:4 + nj - op, I], ref[1][K, 3 + op:4 + nj - op, I])
    assert np.array_equal(got[2][2:nk + 1, J, I], ref[2][2:nk + 1, J, I])
    ctx.close()


@pytest.mark.parametrize("ni,nj,nk,npt", [(29, 9, 6, 0), (30, 10, 9, 2), (31, 15, 33, 3), (61, 16, 12, 6),
                                          (152, 91, 41, 2), (180, 130, 33, 1)])
def test_turbsmag_matches_oracle(ni, nj, nk, npt, cm1g, oracle_lib):
    """At the bar of test_gpu_turb (the log of N^2 is the only difference)."""
    torch = _torch()
    case = make_case("cbl", ni=ni, nj=nj, nk=nk, npt=npt)
    st = turb.les_state(case)
    rng = np.random.default_rng(3)
    ten = {n: rng.normal(0, 1e-3, st[n].shape).astype(np.float32) for n in ("uten1", "vten1", "wten1", "thten1")}
    ten["ptten"] = rng.normal(0, 1e-6, st["pta"].shape).astype(np.float32)
    ref, kmh_ref, kmv_ref = turb._run_oracle(oracle_lib, case, st, ten, 0.18, 2, 2, 2, 1)
    cgs, cgt = turb._cg(case)
    ctx = cm1g.Context(case.cfg, case.grid)
    d = cm1g.to_device(dict(st, **ten))
    lay = case.lay
    kmh, kmv = (torch.zeros(lay.shape(4), device="cuda") for _ in range(2))
    ctx.turbsmag(0.18, 2, 2, 2, 1, cgs, cgt, d["ua"], d["va"], d["wa"], d["rho"], d["tha"], d["pta"] if npt else None,
                 d["uten1"], d["vten1"], d["wten1"], d["thten1"], d["ptten"] if npt else None, kmh, kmv)
    torch.cuda.synchronize()
    for n, stag in (("uten1", 2), ("vten1", 3), ("wten1", 4), ("thten1", 1)):
        I = lay.interior(stag)
        assert turb._rel(d[n].cpu().numpy()[I], ref[n][I], ten[n][I]) <= turb.TOL, n
    for q in range(npt):
        I = lay.interior(1)
        assert turb._rel(d["ptten"].cpu().numpy()[q][I], ref["ptten"][q][I], ten["ptten"][q][I]) <= turb.TOL, q
    ring = (slice(None), slice(lay.jx(0), lay.jx(nj + 1) + 1), slice(lay.ix(0), lay.ix(ni + 1) + 1))
    for got, exp in ((kmh, kmh_ref[ring]), (kmv, kmv_ref[ring])):
        assert np.abs(got.cpu().numpy()[ring] - exp).max() <= turb.TOL * exp.max()
    ctx.close()


@pytest.mark.parametrize("name,over,bbc,tbc,idiff", [
    ("cbl", dict(ni=29, nj=9, nk=6, npt=0), 2, 1, 1),
    ("cbl", dict(ni=30, nj=10, nk=9, npt=2), 1, 2, 1),
    ("supercell", dict(ni=31, nj=11, nk=33, npt=5), 2, 2, 1),          # open boundaries, theta, qv and five tracers
    ("cbl", dict(ni=61, nj=20, nk=12, npt=3), 1, 1, 2),                # momentum only
])
def test_diff2_matches_oracle(name, over, bbc, tbc, idiff, cm1g, oracle_lib):
    diff2.test_diff2_matches_oracle(name, over, bbc, tbc, idiff, cm1g, oracle_lib)


@pytest.mark.parametrize("name,over,steps", [
    ("dry_bubble", dict(ni=6, nj=4, nk=6), 1),                         # fewer points than a block has threads
    ("dry_bubble", dict(ni=300, nj=4, nk=7), 1),                       # rows longer than a block, fewer rows than warps
    ("supercell", dict(ni=32, nj=33, nk=44, npt=2), 1),
    ("dry_bubble", dict(ni=4, nj=4, nk=8200, dz=1.0, npt=8), 0),       # more levels of tracers than a launch grid has rows
])
def test_statpack_matches_oracle(name, over, steps, cm1g, oracle_lib):
    statpack.test_statpack_matches_oracle(name, over, steps, cm1g, oracle_lib)


@pytest.mark.parametrize("n,shift", [(1, 0), (15, 0), (16, 1), (17, 0), (63, 1), (64, 0), (65, 0), (20000, 0)])
def test_backward_matches_reference(n, shift, cm1g):
    """Gradients from given pre-activations against the float64 restatement;
    arrays 4 bytes off an 8-byte boundary take the scalar accesses.  The dy,
    dz2 and dz1 operands are carried to 24 bits and sums are binary32, so a
    gradient is off by at most a few 2^-24 of the sum of its terms' magnitudes
    (64 terms an operand, then n rows): 1e-5 of the largest bounds that."""
    torch = _torch()
    rng = np.random.default_rng(n)
    p = mlp_ref.init_params(2)
    x = rng.normal(0, 0.3, (n, 8)).astype(np.float32)
    x[:, 7] = 0
    z1, z2 = (rng.normal(0, 1, (n, 64)).astype(np.float32) for _ in range(2))
    dy = rng.normal(0, 1, (n, 8)).astype(np.float32)

    def dev(a):
        b = torch.zeros(a.size + 4, device="cuda")[shift:shift + a.size]
        b.copy_(torch.from_numpy(a.ravel()))
        return b

    D = {k: dev(a) for k, a in dict(p=p, x=x, z1=z1, z2=z2, dy=dy).items()}
    G = torch.zeros(mlp_ref.P_TOTAL, device="cuda")
    f = cm1g.ptr
    cm1g.check(cm1g.lib().cm1g_mlp_backward(f(D["p"]), n, f(D["x"]), f(D["z1"]), f(D["z2"]), f(D["dy"]), f(G), None))
    torch.cuda.synchronize()
    got, exp = G.cpu().numpy(), mlp_ref.backward(p, x, z1, z2, dy)
    R = mlp_ref
    for a, b in ((R.P_W1, R.P_B1), (R.P_B1, R.P_W2), (R.P_W2, R.P_B2), (R.P_B2, R.P_W3), (R.P_W3, R.P_B3), (R.P_B3, R.P_TOTAL)):
        assert np.abs(got[a:b] - exp[a:b]).max() <= 1e-5 * np.abs(exp[a:b]).max(), (a, b)


@pytest.mark.parametrize("n", [1, 17, 200])
def test_backward_of_infinite_gradients(n, cm1g):
    """Infinite and not-a-number loss gradients of single rows, and one near
    binary32's largest value: the same entries of the parameter gradient are
    infinite, of either sign, and not a number as with unsplit operands, and the
    others keep the bar above."""
    torch = _torch()
    rng = np.random.default_rng(n)
    p = (mlp_ref.init_params(2) * 0.1).astype(np.float32)
    x = rng.uniform(0.1, 1, (n, 8)).astype(np.float32)
    x[:, 7] = 0
    z1, z2 = (rng.uniform(-0.5, 1, (n, 64)).astype(np.float32) for _ in range(2))
    for value in (np.inf, -np.inf, np.nan, 3.4e38):
        dy = np.zeros((n, 8), np.float32)
        dy[n // 2, 2] = value
        dy[0, 0] += 1.0
        D = {k: torch.from_numpy(a).cuda() for k, a in dict(p=p, x=x, z1=z1, z2=z2, dy=dy).items()}
        G = torch.zeros(mlp_ref.P_TOTAL, device="cuda")
        f = cm1g.ptr
        cm1g.check(cm1g.lib().cm1g_mlp_backward(f(D["p"]), n, f(D["x"]), f(D["z1"]), f(D["z2"]), f(D["dy"]), f(G), None))
        torch.cuda.synchronize()
        with np.errstate(all="ignore"):
            exp = mlp_ref.backward(p, x, z1, z2, dy)
        got, fin = G.cpu().numpy(), np.isfinite(exp)
        for pattern in (np.isnan, np.isposinf, np.isneginf):
            assert np.array_equal(pattern(got), pattern(exp)), (value, pattern)
        R = mlp_ref
        for a, b in ((R.P_W1, R.P_B1), (R.P_B1, R.P_W2), (R.P_W2, R.P_B2), (R.P_B2, R.P_W3), (R.P_W3, R.P_B3), (R.P_B3, R.P_TOTAL)):
            k = fin[a:b]
            if k.any():
                assert np.abs(got[a:b][k] - exp[a:b][k]).max() <= 1e-5 * np.abs(exp[a:b][k]).max(), (value, a, b)
