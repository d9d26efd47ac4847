"""The step's reductions at the edges of their chunks: the Courant number's
maximum is found wherever one cell dominates, in the first and last cell, row
and level of odd grids and on both sides of a block's edge in each direction, for
each wind component (sqrt and the products are the oracle's to a rounding); and
the clipping budgets are the oracle's with fewer and more rows and columns than
one tile."""
import numpy as np
import pytest

from cm1_b200.cases import make_case

pytestmark = pytest.mark.gpu


def _torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("ni,nj,nk", [(4, 4, 6), (33, 9, 8), (64, 8, 9), (31, 17, 17)])
def test_cfl_is_the_oracles(ni, nj, nk, cm1g, oracle_lib):
    _torch()
    case = make_case("supercell", ni=ni, nj=nj, nk=nk, bc=1)
    rng = np.random.default_rng(nk)
    for n in ("ua", "u3d", "va", "v3d"):
        case.state[n] += rng.normal(0, 2, case.state[n].shape).astype(np.float32)
    _, _, cfl_ref = oracle_lib.step(case)
    ctx = cm1g.Context(case.cfg, case.grid)
    _, cfl = ctx.step(cm1g.to_device(case.state), case.dt, case.mass1)
    assert abs(cfl - cfl_ref) <= 1e-6 * cfl_ref
    ctx.close()


CELLS = [(1, 1, 1), (32, 8, 8), (33, 9, 9), (37, 19, 17), (1, 19, 17), (37, 1, 16), (37, 19, 1)]


def _gust(case, wind, cell):
    """Winds of one cell in calm air (10 % less on the next cells of a w column,
    where the first and last level have one face that is not zero)."""
    lay, (i, j, k) = case.lay, cell
    for n in ("ua", "u3d", "va", "v3d", "wa", "w3d"):
        case.state[n][...] = 0.0
    J, I, nk = lay.jx(j), lay.ix(i), case.cfg.nk
    for t in ("a", "3d"):
        f = case.state[wind + t]
        if wind == "u":
            f[lay.kx(k), J, I:I + 2] = 40.0
        elif wind == "v":
            f[lay.kx(k), J:J + 2, I] = 40.0
        elif 1 < k < nk:
            f[lay.kx(k):lay.kx(k + 2), J, I] = 10.0
        else:
            faces = (2, 3, 4) if k == 1 else (nk, nk - 1, nk - 2)
            for face, w in zip(faces, (10.0, -10.0, 9.0)):
                f[lay.kx(face), J, I] = w


@pytest.mark.parametrize("wind", ["u", "v", "w"])
@pytest.mark.parametrize("nk", [16, 17])
@pytest.mark.parametrize("cell", CELLS)
def test_cfl_of_one_cell(cell, nk, wind, cm1g, oracle_lib):
    """Blocks are 32 x 8 x 8 cells; the last level ends one (nk 16) or is alone in
    one.  The step is so short that the winds stay as they are."""
    _torch()
    case = make_case("supercell", ni=37, nj=19, nk=nk, bc=1)
    case.dt = 0.01
    cell = (cell[0], cell[1], min(cell[2], nk))
    _gust(case, wind, cell)
    after, _, ref = oracle_lib.step(case)
    # the cell's number is the largest, by 5 % or more
    K, J, I = case.lay.interior(1)
    u, v, w = after["u3d"], after["v3d"], after["w3d"]
    e = lambda s: slice(s.start + 1, s.stop + 1)     # noqa: E731
    c = case.cfg
    cfl = 0.5 * case.dt * np.sqrt(((u[K, J, I] + u[K, J, e(I)]) / c.dx) ** 2 + ((v[K, J, I] + v[K, e(J), I]) / c.dy) ** 2
                                  + ((w[K, J, I] + w[e(K), J, I]) / c.dz) ** 2)
    assert np.unravel_index(cfl.argmax(), cfl.shape) == (cell[2] - 1, cell[1] - 1, cell[0] - 1)
    assert np.sort(cfl.ravel())[-2] <= 0.95 * cfl.max() and abs(cfl.max() - ref) <= 1e-5 * ref
    ctx = cm1g.Context(case.cfg, case.grid)
    _, got = ctx.step(cm1g.to_device(case.state), case.dt, case.mass1)
    assert abs(got - ref) <= 1e-6 * ref
    ctx.close()



@pytest.mark.parametrize("ni,nj,nk", [(15, 4, 6), (17, 129, 6), (32, 257, 6)])
def test_clipping_budget(ni, nj, nk, cm1g, oracle_lib):
    """At the bar of test_gpu_kessler's budgets."""
    _torch()
    case = make_case("kessler", ni=ni, nj=nj, nk=nk)
    rng = np.random.default_rng(ni)
    case.state["q3d"][1:] = rng.normal(2e-4, 3e-4, case.state["q3d"][1:].shape).astype(np.float32)
    ref = {k: v.copy() for k, v in case.state.items()}
    qb_ref, asq_ref = oracle_lib.mp_driver(case, ref)
    ctx = cm1g.Context(case.cfg, case.grid)
    ctx.mp_driver(cm1g.to_device(case.state), case.dt)
    _, asq = ctx.mp_budget()
    for a, b in zip(asq, asq_ref):
        assert a == pytest.approx(b, rel=1e-5, abs=1e-6 * max(abs(x) for x in qb_ref)), (asq, asq_ref)
    ctx.close()
