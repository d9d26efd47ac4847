"""The step's reductions at the edges of their chunks: the Courant number's
maximum in the first and last cell and level of odd grids is found exactly (a
maximum has no order; sqrt and the products are the oracle's to a rounding), and
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
