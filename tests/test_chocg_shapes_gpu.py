"""ChoCG's node passes where their launch shape changes: every node a boundary
node, boundary lanes ending in mid-warp, a ragged last block, with each flux
and stabilisation option, with and without viscosity.  Bounds as in
test_chocg_gpu.py: the passes 1e-12 relative (summation order, one-ulp
quotients), steps with solves to 1e-10 within 1e-9."""

import numpy as np
import pytest

from gpu_util import ctx, relerr
from test_chocg_gpu import _cube_ops, _oracle, same_its
from xyst_gb300 import chocg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 8, 21])
@pytest.mark.parametrize("kw", [dict(flux="damp2", mu=0.0), dict(flux="damp2", mu=0.3, stab2=True),
                                dict(flux="damp4", mu=0.2),
                                dict(flux="damp4", mu=0.0, stab=False, stab2=True)])
def test_passes_match_oracle(n, kw):
    ops = _cube_ops(n)
    d = chocg.ChoCG(ctx(), ops, **kw)
    o = _oracle(ops, **kw)
    rng = np.random.default_rng(n)
    N = ops["coord"].shape[1]
    U, P = rng.standard_normal((N, 3)), rng.standard_normal(N)
    U[:, 1] = 0.7  # a uniform component: the damp4 reconstruction's zero differences
    G3, G9 = rng.standard_normal((N, 3)), rng.standard_normal((N, 9))
    assert relerr(d.grad(P), o.vgrad(P, 1).reshape(N, 3)) < 1e-12
    assert relerr(d.vgrad(U), o.vgrad(U, 3).reshape(N, 9)) < 1e-12
    assert relerr(d.flux(U, G9), o.flux(U, G9)) < 1e-12
    assert relerr(d.rhs(P, U, G9), o.rhs(U, G9, P)) < 1e-12
    for stab in (0, 1):
        assert relerr(d.div(U, P, G3, 0.01, stab), o.div(U, P, G3, 0.01, stab)) < 1e-12


@pytest.mark.parametrize("flux,rk", [("damp2", 1), ("damp4", 3)])
def test_steps_match_oracle(flux, rk):
    ops = _cube_ops(13)
    kw = dict(mu=0.02, cfl=0.5, flux=flux, rk=rk, pc="jacobi", ptol=1e-10, pmaxit=2000)
    d = chocg.ChoCG(ctx(), ops, **kw)
    o = _oracle(ops, **kw)
    u0 = chocg.taylor_green(ops["coord"])
    d.set_state(u0)
    o.set_state(u0, np.zeros(u0.shape[0]))
    assert same_its(d.init(), o.init())
    dts, its, _, _ = d.run(3)
    for k in range(3):
        dto, ito = o.step()
        assert abs(dts[k] / dto - 1) < 1e-12
        assert same_its(its[k], ito)
    u, p, _ = d.state()
    assert relerr(u, o.get(0)) < 1e-9
    assert relerr(p, o.get(2)) < 1e-9
