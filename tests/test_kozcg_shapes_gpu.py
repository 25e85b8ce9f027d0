"""KozCG's element and node passes where their launch shape changes: fewer
elements than one warp, a ragged last warp and block, sizes on either side of
the block-size lines, every limiter option, sources, Dirichlet beside symmetry
nodes, and components that are uniform (whose antidiffusive terms vanish).
Bounds as in test_kozcg_gpu.py: FP64 1e-12 relative (summation order and
one-ulp quotients), FP32 elements 1e-5 after a few smooth steps."""

import numpy as np
import pytest

import oracle
from common import random_state, wave_ic
from gpu_util import ctx, relerr
from test_oracle_pins import source_prm
from xyst_gb300 import kozcg, mesh, riecg

pytestmark = pytest.mark.gpu


def _pair(n, precision, seed=3, numbering="random", **kw):
    m = mesh.cube(n, jitter=0.2, seed=seed, numbering=numbering, perm_seed=seed)
    v = riecg.volumes(m["coord"], m["inpoel"])
    d = kozcg.KozCG(ctx(), m["coord"], v, m["inpoel"], cfl=0.1, precision=precision, **kw)
    o = oracle.KozCG(m["coord"], v, m["inpoel"], cfl=0.1, **kw)
    sym = oracle.sym_bc(m["coord"], m["bface"], [1, 2, 3, 4])[:2]
    dn = np.unique(m["bface"][5])
    mask = np.tile([1, 0, 1, 1, 0], (dn.size, 1)).astype(np.int32)
    val = wave_ic(m["coord"][:, dn])
    d.set_bc(sym=sym, dir=(dn, mask, val))
    o.set_sym(*sym)
    o.set_dir(dn, mask, val)
    return m, d, o


@pytest.mark.parametrize("n", [2, 3, 4, 12, 28])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kw", [dict(fct=True), dict(fct=False),
                                dict(fct=True, fctclip=True, fctsys=(0, 4), ctau=0.7)])
def test_steps_match_oracle(n, precision, kw):
    m, d, o = _pair(n, precision, **kw)
    U = wave_ic(m["coord"])
    for s in (d, o):
        s.set_state(U)
    tol = 1e-12 if precision == "fp64" else 1e-5
    dts, _ = d.run(3)
    assert np.allclose(dts, o.run(3), rtol=tol, atol=0)
    assert relerr(d.state()[0], o.state()) < tol
    R = random_state(U.shape[0], n)
    assert relerr(d.rhs(R, 1e-3), o.rhs(R, 1e-3)) < (1e-12 if precision == "fp64" else 1e-5)


def test_uniform_state_stays():
    """A uniform state without walls is a steady solution: its antidiffusive
    terms are exactly zero, so no limiter acts on rounding noise."""
    m = mesh.cube(9, jitter=0.2, seed=5)
    v = riecg.volumes(m["coord"], m["inpoel"])
    U = np.tile([1.0, 0.0, 0.0, 0.0, 2.5], (v.size, 1))
    for fctsys in ((), (0, 1, 2, 3, 4)):
        d = kozcg.KozCG(ctx(), m["coord"], v, m["inpoel"], fctsys=fctsys)
        o = oracle.KozCG(m["coord"], v, m["inpoel"], fctsys=fctsys)
        d.set_state(U)
        o.set_state(U)
        d.run(2)
        o.run(2)
        assert relerr(d.state()[0], o.state()) < 1e-12


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_source_terms(precision):
    m, d, o = _pair(6, precision, fct=True)
    U = wave_ic(m["coord"])
    for s in (d, o):
        s.set_source("taylor_green", source_prm("taylor_green"))
        s.set_state(U, 0.2)
    assert relerr(d.rhs(U, 1e-3), o.rhs(U, 1e-3)) < (1e-12 if precision == "fp64" else 2e-6)


@pytest.mark.parametrize("ne", [1, 63, 64, 65, 200])
@pytest.mark.parametrize("fct", [True, False])
def test_elements_without_shared_nodes(ne, fct):
    """The FP32 block sums where every element's nodes are its own (as many
    distinct nodes as a block can hold) and where the last block is ragged."""
    rng = np.random.default_rng(ne)
    corner = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], float)
    coord = (corner[None] + 0.1 * rng.random((ne, 4, 3)) +
             3.0 * np.arange(ne)[:, None, None]).reshape(-1, 3).T.copy()
    inpoel = rng.permutation(4 * ne).reshape(ne, 4)
    where = np.empty(4 * ne, np.int64)
    where[inpoel.reshape(-1)] = np.arange(4 * ne)
    coord = np.ascontiguousarray(coord[:, where])
    v = riecg.volumes(coord, inpoel)
    d = kozcg.KozCG(ctx(), coord, v, inpoel, precision="fp32", fct=fct)
    o = oracle.KozCG(coord, v, inpoel, fct=fct)
    U = random_state(v.size, ne)
    assert relerr(d.rhs(U, 1e-3), o.rhs(U, 1e-3)) < 1e-5
