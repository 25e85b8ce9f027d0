"""What an edge hands to its two ends in ChoCG's passes: the same number with
opposite signs, to the last bit, so that an edge exchanges momentum and volume
and makes none.  On edges that share no node a node's sum is its one edge's
term."""

import numpy as np
import pytest

from gpu_util import ctx
from xyst_gb300 import chocg

pytestmark = pytest.mark.gpu

OPTS = [dict(flux="damp2", mu=0.0), dict(flux="damp2", mu=0.3, stab2=True),
        dict(flux="damp2", mu=0.1, stab=False), dict(flux="damp4", mu=0.2),
        dict(flux="damp4", mu=0.0, stab=False, stab2=True)]


@pytest.mark.parametrize("kw", OPTS)
def test_ends_receive_opposite_terms(kw):
    rng = np.random.default_rng(11)
    ne = 999
    n = 2 * ne
    e = rng.permutation(n).reshape(ne, 2)  # either end may have the smaller id
    none = np.zeros(0, np.int64)
    ops = {"coord": rng.uniform(0, 1, (3, n)), "vol": rng.uniform(0.5, 2, n), "edges": e,
           "dint": rng.standard_normal((ne, 5)), "tri": np.zeros((0, 3), np.int64),
           "matrix": (np.arange(n + 1), np.arange(n), -np.ones(n)),
           "dir": (none, np.zeros((0, 3), np.int32), np.zeros((0, 3))),
           "sym": (none, np.zeros((0, 3))), "noslip": none, "pdir": (none, np.zeros(0))}
    d = chocg.ChoCG(ctx(), ops, **kw)
    U, P = rng.standard_normal((n, 3)), rng.standard_normal(n)
    U[::7, 1] = 0.7
    G3, G9 = rng.standard_normal((n, 3)), rng.standard_normal((n, 9))
    for out in (d.rhs(P, U, G9), d.grad(P), d.vgrad(U), d.flux(U, G9), d.div(U, P, G3, 0.01, 0),
                d.div(U, P, G3, 0.01, 1)):
        out = np.asarray(out).reshape(n, -1)
        assert np.abs(out).max() > 0.1
        assert np.array_equal(out[e[:, 0]], -out[e[:, 1]])
