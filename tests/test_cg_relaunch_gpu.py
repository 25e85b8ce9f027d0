"""A whole solve in several launches: the iterates, counts and norms are one
launch's, to the last bit, whatever the iterations per launch (one; a few, with a
last launch of fewer; as many as the solve takes), for the one-cluster, the
all-SM and the mixed solves; and a solve that ended is not taken up again
without a new init."""

import numpy as np
import pytest

from gpu_util import ctx
from xyst_gb300 import cg, mesh
from xyst_gb300.lib import XgError

pytestmark = pytest.mark.gpu


def _system(n):
    m = mesh.cube(n, jitter=0.2, seed=n, numbering="random" if n == 41 else "rcm")
    ia, ja, a = cg.pressure_matrix(m["coord"], m["inpoel"])
    rng = np.random.default_rng(n)
    dn = np.unique(m["bface"][4])
    s = cg.ConjugateGradients(ctx(), ia, ja, a)
    s.set_guard("underflow")
    return s, rng.standard_normal(s.n), (dn, rng.standard_normal(dn.size))


# 9^3 and 20^3: one cluster (with empty blocks; full); 27^3, 41^3: all SMs,
# 16- and 32-bit columns; the mixed solve takes any
@pytest.mark.parametrize("n", [9, 20, 27, 41])
@pytest.mark.parametrize("kind", ["jacobi", "none", "mixed", "mixed factor"])
def test_same_bits_whatever_the_launches(n, kind):
    s, b, bc = _system(n)
    pc = kind.split()[-1] if kind != "mixed" else "jacobi"

    def solve(limit, maxit=40):
        s.set_launch_limit(limit)
        s.init(x=np.zeros(s.n), b=b, dirbc=bc, apply=True, pc=pc)
        if kind.startswith("mixed"):
            s.solve_mixed(20, 1e-9, inner_tol=1e-2, inner_maxit=maxit)
        else:
            s.solve(maxit, 1e-9)
        return s.solution(), s.it(), s.normr, s.converged()

    x, it, nr, conv = solve(0)
    assert 7 < it <= 40
    for limit in (1, 3, it, 1000):
        xl, itl, nrl, cl = solve(limit)
        assert np.array_equal(xl, x) and (itl, nrl, cl) == (it, nr, conv)
    x, it, nr, conv = solve(0, 2000)  # to the tolerance
    assert conv
    xl, itl, nrl, cl = solve(7, 2000)
    assert np.array_equal(xl, x) and (itl, nrl, cl) == (it, nr, conv)


def test_beyond_a_launch_of_the_default_length():
    """A chain of 20,000 unknowns: about as many iterations, three launches of
    the default length."""
    n = 20000
    ia = np.concatenate([[0, 2], 2 + 3 * np.arange(1, n - 1), [3 * n - 2]])
    ja = np.concatenate([[0, 1], (np.arange(1, n - 1)[:, None] + [-1, 0, 1]).ravel(),
                         [n - 2, n - 1]])
    a = np.where(ja == np.repeat(np.arange(n), np.diff(ia)), -2.0, 1.0)
    s = cg.ConjugateGradients(ctx(), ia, ja, a)
    s.set_guard("underflow")
    b = np.random.default_rng(0).standard_normal(n)
    got = []
    for limit in (0, 100000):
        s.set_launch_limit(limit)
        s.init(x=np.zeros(n), b=b, pc="jacobi")
        s.solve(60000, 1e-6)
        got.append((s.it(), s.normr, s.converged(), s.solution().tobytes()))
    assert got[0] == got[1] and got[0][2] and got[0][0] > 8192
    x = np.frombuffer(got[0][3])
    r = b - (-2 * x + np.append(x[1:], 0) + np.append(0, x[:-1]))
    # the recursive residual's tolerance and its distance from the true one: some
    # 20,000 iterations round each by a few u of the terms, with either sign
    size = np.abs(b) + 2 * np.abs(x) + np.abs(np.append(x[1:], 0)) + np.abs(np.append(0, x[:-1]))
    assert np.linalg.norm(r) < 1.1e-6 * np.linalg.norm(b) + 1e4 * 2.0 ** -53 * np.linalg.norm(size)


def test_ended_solve_stays():
    s, b, bc = _system(9)
    with pytest.raises(XgError):
        s.set_launch_limit(-1)
    s.init(x=np.zeros(s.n), b=b, dirbc=bc, apply=True, pc="jacobi")
    s.solve(7, 1e-12)
    x = s.solution()
    s.solve(100, 1e-12)
    assert s.it() == 7 and np.array_equal(s.solution(), x)
