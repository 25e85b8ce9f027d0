"""Contexts on different host threads solve at the same time: whatever another
thread's system needs, a solve's launches are accepted and give the bits that
the same solve gives alone.  Systems of several sizes on each side of the
line between the one-cluster and the all-SM solve, and mixed solves."""

import threading

import numpy as np
import pytest

from xyst_gb300 import cg, lib, mesh

pytestmark = pytest.mark.gpu


def _system(n, seed):
    m = mesh.cube(n, jitter=0.2, seed=seed)
    ia, ja, a = cg.pressure_matrix(m["coord"], m["inpoel"])
    rng = np.random.default_rng(seed)
    s = cg.ConjugateGradients(lib.Context(0), ia, ja, a)
    s.set_guard("underflow")
    return s, rng.standard_normal(s.n), np.unique(m["bface"][4])


def _solve(s, b, dn, mixed):
    s.init(x=np.zeros(s.n), b=b, dirbc=(dn, np.zeros(dn.size)), apply=True, pc="jacobi")
    if mixed:
        s.solve_mixed(5, 1e-6, inner_maxit=4)
    else:
        s.solve(3, 1e-30)
    return s.solution()


@pytest.mark.parametrize("sizes,mixed", [((9, 23, 15), False), ((27, 41, 30), False),
                                         ((9, 23, 41), True)])
def test_threads_with_systems_of_their_own(sizes, mixed):
    sys = [_system(n, n) for n in sizes]
    alone = [_solve(s, b, dn, mixed) for s, b, dn in sys]
    wrong = [None] * len(sys)
    go = threading.Barrier(len(sys))

    def work(k):
        s, b, dn = sys[k]
        try:
            go.wait()
            for _ in range(1500):
                if not np.array_equal(_solve(s, b, dn, mixed), alone[k]):
                    raise AssertionError(f"{sizes[k]}^3: other bits than alone")
        except Exception as e:
            wrong[k] = e

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sys))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == [None] * len(sys)
