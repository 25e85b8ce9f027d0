"""The one-launch FP64 solves (one cluster for a few thousand rows, all SMs for
systems whose rows fit their shared memory) against the oracle's PCG at the
sizes where the row split changes shape: one block with a ragged slice, a
cluster with empty blocks and with a ragged last one, the largest cluster, blocks
of the smallest row count, more rows than a block has threads, 32-bit columns (a bandwidth beyond
16 bits), several launches' worth of limits, and a solve continued after its
iteration limit.  Tolerances: both sides run the same recurrence in FP64 with
sums in another order, so counts agree and x to the accuracy of the solve
(1e-10 residual, amplified by at most the condition number's square root,
about n per side)."""

import numpy as np
import pytest

import oracle
from gpu_util import ctx, relerr
from xyst_gb300 import cg, mesh

pytestmark = pytest.mark.gpu


def _case(n, seed, numbering):
    m = mesh.cube(n, jitter=0.2, seed=seed, numbering=numbering, perm_seed=seed + 1)
    ia, ja, a = cg.pressure_matrix(m["coord"], m["inpoel"])
    rng = np.random.default_rng(seed)
    dn = np.unique(m["bface"][4])
    # scaled well above the oracle's absolute (p,q) breakdown guard
    # (src/LinearSolver/ConjugateGradients.cpp:681-690)
    return (ia, ja, a, dn, rng.standard_normal(dn.size) * 1e6,
            rng.standard_normal(ia.size - 1) * 1e7)


@pytest.mark.parametrize("n,numbering", [(2, "lex"), (3, "lex"), (5, "random"), (6, "rcm"),
                                         (8, "rcm"), (13, "random"), (18, "rcm"), (24, "rcm"),
                                         (27, "rcm"), (41, "random"), (55, "rcm")])
@pytest.mark.parametrize("pc", ["jacobi", "none"])
def test_loop_solve_matches_oracle(n, numbering, pc):
    ia, ja, a, dn, dv, b = _case(n, n, numbering)
    if numbering == "random" and n > 32:  # columns farther than 16 bits reach
        rows = np.repeat(np.arange(ia.size - 1), np.diff(ia))
        assert np.abs(ja - rows).max() > 32768
    s = cg.ConjugateGradients(ctx(), ia, ja, a)
    s.set_guard("underflow")
    s.init(x=np.zeros(s.n), b=b, dirbc=(dn, dv), apply=True, pc=pc)
    s.solve(20000, 1e-10)
    a2, b2 = oracle.csr_dirichlet(ia, ja, a, b, dn, dv)
    assert s.converged()
    x = s.solution()
    res = b2 - oracle.csr_mult(ia, ja, a2, x)
    assert np.linalg.norm(res) < 1.1e-10 * np.linalg.norm(b2)
    if n <= 27:
        xo, ito, *_ = oracle.pcg(ia, ja, a2, b2, np.zeros(s.n), 20000, 1e-10, pc)
        if pc == "jacobi":  # unscaled, the oracle's own count varies with the host's rounding
            assert abs(s.it() - ito) <= 1
        assert relerr(x, xo) < 1e-9 * n


def test_loop_solve_limits():
    """An iteration limit ends the solve there, not converged, with the
    iterate the oracle has after as many iterations; a zero right-hand side
    ends at once; the same solve gives the same bits again."""
    ia, ja, a, dn, dv, b = _case(9, 3, "rcm")
    s = cg.ConjugateGradients(ctx(), ia, ja, a)
    a2, b2 = oracle.csr_dirichlet(ia, ja, a, b, dn, dv)
    got = []
    for _ in range(2):
        s.init(x=np.zeros(s.n), b=b, dirbc=(dn, dv), apply=True, pc="jacobi")
        s.solve(7, 1e-12)
        assert s.it() == 7 and not s.converged()
        got.append(s.solution())
    assert np.array_equal(got[0], got[1])
    xo, ito, *_ = oracle.pcg(ia, ja, a2, b2, np.zeros(s.n), 7, 1e-12, "jacobi")
    assert relerr(got[0], xo) < 1e-12
    s.init(x=np.zeros(s.n), b=np.zeros(s.n), dirbc=(dn, 0 * dv), apply=True, pc="jacobi")
    s.solve(50, 1e-8)
    assert s.it() == 1 and np.array_equal(s.solution(), np.zeros(s.n))
