"""The mixed-precision solve's one-launch FP32 iteration where its work split
changes shape: fewer rows than a slice, a ragged last slice, fewer slices than
warps, one more slice than a block's warps take at once, columns beyond 16-bit
offsets, rows and triangles wider than what is staged in shared memory, and
triangles without entries; with and without the factored preconditioner.

The outer loop stops on the true FP64 residual, so the bound is the requested
one on ||b - A x||, plus the rounding of forming that residual twice (here and
on the device): at most (w + 2) eps of |A||x| + |b| per row of w entries."""

import numpy as np
import pytest

import oracle
from gpu_util import ctx
from xyst_gb300 import cg, mesh

pytestmark = pytest.mark.gpu


def _cube(n, numbering):
    m = mesh.cube(n, jitter=0.2, seed=n, numbering=numbering, perm_seed=n + 1)
    ia, ja, a = cg.pressure_matrix(m["coord"], m["inpoel"])
    rng = np.random.default_rng(n)
    dn = np.unique(m["bface"][4])
    return ia, ja, a, dn, rng.standard_normal(dn.size), rng.standard_normal(ia.size - 1)


def _graph(n, degree):
    """Negative definite, diagonally dominant, on a random symmetric graph."""
    rng = np.random.default_rng(n + degree)
    i = rng.integers(0, n, n * degree // 2)
    j = rng.integers(0, n, n * degree // 2)
    pairs = np.unique(np.stack([np.minimum(i, j), np.maximum(i, j)])[:, i != j], axis=1)
    w = rng.uniform(0.1, 1.0, pairs.shape[1])
    rows = np.concatenate([pairs[0], pairs[1], np.arange(n)])
    cols = np.concatenate([pairs[1], pairs[0], np.arange(n)])
    diag = np.full(n, 0.5)
    np.add.at(diag, pairs[0], w)
    np.add.at(diag, pairs[1], w)
    vals = np.concatenate([w, w, -diag])
    order = np.lexsort((cols, rows))
    ia = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=ia[1:])
    return ia, cols[order], vals[order], None, None, rng.standard_normal(n)


CASES = {"cube3": lambda: _cube(3, "lex"), "cube6": lambda: _cube(6, "rcm"),
         "cube16": lambda: _cube(16, "random"), "cube30": lambda: _cube(30, "rcm"),
         "cube41": lambda: _cube(41, "random"), "wide": lambda: _graph(1500, 36),
         "wide_far": lambda: _graph(70001, 24), "diagonal": lambda: _graph(203, 0),
         "large": lambda: _cube(56, "rcm")}


@pytest.mark.parametrize("case", list(CASES))
@pytest.mark.parametrize("pc", ["jacobi", "factor"])
def test_mixed_residual(case, pc):
    ia, ja, a, dn, dv, b = CASES[case]()
    if case in ("cube41", "wide_far"):
        rows = np.repeat(np.arange(ia.size - 1), np.diff(ia))
        assert np.abs(ja - rows).max() > 32768
    s = cg.ConjugateGradients(ctx(), ia, ja, a)
    s.set_guard("underflow")
    bc = None if dn is None else (dn, dv)
    s.init(x=np.zeros(s.n), b=b, dirbc=bc, apply=bc is not None, pc=pc)
    tol = 1e-8
    s.solve_mixed(60, tol, inner_tol=1e-3)
    assert s.converged()
    a2, b2 = (a, b) if dn is None else oracle.csr_dirichlet(ia, ja, a, b, dn, dv)
    x = s.solution()
    res = b2 - oracle.csr_mult(ia, ja, a2, x)
    width = int(np.diff(ia).max())
    size = np.abs(b2) + oracle.csr_mult(ia, ja, np.abs(a2), np.abs(x))
    rounding = 2 * (width + 2) * np.finfo(float).eps * np.linalg.norm(size)
    assert np.linalg.norm(res) < tol * np.linalg.norm(b2) + rounding


@pytest.mark.parametrize("pc", ["jacobi", "factor"])
def test_mixed_limit_and_repeat(pc):
    """An iteration limit ends the solve there, not converged; the same solve
    twice gives the same bits."""
    ia, ja, a, dn, dv, b = _cube(17, "rcm")
    s = cg.ConjugateGradients(ctx(), ia, ja, a)
    s.set_guard("underflow")
    s.init(x=np.zeros(s.n), b=b, dirbc=(dn, dv), apply=True, pc=pc)
    s.solve_mixed(60, 1e-8, inner_tol=1e-3, inner_maxit=7)
    assert not s.converged()
    xs = []
    for _ in range(2):
        s.init(x=np.zeros(s.n), b=b, dirbc=(dn, dv), apply=True, pc=pc)
        s.solve_mixed(60, 1e-8, inner_tol=1e-3)
        assert s.converged()
        xs.append(s.solution().copy())
    assert np.array_equal(xs[0], xs[1])
