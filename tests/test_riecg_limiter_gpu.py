"""The FP64 edge flux's limiter, quotients and roots away from smooth flow:
fluids at rest and uniform fields (numerator and slope zero), plateaus with
jumps, density and pressure ratios up to 1e8, gradients of either sign and
far larger than the differences along the edges (the positivity test), and
none.  Bound: a flux takes under 300 FP64 operations and a node adds under 30
of them, so 300 * 30 * 2^-53 = 1e-12 of the largest term a flux can hold (the
residual of a uniform state is only the terms' rounding)."""

import numpy as np
import pytest

from gpu_util import cube_ops, pair

pytestmark = pytest.mark.gpu


def _conserved(rho, v, p, g=1.4):
    E = p / (g - 1.0) + 0.5 * rho * (v ** 2).sum(1)
    return np.concatenate([rho[:, None], rho[:, None] * v, E[:, None]], 1)


def _state(kind, n, rng):
    one, zero = np.ones(n), np.zeros((n, 3))
    if kind == "rest":
        return _conserved(one, zero, one)
    if kind == "uniform":
        return _conserved(1.3 * one, np.tile([0.3, -0.7, 1e-9], (n, 1)), 0.8 * one)
    if kind == "plateaus":
        lvl = rng.integers(0, 2, n)
        return _conserved(np.where(lvl, 1.0, 0.125), zero, np.where(lvl, 1.0, 0.1))
    return _conserved(10.0 ** rng.uniform(-4, 4, n), rng.uniform(-1, 1, (n, 3)),
                      10.0 ** rng.uniform(-4, 4, n))


def _largest_term(ops, U, g=1.4):
    """max |D| * max over nodes and components of (|v| + c) |u| + p (1 + |v|)."""
    v = np.abs(U[:, 1:4] / U[:, :1]).sum(1)
    p = (g - 1.0) * (U[:, 4] - 0.5 * (U[:, 1:4] ** 2).sum(1) / U[:, 0])
    c = np.sqrt(g * p / U[:, 0])
    return np.abs(ops["dint"]).max() * ((v + c) * np.abs(U).max(1) + p * (1.0 + v)).max()


@pytest.mark.parametrize("kind", ["rest", "uniform", "plateaus", "ratios"])
@pytest.mark.parametrize("slope", ["own", 0.0, 1e-9, 1.0, 1e6])
@pytest.mark.parametrize("flux,stab2", [("rusanov", False), ("hllc", True)])
def test_fp64_flux(kind, slope, flux, stab2):
    rng = np.random.default_rng(3)
    ops = cube_ops(7, seed=5)
    d, o = pair(ops, flux=flux, stab2=stab2)
    n = ops["coord"].shape[1]
    U = _state(kind, n, rng)
    if slope == "own":
        G = o.grad(U) / ops["vol"][:, None]
    else:
        G = slope * rng.uniform(-1, 1, (n, 15))
    assert np.abs(d.rhs(G, U) - o.rhs(G, U)).max() < 1e-12 * _largest_term(ops, U)
