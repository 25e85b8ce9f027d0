"""The FP64 edge flux node by node where two fluids of very different density and
pressure meet: each node's residual is held to the size of its own edges' and
triangles' terms, so that the thin fluid's errors are not measured against the
dense one's fluxes.

Bound: a term takes under 300 FP64 operations and a node adds under 100 of them:
400 * 2^-53 of the sum of the node's terms' sizes.  A term's size is |D| (|v| + c)
|U| + |D| p (1 + |v|) with each component's largest value at the edge's ends (the
limited states lie between them), each grown by the terms of the gradient's
projection on the edge, whose rounding the limiter passes on; at a triangle the
area's third takes the place of |D|."""

import numpy as np
import pytest

from gpu_util import cube_ops, pair

pytestmark = pytest.mark.gpu

G0 = 1.4


def _size(w):
    """(|v| + c) |U| + p (1 + |v|) from the largest density, velocity components
    and internal energy."""
    rho, v, e = w[..., 0], w[..., 1:4].sum(-1), w[..., 4]
    c, p = np.sqrt(G0 * (G0 - 1) * e), (G0 - 1) * rho * e
    U = rho * np.maximum(1.0, np.maximum(v, e + 0.5 * v * v))
    return (v + c) * U + p * (1.0 + v)


@pytest.mark.parametrize("scale", [1e-8, 1e-4, 1.0, 1e4])
@pytest.mark.parametrize("slope", ["own", 0.0])
@pytest.mark.parametrize("flux,stab2", [("rusanov", False), ("rusanov", True), ("hllc", False)])
def test_each_node_within_its_own_terms(scale, slope, flux, stab2):
    ops = cube_ops(9, seed=4)
    d, o = pair(ops, flux=flux, stab2=stab2)
    x = ops["coord"].T
    n = len(x)
    k = np.where(x[:, 0] < 0.5, scale, 1.0)
    W = np.empty((n, 5))
    W[:, 0] = k * (1.0 + 0.2 * np.sin(3 * x).sum(1) / 3)
    W[:, 1:4] = 0.1 * np.cos(2 * x + [0, 1, 2])
    W[:, 4] = (1.0 + 0.3 * np.sin(2 * x[:, 1] + x[:, 2])) / (G0 - 1)
    U = np.concatenate([W[:, :1], W[:, :1] * W[:, 1:4],
                        W[:, :1] * (W[:, 4:] + 0.5 * (W[:, 1:4] ** 2).sum(1)[:, None])], 1)
    G = o.grad(U) / ops["vol"][:, None] if slope == "own" else np.zeros((n, 15))
    e, D = ops["edges"], np.linalg.norm(ops["dint"], axis=1)
    v = x[e[:, 1]] - x[e[:, 0]]
    proj = [np.abs(G[e[:, j]].reshape(-1, 5, 3) * v[:, None]).sum(2) for j in (0, 1)]
    A = np.abs(W)
    term = D * _size(np.maximum(A[e[:, 0]], A[e[:, 1]]) + np.maximum(*proj))
    t = ops["tri"]
    area = 0.5 * np.linalg.norm(np.cross(x[t[:, 1]] - x[t[:, 0]], x[t[:, 2]] - x[t[:, 0]]), axis=1)
    tterm = area / 3 * _size(A[t].max(1))
    size = np.zeros(n)
    for j in (0, 1):
        np.add.at(size, e[:, j], term)
    for j in range(3):
        np.add.at(size, t[:, j], tterm)
    err = np.abs(d.rhs(G, U) - o.rhs(G, U)).max(1)
    assert np.all(err <= 400 * 2.0 ** -53 * size)
