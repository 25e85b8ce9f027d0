"""RieCG's node passes where their launch shape changes: every node a boundary
node (2^3), one interior node (3^3), boundary lanes ending in mid-warp, the
sizes on either side of each block-size line (64, 128 and 256 threads on 152
multiprocessors), farfield, Dirichlet and pressure nodes beside symmetry, and
no boundary triangles at all.  Bounds: FP64 1e-12 relative (summation order
and one-ulp quotients); FP32 gradients entry by entry the a-priori bound of
their sums (grad_bound), FP32 residuals and steps the bounds of
test_dropin_fp32_bound and test_run_fp32_bound."""

import numpy as np
import pytest

from common import random_state, wave_ic
from gpu_util import cube_ops, ctx, pair, relerr
from xyst_gb300 import mesh, riecg
import oracle

pytestmark = pytest.mark.gpu


def grad_bound(ops, U):
    """|error| of an FP32 weak gradient: each term D (u_p + u_q) carries the
    roundings of its inputs, its sum and product (5), each of the node's terms
    one more per addition (degree + triangles, under 25 on these cubes):
    30 * 2^-24 * sum |D| (|u_p| + |u_q|), the boundary terms likewise, and
    there the FP32 coordinates (at most 1, so each difference is off by up to
    2 * 2^-24) in the triangle normals."""
    u = 2.0 ** -24
    w = np.abs(np.concatenate([U[:, :1], U[:, 1:4] / U[:, :1],
                               (U[:, 4:] / U[:, :1] +
                                0.5 * (U[:, 1:4] ** 2).sum(1, keepdims=True) / U[:, :1] ** 2)], 1))
    e, D, tri, x = ops["edges"], np.abs(ops["dint"]), ops["tri"], ops["coord"].T
    B = np.zeros((w.shape[0], 5, 3))
    t = (w[e[:, 0]] + w[e[:, 1]])[:, :, None] * D[:, None, :]
    np.add.at(B, e[:, 0], t)
    np.add.at(B, e[:, 1], t)
    ba, ca = (np.abs(x[tri[:, k]] - x[tri[:, 0]]) for k in (1, 2))
    nn = np.stack([ba[:, i] * ca[:, j] + ba[:, j] * ca[:, i]
                   for i, j in ((1, 2), (2, 0), (0, 1))], 1) / 48.0
    s = w[tri[:, 0]] + w[tri[:, 1]] + w[tri[:, 2]]
    dn = 2.0 * u * np.stack([ba[:, i] + ca[:, j] + ba[:, j] + ca[:, i]
                             for i, j in ((1, 2), (2, 0), (0, 1))], 1) / 48.0
    f = np.stack([(s + 5.0 * w[tri[:, k]]) * (nn + dn / (30.0 * u))[:, k:k + 1]
                  for k in range(3)], 2)
    for k in range(3):
        np.add.at(B, tri[:, k], f)
    return 30.0 * u * B.reshape(-1, 15)


@pytest.mark.parametrize("n", [2, 3, 9, 33, 35, 42, 44])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_dropins_and_steps(n, precision):
    ops = cube_ops(n, seed=n, numbering="lex")
    d, o = pair(ops, precision=precision)
    U = random_state(ops["coord"].shape[1], n)
    tr, ts = (1e-12, 1e-12) if precision == "fp64" else (1e-4, 1e-5)
    Go = o.grad(U)
    if precision == "fp64":
        assert relerr(d.grad(U), Go) < 1e-12
    else:
        assert np.all(np.abs(d.grad(U) - Go) <= grad_bound(ops, U))
    Gv = Go / ops["vol"][:, None]
    assert relerr(d.rhs(Gv, U), o.rhs(Gv, U)) < tr
    W = wave_ic(ops["coord"])
    for s in (d, o):
        s.set_state(W)
        s.bc()
    dts, _ = d.run(3)
    assert np.allclose(dts, o.run(3), rtol=ts)
    assert relerr(d.state()[0], o.state()) < ts


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_mixed_boundary_kinds(precision):
    ops = cube_ops(11, seed=4, sym=(2, 3), far=(1,), dirs=(4,), pres=(5,))
    far = (1.0, 0.5, 0.1, 0.0, 1.0)
    d, o = pair(ops, precision=precision, far_state=far,
                dir_vals=lambda x: wave_ic(x), pre_vals=(1.0, 1.0))
    for s in (d, o):
        s.set_state(wave_ic(ops["coord"]))
        s.bc()
    d.run(4)
    o.run(4)
    assert relerr(d.state()[0], o.state()) < (1e-12 if precision == "fp64" else 1e-5)


def test_no_boundary_triangles():
    m = mesh.cube(7, jitter=0.2, seed=2)
    ops = riecg.operators({**m, "bface": {}})
    d = riecg.from_operators(ctx(), ops)
    o = oracle.RieCG(ops["coord"], ops["vol"], ops["edges"], ops["dint"], ops["tri"],
                     ops["besym"])
    U = random_state(ops["coord"].shape[1], 5)
    G = o.grad(U)
    assert relerr(d.grad(U), G) < 1e-12
    Gv = G / ops["vol"][:, None]
    assert relerr(d.rhs(Gv, U), o.rhs(Gv, U)) < 1e-12
