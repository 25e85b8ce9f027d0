"""The network's gradient kernels at the sizes where their tiles and
reductions change shape: fewer rows than one 128-row GEMM tile, a ragged last
tile, several tiles per block, and enough rows for several first-level chunks
of the edge reduction.  FP32 layers against the FP64 oracle with the bounds of
test_network_gradient_matches_oracle; BF16 layers against the FP32 ones with
the bounds of the tensor-core test (BF16 rounds each operand to 8 bits)."""

import numpy as np
import pytest

from oracle import lpc as olpc
from gpu_util import ctx
from test_lpc_gpu import _cg, _random_params, _system
from xyst_gb300 import lpc

pytestmark = pytest.mark.gpu


def _grad(s, theta, precision):
    model = lpc.LearnedPreconditioner(ctx(), precision=precision, params=theta)
    model.zero_grads()
    loss = model.grad(s)
    g = model.grads().astype(np.float64)
    model.close()
    return loss, g


@pytest.mark.parametrize("n,numbering", [(5, "random"), (8, "rcm"), (17, "random"), (23, "rcm")])
def test_gradient_shapes(n, numbering):
    S = _system(n=n, seed=n, numbering=numbering)
    s = _cg(S, "jacobi")
    theta = _random_params(n)
    g = olpc.Graph(S["ia"], S["ja"], S["a2"], S["mask"])
    lo, go, _ = olpc.loss_grad(theta.astype(np.float64), g)
    l32, g32 = _grad(s, theta, "fp32")
    l16, g16 = _grad(s, theta, "bf16")
    assert abs(l32 - lo) < 1e-5 * abs(lo)
    assert abs(l16 - lo) < 1e-2 * abs(lo)
    k = 0
    for name, shp in olpc.SHAPES:
        m = int(np.prod(shp))
        a, b, c = g32[k:k + m], go[k:k + m], g16[k:k + m]
        assert np.abs(a - b).max() <= 1e-3 * np.abs(go).max() + 1e-4 * np.abs(b).max(), name
        assert np.abs(c - b).max() <= 3e-2 * np.abs(go).max(), name
        k += m
