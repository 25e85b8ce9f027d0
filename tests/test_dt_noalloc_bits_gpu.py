"""xg_riecg_dt_noalloc returns xg_riecg_dt's number for an FP64 context, to the
last bit: both evaluate one formula."""

import ctypes as C

import numpy as np
import pytest

from gpu_util import cube_ops, pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 5, 13])
def test_same_bits(n):
    torch = pytest.importorskip("torch")
    ops = cube_ops(n)
    d, _ = pair(ops)
    rng = np.random.default_rng(n)
    vol = torch.as_tensor(ops["vol"], device="cuda")
    for _ in range(20):
        N = ops["vol"].size
        U = np.empty((N, 5))
        U[:, 0] = 10.0 ** rng.uniform(-3, 3, N)
        U[:, 1:4] = U[:, :1] * rng.standard_normal((N, 3))
        U[:, 4] = 10.0 ** rng.uniform(-3, 3, N) + 0.5 * (U[:, 1:4] ** 2).sum(1) / U[:, 0]
        d.set_state(U)
        Ud = torch.as_tensor(U, device="cuda")
        torch.cuda.synchronize()
        out = C.c_double(-1.0)
        rc = d.lib.xg_riecg_dt_noalloc(C.c_void_p(Ud.data_ptr()), C.c_void_p(vol.data_ptr()), N,
                                       1.4, 0.5, 0.0, None, C.byref(out))
        assert rc == 0 and out.value == d.dt()
