"""A box whose scratch does not fit the device is refused with an error, nothing launched, and
leaves nothing behind: the same call fails the same way again, and a box that fits gives the
oracle's bits at once."""
import ctypes

import numpy as np
import pytest
import torch

from amrsolver_gb300 import capi
from amrsolver_gb300 import problems as P
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def test_refused_then_served():
    L = capi.load(build_if_missing=True)
    sc, cl, dxinv = P.Scheme(flux_euler=1, order_keep=4, rhs_visc=1), P.Closures.nondimensional(1e-2), (3.0, 5.0, 7.0)
    h = capi.Handle(sc, cl)
    n = (9, 6, 7)
    U = P.random_state(n, seed=1)
    ref = pyoracle.oracle().rhs(sc, cl, U, dxinv)
    Ud = torch.from_numpy(U).cuda()
    out = torch.empty((5,) + n[::-1], dtype=torch.float64, device="cuda")
    # 1284^3: 120 GB of primitives and 204 GB of viscous fluxes; the arrays are described, never touched
    e = 1284
    assert torch.cuda.get_device_properties(0).total_memory < 300e9
    bx = capi.c_box((0, 0, 0), (e, e, e))

    def described(g):
        m = e + 2 * g
        return capi.Array4(Ud.data_ptr(), m, m * m, m ** 3, (ctypes.c_int32 * 3)(-g, -g, -g),
                           (ctypes.c_int32 * 3)(e + g, e + g, e + g), 5)

    for _ in range(2):
        for _ in range(2):
            st = L.amrs_rhs_box(h.h, ctypes.byref(bx), capi.d3(dxinv), described(3), described(0), None)
            assert st == 6, st  # AMRS_ERR_CUDA
            assert b"out of memory" in L.amrs_last_cuda_error()
        out.fill_(7.0)
        h.rhs_box(Ud, dxinv, out)
        h.sync_check()
        assert np.array_equal(out.cpu().numpy(), ref)
    h.close()
