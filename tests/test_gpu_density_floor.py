"""max(1e-40, rho) is taken by comparing bits: densities at, next to, below and
far from the floor, negative, infinite and NaN (which the floor replaces) give the
oracle's bits.  Tolerance: none, both sides round the same operations."""
import numpy as np
import pytest
import torch

from amrsolver_gb300 import capi
from amrsolver_gb300 import problems as P

pytestmark = pytest.mark.gpu
FLOOR = 1e-40


@pytest.mark.parametrize("rho", [0.0, -0.0, FLOOR, np.nextafter(FLOOR, 1), np.nextafter(FLOOR, 0), 5e-324, -1.0,
                                 1e300, np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("visc", [0, 1])
def test_rhs_bits(orc, rho, visc):
    capi.load(build_if_missing=True)
    n = (6, 5, 7)
    rng = np.random.default_rng(3)
    U = 1 + 0.1 * rng.uniform(-1, 1, (5, n[2] + 6, n[1] + 6, n[0] + 6))
    U[4] += 3
    U[0, 5, 6, 4] = rho
    sc = P.Scheme(flux_euler=1, order_keep=4, rhs_visc=visc)
    cl = P.Closures.nondimensional(1e-3)
    dxinv = (3.0, 5.0, 7.0)
    h = capi.Handle(sc, cl)
    out = torch.empty((5,) + n[::-1], dtype=torch.float64, device="cuda")
    h.rhs_box(torch.from_numpy(U).cuda(), dxinv, out)
    h.sync_check()
    with np.errstate(all="ignore"):
        ref = orc.rhs(sc, cl, U, dxinv)
    assert np.array_equal(out.cpu().numpy(), ref, equal_nan=True)
    h.close()
