"""Fluid at rest beside moving fluid: velocities through all decades down to the smallest
double, and rounding noise of any size around rest, in the schemes that keep their
operations on the integer pipe inside ranges.  Every state has to give the oracle's bits.
(The KEEP pairs' regrouped powers of two are exact for normal results only, on either pipe.)

Tolerance: none.  Both sides perform the same correctly rounded operations in the same
order, so the bits are equal."""
import numpy as np
import pytest
import torch

from amrsolver_gb300 import capi
from amrsolver_gb300 import problems as P
from oracle import pyoracle

pytestmark = pytest.mark.gpu
CL = P.Closures.nondimensional(1e-3)
DXINV = (3.0, 5.0, 7.0)
SCHEMES = {"muscl": dict(flux_euler=0), "weno_riemann": dict(flux_euler=0, riemann_weno=1), "weno": dict(flux_euler=2)}


def _state(kind, uniform):
    n = (90, 5, 6)
    rng = np.random.default_rng(17)
    shape = (n[2] + 6, n[1] + 6, n[0] + 6)
    r = lambda a: a * rng.uniform(-1, 1, shape)  # noqa: E731
    one = np.ones(shape)
    if kind == "rest":  # rho and gamma p a few units in the last place around one
        k = rng.integers(-9, 10, (2,) + shape) * 2.0**-53
        return P.prims_to_cons(1 + k[0], 0 * one, 0 * one, 0 * one, (1 + k[1]) / 1.4, 1.4)
    rho, p = (one, one / 1.4) if uniform else (1 + r(0.2), 1 + r(0.2))
    if kind == "tail":  # 10^-4 per cell along x, signs and factors at random
        dec = np.broadcast_to(-4.0 * np.arange(shape[2]), shape)
        with np.errstate(under="ignore"):
            v = [10.0 ** np.maximum(dec, -330.0) * r(1.0) for _ in range(3)]
    else:
        v = [r(1.0) * kind for _ in range(3)]
    with np.errstate(under="ignore"):
        return P.prims_to_cons(rho, *v, p, 1.4)


@pytest.mark.parametrize("kind", ["rest", "tail", 1e-28, 1e-35, 1e-42, 1e-61, 1e-78, 1e-118, 1e-123, 1e-148, 1e-155, 1e-200,
                                  1e-290, 1e-306, 1e-315])
@pytest.mark.parametrize("scheme", sorted(SCHEMES))
def test_bits(scheme, kind):
    capi.load(build_if_missing=True)
    sc = P.Scheme(rhs_visc=0, **SCHEMES[scheme])
    h = capi.Handle(sc, CL)
    for uniform in (True, False):
        U = _state(kind, uniform)
        out = torch.empty((5,) + tuple(s - 6 for s in U.shape[1:]), dtype=torch.float64, device="cuda")
        h.rhs_box(torch.from_numpy(U).cuda(), DXINV, out)
        h.sync_check()
        ref = pyoracle.oracle().rhs(sc, CL, U, DXINV)
        assert np.isfinite(ref).all()
        got = out.cpu().numpy()
        assert np.array_equal(got, ref), (uniform, int((got != ref).sum()), np.abs(got - ref).max(), np.argwhere(got != ref)[:4])
    h.close()
