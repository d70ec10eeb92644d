"""Zeros of the KEEP right-hand side keep their sign whichever pipe forms the
products: a state in the ranges of the integer-pipe form against the same state
with one cell outside them that no face reads (a corner of the primitives'
ghosts), which takes the FP64 form.

Tolerance: none, the bits are compared (-0 and +0 differ)."""
import numpy as np
import pytest
import torch

from amrsolver_gb300 import capi
from amrsolver_gb300 import problems as P

pytestmark = pytest.mark.gpu
CL = P.Closures.nondimensional(1e-2)
DXINV = (3.0, 5.0, 7.0)


def _state(kind, n, seed):
    rng = np.random.default_rng(seed)
    shape = (n[2] + 6, n[1] + 6, n[0] + 6)
    one, zero = np.ones(shape), np.zeros(shape)
    rho = rng.uniform(0.05, 0.95, shape)  # sums of two on both sides of one
    sign = np.where(rng.random(shape) < 0.5, 1.0, -1.0)
    if kind == "rest":
        f = (rho, zero, zero, zero, one)
    elif kind == "minus":  # at rest with either sign of zero
        f = (rho, sign * zero, -zero, sign * zero, one)
    elif kind == "along":  # one component moves, the others are zeros
        f = (rho, rng.uniform(-1, 1, shape), zero, -zero, one)
    else:  # sums of the velocities cancel along x
        s = np.where((np.arange(shape[2]) % 2) == 0, 1.0, -1.0)
        f = (rho, s * one, sign * zero, zero, one)
    return P.prims_to_cons(*f, 1.4)


@pytest.mark.parametrize("visc", [0, 1])
@pytest.mark.parametrize("order", [2, 4, 6])
def test_zero_signs(order, visc):
    capi.load(build_if_missing=True)
    n = (9, 6, 7)
    h = capi.Handle(P.Scheme(flux_euler=1, order_keep=order, rhs_visc=visc), CL)

    def rhs(U):
        out = torch.empty((5,) + tuple(s - 6 for s in U.shape[1:]), dtype=torch.float64, device="cuda")
        h.rhs_box(torch.from_numpy(U).cuda(), DXINV, out)
        h.sync_check()
        return out.cpu().numpy()

    g = max(order // 2, 2 if visc else 0)  # ghosts of the primitives
    c = P.NGHOST - g  # a corner of them: pairs run along axes, viscous cells reach one cell in two directions
    for kind in ("rest", "minus", "along", "opposed"):
        U = _state(kind, n, order)
        V = U.copy()
        V[1, c, c, c] = 1e-90  # outside the tested range
        a, b = rhs(U), rhs(V)
        assert np.isfinite(a).all()
        bad = a.view(np.int64) != b.view(np.int64)
        assert not bad.any(), (kind, int(bad.sum()), a[bad][:4], b[bad][:4])
    h.close()
