"""The KEEP face kernels: the x kernel's blocks (row slots end to end, neighbours
overlapping) and the marches' column blocks at sizes around their edges, and the
range flag that moves a stage's products between the integer and the FP64
pipe, against the oracle.

Tolerance: none.  Both sides perform the same correctly rounded operations in
the same order, so the bits are equal."""
import numpy as np
import pytest
import torch

from amrsolver_gb300 import capi
from amrsolver_gb300 import problems as P
from oracle import pyoracle

pytestmark = pytest.mark.gpu
CL = P.Closures.nondimensional(1e-2)
DXINV = (3.0, 5.0, 7.0)


def _rhs(h, U):
    out = torch.empty((5,) + tuple(s - 6 for s in U.shape[1:]), dtype=torch.float64, device="cuda")
    h.rhs_box(torch.from_numpy(U).cuda(), DXINV, out)
    h.sync_check()
    return out.cpu().numpy()


@pytest.mark.parametrize("order", [2, 4, 6])
@pytest.mark.parametrize("n", [(1, 1, 1), (2, 3, 1), (31, 1, 2), (33, 3, 5), (62, 2, 1), (64, 1, 3), (7, 9, 11),
                               (255, 2, 2), (8, 33, 4), (5, 4, 40)])
def test_sizes(order, n):
    capi.load(build_if_missing=True)
    sc = P.Scheme(flux_euler=1, order_keep=order, rhs_visc=1)
    h = capi.Handle(sc, CL)
    U = P.random_state(n, seed=order)
    assert np.array_equal(_rhs(h, U), pyoracle.oracle().rhs(sc, CL, U, DXINV))
    h.close()


def _state(kind, n):
    rng = np.random.default_rng(3)
    shape = (n[2] + 6, n[1] + 6, n[0] + 6)
    r = lambda a: a * rng.uniform(-1, 1, shape)  # noqa: E731
    one, zero = np.ones(shape), np.zeros(shape)
    if kind == "rest":
        f = (1 + r(0.2), zero, zero, zero, 1 + r(0.2))
    elif kind == "plane":  # two components exactly zero, one sign of zero each
        f = (1 + r(0.2), r(0.5), zero, -zero, 1 + r(0.2))
    elif kind == "opposed":  # sums of velocities cancel to zero
        s = np.where((np.arange(shape[2]) % 2) == 0, 1.0, -1.0)
        f = (one, 0.5 * s * one, 0.25 * s * one, s * one, one)
    elif kind == "faint":  # velocities below the tested range
        f = (1 + r(0.2), r(1e-70), 1e-300 * r(1.0), r(0.1), 1 + r(0.2))
    elif kind == "huge":
        f = (1e31 * (2 + r(1.0)), r(1e10), r(1e10), r(1e10), 1e52 * (2 + r(1.0)))
    elif kind == "thin":
        f = (1e-32 * (2 + r(1.0)), r(0.1), r(0.1), r(0.1), 1e-33 * (2 + r(1.0)))
    elif kind == "one cell":  # a single ghost cell outside the ranges
        f = [1 + r(0.2), r(0.5), r(0.5), r(0.5), 1 + r(0.2)]
        f[1][4, 4, 1] = 1e-90
    else:
        f = (1 + r(0.2), r(0.5), r(0.5), r(0.5), 1 + r(0.2))
    return P.prims_to_cons(*f, 1.4)


@pytest.mark.parametrize("order", [2, 4, 6])
def test_ranges(order):
    """One handle, states in turn: a raised flag must reach its own stage and no later one wrongly."""
    capi.load(build_if_missing=True)
    n = (9, 6, 7)
    sc = P.Scheme(flux_euler=1, order_keep=order, rhs_visc=1)
    h = capi.Handle(sc, CL)
    for kind in ("smooth", "rest", "faint", "smooth", "plane", "huge", "one cell", "opposed", "thin", "smooth"):
        U = _state(kind, n)
        ref = pyoracle.oracle().rhs(sc, CL, U, DXINV)
        assert np.isfinite(ref).all()
        assert np.array_equal(_rhs(h, U), ref), kind
    h.close()


def test_nonfinite_passes_through():
    """NaN and infinity in the state reach the same cells as in the oracle."""
    capi.load(build_if_missing=True)
    n = (9, 6, 7)
    sc = P.Scheme(flux_euler=1, order_keep=4, rhs_visc=1)
    h = capi.Handle(sc, CL)
    for v in (np.nan, np.inf):
        U = _state("smooth", n)
        U[2, 6, 5, 7] = v
        ref = pyoracle.oracle().rhs(sc, CL, U, DXINV)
        got = _rhs(h, U)
        assert np.array_equal(np.isfinite(got), np.isfinite(ref))
        assert np.array_equal(got[np.isfinite(ref)], ref[np.isfinite(ref)])
    h.close()
