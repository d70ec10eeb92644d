"""The slopes and the two-shock solver take their quotients, roots and products
on the integer pipe where a few range tests hold, and the hardware's elsewhere;
every state has to give the oracle's bits: smooth, uniform, rounding noise, very
large and very small values, at rest, supersonic both ways, transonic fans,
strong jumps.

Tolerance: none.  Both sides perform the same correctly rounded operations in
the same order, so the bits are equal."""
import numpy as np
import pytest
import torch

from amrsolver_gb300 import capi
from amrsolver_gb300 import problems as P
from oracle import pyoracle
from tests.test_gpu_weno_ranges import N
from tests.test_gpu_weno_ranges import _state as _weno_state

pytestmark = pytest.mark.gpu


def _state(kind):
    rng = np.random.default_rng(11)
    shape = (N[2] + 6, N[1] + 6, N[0] + 6)
    r = lambda a: a * rng.uniform(-1, 1, shape)  # noqa: E731
    zero = np.zeros(shape)
    if kind == "rest":
        f = (1 + r(0.3), zero, zero, zero, 1 + r(0.3))
    elif kind == "fast":
        f = (1 + r(0.2), np.where(r(1.0) > 0, 6.0, -6.0), 5 + r(0.5), -7 + r(0.5), 1 + r(0.2))
    elif kind == "fan":  # speeds around the sound speed
        f = (1 + r(0.5), 1.2 + r(0.4), -1.2 + r(0.4), r(1.5), 1 + r(0.6))
    elif kind == "strong":
        f = (10.0 ** r(3.0), r(3.0), r(3.0), r(3.0), 10.0 ** r(5.0))
    else:
        return _weno_state(kind)
    return P.prims_to_cons(*f, 1.4)


@pytest.mark.parametrize("weno", [0, 1])
@pytest.mark.parametrize("kind", ["smooth", "uniform", "noise", "faint", "large", "small", "jump", "rest", "fast", "fan",
                                  "strong"])
def test_rhs_bits(kind, weno):
    capi.load(build_if_missing=True)
    U = _state(kind)
    sc = P.Scheme(flux_euler=0, riemann_weno=weno, rhs_visc=0)
    cl = P.Closures.nondimensional(1e-3)
    dxinv = (3.0, 5.0, 7.0)
    h = capi.Handle(sc, cl)
    out = torch.empty((5,) + N[::-1], dtype=torch.float64, device="cuda")
    h.rhs_box(torch.from_numpy(U).cuda(), dxinv, out)
    h.sync_check()
    ref = pyoracle.oracle().rhs(sc, cl, U, dxinv)
    got = out.cpu().numpy()
    assert np.array_equal(got, ref, equal_nan=True), (np.argwhere(got != ref)[:5], float(np.nanmax(np.abs(got - ref))))
    h.close()
