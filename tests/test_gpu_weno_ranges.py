"""The WENO5 face kernel keeps its products and quotients on the integer pipe
where one range test per value holds, and takes the hardware's operations
elsewhere; every value range has to give the oracle's bits.  Fields whose
smoothness differences are smooth, exactly zero, rounding noise (eps + beta in
between), beyond the tested range, tiny, and mixtures of these.

Tolerance: none.  Both sides perform the same correctly rounded operations in
the same order, so the bits are equal."""
import numpy as np
import pytest
import torch

from amrsolver_gb300 import capi
from amrsolver_gb300 import problems as P
from oracle import pyoracle

pytestmark = pytest.mark.gpu
N = (9, 6, 7)


def _state(kind):
    rng = np.random.default_rng(7)
    shape = (N[2] + 6, N[1] + 6, N[0] + 6)
    one, zero = np.ones(shape), np.zeros(shape)
    noise = lambda a: a * rng.uniform(-1, 1, shape)  # noqa: E731
    if kind == "smooth":
        f = (1 + noise(0.1), noise(0.3), noise(0.3), noise(0.3), 1 + noise(0.1))
    elif kind == "uniform":
        f = (one, 0.25 * one, zero, -0.5 * one, one)
    elif kind == "noise":
        f = (1 + noise(4e-16), 0.25 + noise(4e-16), noise(1e-17), noise(1e-30), 1 + noise(4e-16))
    elif kind == "faint":  # beta around eps = 1e-40 and around 2^-78
        f = (1 + noise(1e-13), noise(1e-20), noise(1e-12), 1e-16 * noise(1.0) ** 7, 1 + noise(1e-14))
    elif kind == "large":  # differences beyond 2^60
        f = (1 + noise(0.1), 1e9 * noise(1.0), 1e9 * noise(1.0), zero, 1e25 * (2 + noise(1.0)))
    elif kind == "small":
        f = (1e-30 * (2 + noise(1.0)), noise(1e-3), noise(1e-90), zero, 1e-33 * (2 + noise(1.0)))
    else:  # half the cells uniform, a jump between, single odd cells
        left = np.arange(shape[2]) < shape[2] // 2
        f = [np.where(left, a, b) for a, b in ((1.0, 0.125), (0.0, 0.0), (0.0, -0.0), (0.1, 0.1), (1.0, 0.1))]
        f = [np.broadcast_to(a, shape).copy() for a in f]
        f[0][5, 4, 6] += 1e-9
        f[4][6, 6, 3] += 1e-15
    return P.prims_to_cons(*f, 1.4)


@pytest.mark.parametrize("kind", ["smooth", "uniform", "noise", "faint", "large", "small", "jump"])
def test_rhs_bits(kind):
    capi.load(build_if_missing=True)
    U = _state(kind)
    sc = P.Scheme(flux_euler=2, rhs_visc=0)
    cl = P.Closures.nondimensional(1e-3)
    dxinv = (3.0, 5.0, 7.0)
    h = capi.Handle(sc, cl)
    out = torch.empty((5,) + N[::-1], dtype=torch.float64, device="cuda")
    h.rhs_box(torch.from_numpy(U).cuda(), dxinv, out)
    h.sync_check()
    ref = pyoracle.oracle().rhs(sc, cl, U, dxinv)
    assert np.isfinite(ref).all()
    assert np.array_equal(out.cpu().numpy(), ref), float(np.abs(out.cpu().numpy() - ref).max())
    h.close()
