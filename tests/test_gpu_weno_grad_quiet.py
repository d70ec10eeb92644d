"""The WENO5 gradient around fluid at rest: momenta whose smoothness differences lie
below the bound under which they enter the weights as a constant (2^-130), just above
it, and on both sides of it within a stencil, beside uniform density and pressure.

Check and tolerance as in test_gpu_weno_grad_ranges: <v, J w> = <J^T v, w> within 1e-11
of |<v, J w>| + |v| |J w|, J w from 100 digits."""
import numpy as np
import pytest
import torch

from amrsolver_gb300 import capi
from amrsolver_gb300 import problems as P

pytestmark = pytest.mark.gpu
ranges = pytest.importorskip("tests.test_gpu_weno_grad_ranges")
N = ranges.N


@pytest.mark.parametrize("kind", [1e-35, 1e-39, 1e-42, 1e-60, 1e-200, 1e-312, "tail"])
def test_vjp_dot_product(kind):
    capi.load(build_if_missing=True)
    rng = np.random.default_rng(19)
    shape = (N[2] + 6, N[1] + 6, N[0] + 6)
    one = np.ones(shape)
    scale = 10.0 ** (-3.0 * np.arange(shape[2]) - 26.0) if kind == "tail" else kind
    U = P.prims_to_cons(one, *(scale * rng.uniform(-1, 1, shape) for _ in range(3)), one, 1.4)
    sc, cl, dxinv = P.Scheme(flux_euler=2, rhs_visc=0), P.Closures.nondimensional(1e-3), (3.0, 5.0, 7.0)
    v = rng.standard_normal((5,) + N[::-1])
    W = rng.standard_normal(U.shape) * np.abs(U).reshape(5, -1).max(axis=1)[:, None, None, None]
    JW = ranges._exact_jvp(U, W, cl.gamma, dxinv)
    h = capi.Handle(sc, cl)
    ubar = torch.empty(U.shape, dtype=torch.float64, device="cuda")
    h.rhs_vjp_box(torch.from_numpy(U).cuda(), torch.from_numpy(v).cuda(), ubar, dxinv)
    h.sync_check()
    lhs, rhs = float(np.sum(v * JW)), float(np.sum(ubar.cpu().numpy() * W))
    assert abs(lhs - rhs) <= 1e-11 * (abs(lhs) + np.linalg.norm(v) * np.linalg.norm(JW)), (lhs, rhs)
    h.close()
