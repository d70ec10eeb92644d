"""Lists whose divergence scratch exceeds its bound run the KEEP face kernels in pieces:
boxes of more than 2^31 / 80 = 26.8 million cells in slabs of planes, lists of more in
groups of boxes.  Reference: the same cells as separate boxes below the bound.

Tolerance: none.  A cell's operations do not depend on the box that it is in."""
import pytest
import torch

from amrsolver_gb300 import capi
from amrsolver_gb300 import problems as P

pytestmark = pytest.mark.gpu
CL = P.Closures.nondimensional(1e-2)
DXINV = (3.0, 5.0, 7.0)


def _random(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (n[2] + 6, n[1] + 6, n[0] + 6)
    r = lambda a: a * (2.0 * torch.rand(shape, generator=g, dtype=torch.float64, device="cuda") - 1.0)  # noqa: E731
    U = torch.empty((5,) + shape, dtype=torch.float64, device="cuda")
    U[0] = 1.0 + r(0.2)
    for c in (1, 2, 3):
        U[c] = r(0.5)
    U[4] = 2.5 * (1.0 + r(0.2)) + 0.5 * (U[1] ** 2 + U[2] ** 2 + U[3] ** 2) / U[0]
    return U


def _rhs(h, U):
    out = torch.empty((5,) + tuple(s - 6 for s in U.shape[1:]), dtype=torch.float64, device="cuda")
    return h.rhs_box(U, DXINV, out)


def _in_parts(h, U, z):
    """The same right-hand side from two boxes that meet at plane z."""
    return torch.cat([_rhs(h, U[:, :z + 6].contiguous()), _rhs(h, U[:, z:].contiguous())], dim=1)


@pytest.mark.parametrize("order,visc", [(4, 1), (6, 0)])
def test_slabs_of_one_box(order, visc):
    capi.load(build_if_missing=True)
    h = capi.Handle(P.Scheme(flux_euler=1, order_keep=order, rhs_visc=visc), CL)
    n = (372, 369, 392)  # 195, 195 and 2 planes
    U = _random(n, 1)
    U[1, 1, 1, 1] = 1e-90  # a corner that no face reads: the stage runs, and counts once, on the FP64 pipe
    a = torch.empty((5,) + n[::-1], dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    h.rhs_box(U, DXINV, a)
    assert h.keep_plain_stages() == 1
    # the primitives, the viscous cell fluxes and the bound; 80 bytes a cell would be 4.3 GB
    cells = lambda g: (n[0] + 2 * g) * (n[1] + 2 * g) * (n[2] + 2 * g)  # noqa: E731
    used = free - torch.cuda.mem_get_info()[0]
    assert used <= 56 * cells(3) + 96 * visc * cells(1) + 2**31 + 2**28, used
    U[1, 1, 1, 1] = 0.3
    b = _rhs(h, U)
    assert h.keep_plain_stages() == 1
    assert torch.equal(a, b)
    assert torch.equal(b, _in_parts(h, U, 150))
    h.close()


def test_groups_and_slabs_of_a_list():
    """A small box, one in slabs, and more boxes than one group holds."""
    capi.load(build_if_missing=True)
    h = capi.Handle(P.Scheme(flux_euler=1, order_keep=4, rhs_visc=1), CL)
    ns = [(33, 20, 17), (300, 300, 299), (9, 8, 7)] + [(220, 200, 210)] * 3 + [(12, 40, 5)]
    los, slots, x = [], [], 0
    for b, n in enumerate(ns):
        los.append((x, 0, 0))
        x += n[0] + 10
        U = _random(n, 10 + b)
        slots.append([U, torch.full_like(U, 7.0)])
    bl = capi.BoxList(h, los, slots, DXINV)
    p = capi.rk_program(0, 1, 0.0)[0]  # S2 = dS
    bl.stage(p, 0, 0, 1)
    assert bl.keep_plain_stages() == 0
    for n, (U, out) in zip(ns, slots):
        ref = _in_parts(h, U, 150) if n[2] > 250 else _rhs(h, U)
        assert torch.equal(out[:, 3:-3, 3:-3, 3:-3], ref), n
    bl.close()
    h.close()
