"""Cotangents that are not finite through the reverse of a stage program: a register
that the program reads takes them even where its coefficient is zero (0 * NaN is a
NaN), one that it does not read stays untouched.

Reference: the program reversed value by value in torch, then the right-hand side's
own VJP and the ghost fold.  The places that are not finite are compared exactly;
the finite ones within 1e-13 of the largest (a few roundings: the kernel multiplies
the cotangent by one product of coefficients, the reference by each in turn)."""
import pytest
import torch

from amrsolver_gb300 import capi
from amrsolver_gb300 import problems as P

pytestmark = pytest.mark.gpu
N = (8, 7, 6)
DXINV = (3.0, 5.0, 7.0)
PER = (-1, -1, -1)


def _reverse(p, w):
    b = [torch.zeros_like(w), w.clone(), torch.zeros_like(w)]
    for o in range(p.nops - 1, -1, -1):
        q = p.ops[o]
        g = b[q.dst].clone()
        if q.kind == 0:
            b[q.dst] = torch.zeros_like(w)
            b[q.x] = b[q.x] + q.a * g
            b[q.y] = b[q.y] + q.b * g
        elif q.kind == 1:
            b[q.x] = b[q.x] + q.a * g
        elif q.kind == 2:
            b[q.dst] = q.a * g
            b[q.x] = b[q.x] + g
        else:
            b[q.dst] = torch.zeros_like(w)
            b[q.x] = b[q.x] + g
    return b


def _progs():
    for order, stages in ((3, 3), (1, 1), (2, 2), (-2, 2)):
        for dt in (0.0, 1e-3):
            for i, p in enumerate(capi.rk_program(order, stages, dt)):
                yield "rk %d %d dt %g stage %d" % (order, stages, dt, i), p
    p = capi.rk_program(1, 1, 1e-3)[0]  # S2 = a S1 + b dS
    p.ops[0].a = 0.0
    yield "S1 times zero", p


@pytest.mark.parametrize("ghosted", [False, True])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_program_reverse(value, ghosted):
    capi.load(build_if_missing=True)
    h = capi.Handle(P.Scheme(flux_euler=1, order_keep=4, rhs_visc=1), P.Closures.nondimensional(1e-2))
    U = torch.from_numpy(P.random_state(N, seed=1)).cuda()
    capi.fill_halo_box(U, PER, PER)
    gen = torch.Generator().manual_seed(5)
    w = torch.randn(5, N[2], N[1], N[0], dtype=torch.float64, generator=gen).cuda()
    w[1, 3, 2, 4] = value
    for name, p in _progs():
        b = _reverse(p, w)
        ub = torch.empty_like(U)
        h.rhs_vjp_box(U, b[2], ub, DXINV)
        s1 = torch.ones_like(w)
        if ghosted:
            got = torch.empty_like(U)
            h.rk_stage_vjp_box_ghosted(p, U, w, s1, got, DXINV)
            ref = ub
            ref[:, 3:-3, 3:-3, 3:-3] += b[1]
        else:
            got = torch.ones_like(w)
            h.rk_stage_vjp_box(p, PER, PER, U, w, s1, got, DXINV)
            capi.fill_halo_box_adjoint(ub, PER, PER)
            ref = ub[:, 3:-3, 3:-3, 3:-3] + b[1] + 1.0
        for what, a, r in (("in", got, ref), ("s1", s1, b[0] + 1.0)):
            fin = torch.isfinite(r)
            assert torch.equal(torch.isfinite(a), fin), (name, what, int((~fin).sum()), int((~torch.isfinite(a)).sum()))
            scale = float(r[fin].abs().max())
            assert float((a[fin] - r[fin]).abs().max()) <= 1e-13 * max(scale, 1.0), (name, what)
    h.close()
