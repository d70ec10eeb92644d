"""The KEEP path's range flag reaches the stages that have a cell outside the tested
ranges and no others: in recorded steps of any number of stages replayed on changing
states, in the time loop on the device, in a graph that the caller captures, after a
gradient and after the stage profiler.  Counted on the device
(keep_plain_stages); the results stay the oracle's bits."""
import numpy as np
import pytest
import torch

from amrsolver_gb300 import capi
from amrsolver_gb300 import problems as P
from oracle import pyoracle

pytestmark = pytest.mark.gpu
CL = P.Closures.nondimensional(1e-2)
DXINV = (3.0, 5.0, 7.0)
N = (9, 6, 7)
PER = (-1, -1, -1)
OUT = 1e-90  # a velocity outside the ranges; where it stands (a corner ghost) no face reads it


def _state():
    rng = np.random.default_rng(3)
    shape = tuple(s + 6 for s in N[::-1])
    r = lambda a: a * rng.uniform(-1, 1, shape)  # noqa: E731
    return P.prims_to_cons(1 + r(0.2), r(0.5), r(0.5), r(0.5), 1 + r(0.2), 1.4)


def _mark(t, on):
    t[1, 1, 1, 1] = OUT if on else 0.3


@pytest.mark.parametrize("boxes", [1, 3])
@pytest.mark.parametrize("order,stages", [(1, 1), (2, 2), (3, 3), (3, 4)])
def test_recorded_step(order, stages, boxes):
    """The first stage's input is marked (its ghosts are not filled); the later stages' are the work slots'."""
    capi.load(build_if_missing=True)
    h = capi.Handle(P.Scheme(flux_euler=1, order_keep=4, rhs_visc=1), CL)
    U = torch.from_numpy(_state()).cuda()
    slots = [[U.clone() for _ in range(3)] for _ in range(boxes)]
    bl = capi.BoxList(h, [(20 * b, 0, 0) for b in range(boxes)], slots, DXINV)
    count = 0
    ref = None
    for marked in (0, 1, 1, 0, 0, 2, 0):  # 2: a work slot's ghosts, read by later stages
        for b in range(boxes):
            for s in range(3):
                slots[b][s].copy_(U)
                _mark(slots[b][s], False)
        last = slots[boxes - 1]
        if marked == 1:
            _mark(last[0], True)
            count += 1
        elif marked == 2:
            _mark(last[1], True)
            _mark(last[2], True)
            count += stages - 1
        res = bl.step(order, stages, 1e-3)
        assert bl.keep_plain_stages() == count, (marked,)
        got = slots[0][res][:, 3:-3, 3:-3, 3:-3].clone()
        ref = got if ref is None else ref
        assert torch.equal(got, ref)
    h.close()


def test_device_loop():
    """A step of three stages, the first one's input marked before every run of two steps."""
    capi.load(build_if_missing=True)
    h = capi.Handle(P.Scheme(flux_euler=1, order_keep=4, rhs_visc=1), CL)
    U = torch.from_numpy(_state()).cuda()
    slots = [[U.clone() for _ in range(3)]]
    bl = capi.BoxList(h, [(0, 0, 0)], slots, DXINV)
    for t in slots[0]:
        _mark(t, False)
    for n, marked in enumerate((True, False, True)):
        slots[0][0].copy_(U)
        _mark(slots[0][0], marked)
        before = bl.keep_plain_stages()
        bl.run(3, 3, 1e9, 2, dt=1e-3)  # the ghosts of slot 0 stay: its stage of either step
        assert bl.keep_plain_stages() - before == (2 if marked else 0), n
    h.close()


def test_box_calls():
    """One handle: plain calls, a captured call replayed, a gradient and the stage profiler in between."""
    capi.load(build_if_missing=True)
    h = capi.Handle(P.Scheme(flux_euler=1, order_keep=4, rhs_visc=1), CL)
    A = torch.from_numpy(_state()).cuda()
    _mark(A, False)
    B = A.clone()
    _mark(B, True)
    X = A.clone()
    out = torch.empty((5,) + N[::-1], dtype=torch.float64, device="cuda")
    ref = pyoracle.oracle().rhs(P.Scheme(flux_euler=1, order_keep=4, rhs_visc=1), CL, A.cpu().numpy(), DXINV)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        h.rhs_box(X, DXINV, out, stream=stream)
        stream.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            h.rhs_box(X, DXINV, out, stream=stream)
        count = 0
        for marked in (1, 0, 1, 1, 0, 0):
            X.copy_(B if marked else A)
            count += marked
            g.replay()
            stream.synchronize()
            assert h.keep_plain_stages() == count
            assert np.array_equal(out.cpu().numpy(), ref)
    torch.cuda.synchronize()
    # the reverse pass forms primitives too, and leaves the flag alone
    h.rhs_vjp_box(B, out, torch.empty_like(A), DXINV)
    h.rhs_box(A, DXINV, out)
    assert h.keep_plain_stages() == count
    p = capi.rk_program(1, 1, 1e-3)[0]
    w = A.clone()
    h.profile_stage_box(p, B, A, w, DXINV, reps=3)
    count = h.keep_plain_stages()
    h.profile_stage_box(p, A, A, w, DXINV, reps=3)
    h.rhs_box(A, DXINV, out)
    assert h.keep_plain_stages() == count
    h.close()
