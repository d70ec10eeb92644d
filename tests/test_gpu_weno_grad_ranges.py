"""The WENO5 gradient keeps its products and its division on the integer pipe
where one range test per value holds, and takes the hardware's operations
elsewhere: smooth fields, exactly zero differences, a jump between uniform
halves (some differences zero), and fields whose differences lie above and
below the tested range, subnormal ones too.

Check: <v, J w> = <J^T v, w>, J w from the oracle's dual numbers or, where some
differences are zero, from 100 digits: there the rounding of s0 - 4 s1 + 3 s2
(1e-16 against eps = 1e-40) would decide the derivative of the rounded formula.
Tolerance: 1e-11 of |<v, J w>| + |v| |J w|; each entry passes some 300 rounded
operations (2^-53 each, about 3e-14) and the sums run over 5 x 504 of them."""
import numpy as np
import pytest
import torch

from amrsolver_gb300 import capi
from amrsolver_gb300 import problems as P

pytestmark = pytest.mark.gpu
mpmath = pytest.importorskip("mpmath")
mp, mpf = mpmath.mp, mpmath.mpf
N = (9, 8, 7)


def _state(kind):
    rng = np.random.default_rng(17)
    shape = (N[2] + 6, N[1] + 6, N[0] + 6)
    one = np.ones(shape)
    noise = lambda a: a * rng.uniform(-1, 1, shape)  # noqa: E731
    if kind == "smooth":
        f = (1 + noise(0.1), noise(0.3), noise(0.3), noise(0.3), 1 + noise(0.1))
    elif kind == "uniform":
        f = (one, 0.25 * one, 0.0 * one, -0.5 * one, one)
    elif kind == "large":
        f = (1 + noise(0.1), 1e9 * noise(1.0), 1e9 * noise(1.0), 0.0 * one, 1e25 * (2 + noise(1.0)))
    elif kind == "subnormal":
        f = (1 + noise(0.1), noise(1e-309), noise(1e-310), 0.0 * one, 1 + noise(0.1))
    elif kind == "small":
        f = (1e-30 * (2 + noise(1.0)), noise(1e-3), noise(1e-90), 0.0 * one, 1e-33 * (2 + noise(1.0)))
    else:
        left = np.arange(shape[2]) < shape[2] // 2
        f = [np.where(left, a, b) * one for a, b in ((1.0, 0.125), (0.0, 0.0), (0.2, 0.3), (0.1, 0.1), (1.0, 0.1))]
    return P.prims_to_cons(*f, 1.4)


def _exact_jvp(U, W, gamma, dxinv):
    """(R(U + h W) - R(U)) / h of the LLF-split WENO5-JS divergence in 100 digits,
    h = 1e-48; each face's largest wave speed is that of the first cell that has it."""
    ng, n = 3, N

    def rhs(V, pick):
        q = [V[m] / V[0] for m in (1, 2, 3)]
        p = (gamma - 1) * (V[4] - V[0] * (q[0] * q[0] + q[1] * q[1] + q[2] * q[2]) / 2)
        c = np.vectorize(mp.sqrt)(gamma * p / V[0])
        for d in range(3):
            F = [V[m] * q[d] for m in range(4)] + [(V[4] + p) * q[d]]
            F[1 + d] = F[1 + d] + p
            box = [slice(ng, ng + n[2]), slice(ng, ng + n[1]), slice(ng, ng + n[0])]

            def at(a, s):  # cells s below / above the faces of the valid box
                b = list(box)
                b[2 - d] = slice(ng + s, ng + s + n[d] + 1)
                return a[tuple(b)]

            speed = np.stack([at(abs(q[d] + c), s) for s in range(-3, 3)])
            if pick.get(d) is None:
                pick[d] = np.argmax(speed, axis=0)
            al = np.take_along_axis(speed, pick[d][None], 0)[0]
            for m in range(5):
                f, u = [at(F[m], s) for s in range(-3, 3)], [at(V[m], s) for s in range(-3, 3)]
                face = _weno([(f[s] + al * u[s]) / 2 for s in range(5)]) + _weno(
                    [(f[s] - al * u[s]) / 2 for s in (5, 4, 3, 2, 1)])
                acc[m] = acc[m] - dxinv[d] * np.diff(face, axis=2 - d)

    def _weno(s):
        b = [mpf(13) / 12 * (s[i] - 2 * s[i + 1] + s[i + 2]) ** 2 for i in range(3)]
        e = [eps + b[0] + (s[0] - 4 * s[1] + 3 * s[2]) ** 2 / 4, eps + b[1] + (s[1] - s[3]) ** 4 / 4,
             eps + b[2] + (3 * s[2] - 4 * s[3] + s[4]) ** 2 / 4]
        w = [a / (x * x) for a, x in zip((mpf(1) / 10, mpf(6) / 10, mpf(3) / 10), e)]
        v = [2 * s[0] - 7 * s[1] + 11 * s[2], -s[1] + 5 * s[2] + 2 * s[3], 2 * s[2] + 5 * s[3] - s[4]]
        return (w[0] * v[0] + w[1] * v[1] + w[2] * v[2]) / (6 * (w[0] + w[1] + w[2]))

    with mp.workdps(100):
        eps, step, gamma = mpf(10) ** -40, mpf(10) ** -48, mpf(gamma)
        exact = np.vectorize(mpf, otypes=[object])
        A, B, pick, res = exact(U), exact(W), {}, []
        for V in (A, A + step * B):
            acc = [mpf(0)] * 5
            rhs(V, pick)
            res.append(np.stack(acc))
        return ((res[1] - res[0]) / step).astype(np.float64)


@pytest.mark.parametrize("kind", ["smooth", "uniform", "jump", "large", "small", "subnormal"])
def test_vjp_dot_product(orc, kind):
    capi.load(build_if_missing=True)
    U = _state(kind)
    sc = P.Scheme(flux_euler=2, rhs_visc=0)
    cl = P.Closures.nondimensional(1e-3)
    dxinv = (3.0, 5.0, 7.0)
    rng = np.random.default_rng(18)
    v = rng.standard_normal((5,) + N[::-1])
    W = rng.standard_normal(U.shape) * np.abs(U).reshape(5, -1).max(axis=1)[:, None, None, None]
    if kind in ("uniform", "jump"):
        JW = _exact_jvp(U, W, cl.gamma, dxinv)
    else:
        _, JW = orc.rhs_jvp(sc, cl, U, W, dxinv, nthreads=4)
    assert np.isfinite(JW).all()
    h = capi.Handle(sc, cl)
    ubar = torch.empty(U.shape, dtype=torch.float64, device="cuda")
    h.rhs_vjp_box(torch.from_numpy(U).cuda(), torch.from_numpy(v).cuda(), ubar, dxinv)
    h.sync_check()
    lhs, rhs = float(np.sum(v * JW)), float(np.sum(ubar.cpu().numpy() * W))
    assert abs(lhs - rhs) <= 1e-11 * (abs(lhs) + np.linalg.norm(v) * np.linalg.norm(JW)), (lhs, rhs)
    h.close()
