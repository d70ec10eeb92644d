"""The ghost fill deals ghost cells (planes beyond z, rows beyond y, cells beyond x)
to threads: every ghost of boxes down to one cell, of unequal edges, under each
boundary code and for component counts other than five, against the oracle's
fill (which itself needs three cells per direction) and against the index map
written in numpy.  Ghosts start as NaN, so a cell the enumeration misses shows.

Tolerance: none.  A fill copies values and changes signs."""
import numpy as np
import pytest
import torch

from amrsolver_gb300 import capi
from oracle import pyoracle

pytestmark = pytest.mark.gpu
G = 3


def _field(n, ncomp):
    rng = np.random.default_rng(sum(n))
    U = np.full((ncomp, n[2] + 2 * G, n[1] + 2 * G, n[0] + 2 * G), np.nan)
    U[:, G:-G, G:-G, G:-G] = rng.uniform(-1, 1, (ncomp,) + n[::-1])
    return U


def _mapped(U, bc):
    """The fill as an index map per direction: periodic wrap, clamp, reflection with its signs."""
    idx, sign = [], []
    for d in range(3):
        m = U.shape[3 - d] - 2 * G
        i, s = [], []
        for c in range(-G, m + G):
            code = bc[0][d] if c < 0 else bc[1][d] if c >= m else None
            mirror = code in (3, 4, 5)
            i.append(c % m if code == -1 else min(max(c, 0), m - 1) if code == 2 else
                     (-c - 1 if c < 0 else 2 * m - 1 - c) if mirror else c)
            s.append([-1.0 if mirror and (1 <= q <= 3 if code == 5 else q == 1 + d) else 1.0
                      for q in range(U.shape[0])])
        idx.append(np.array(i) + G)
        sign.append(np.array(s).T)
    V = U[:, idx[2][:, None, None], idx[1][None, :, None], idx[0][None, None, :]]
    return V * sign[2][:, :, None, None] * sign[1][:, None, :, None] * sign[0][:, None, None, :]


@pytest.mark.parametrize("n", [(1, 1, 1), (2, 1, 3), (40, 1, 2), (1, 9, 1), (3, 4, 5), (33, 3, 17)])
@pytest.mark.parametrize("bc", [((-1, -1, -1), (-1, -1, -1)), ((2, -1, 2), (2, -1, 2)), ((2, 3, 5), (4, 2, 3)),
                                ((5, 4, -1), (3, 5, -1))])
def test_fill(n, bc):
    reflects = any(c not in (-1, 2) and n[d] < G for d in range(3) for c in (bc[0][d], bc[1][d]))
    if reflects:
        pytest.skip("a reflection needs three cells")
    capi.load(build_if_missing=True)
    U = _field(n, 5)
    ref = _mapped(U, bc)
    if min(n) >= G:
        orc = U.copy()
        pyoracle.oracle().fill_halo(orc, bc[0], bc[1])
        assert np.array_equal(orc, ref)
    d = torch.from_numpy(U).cuda()
    capi.fill_halo_box(d, bc[0], bc[1])
    got = d.cpu().numpy()
    assert np.isfinite(ref).all()
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("ncomp", [1, 3, 7])
def test_other_component_counts(ncomp):
    capi.load(build_if_missing=True)
    n, bc = (5, 4, 6), ((2, 3, 5), (4, 2, 3))
    U = _field(n, ncomp)
    d = torch.from_numpy(U).cuda()
    capi.fill_halo_box(d, bc[0], bc[1])
    got = d.cpu().numpy()
    for c in range(ncomp):
        # components beyond the momenta keep their sign, as the density does
        A = _field(n, 5)
        slot = c if c < 5 else 0
        A[slot] = U[c]
        pyoracle.oracle().fill_halo(A, bc[0], bc[1])
        assert np.array_equal(got[c], A[slot]), c
