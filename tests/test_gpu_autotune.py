"""The autotuner times what changes the launches (the waves) and nothing else, reports the
list's own tiles, and takes a saved choice up again."""
import pytest
import torch

from amrsolver_gb300 import autotune, capi
from amrsolver_gb300 import problems as P

pytestmark = pytest.mark.gpu


def test_sweep_and_cache(tmp_path):
    capi.load(build_if_missing=True)
    specs, fields, dx = P.batched_boxes(nboxes=3, seed=5, edges=(8, 24, 40))
    h = capi.Handle(P.Scheme(flux_euler=1, order_keep=4, rhs_visc=1), P.Closures.nondimensional(1e-3))
    slots = [[torch.from_numpy(U).cuda() for _ in range(3)] for U in fields]
    before = [s[0].clone() for s in slots]
    bl = capi.BoxList(h, [s.lo for s in specs], slots, [1.0 / v for v in dx])
    shapes = [tuple(s.shape) for s in specs]
    tiles = bl.get_tiles()
    path = str(tmp_path / "tune.json")
    rep = autotune.tune_level(bl, shapes, cache_path=path)
    assert rep["candidates_timed"] == len(rep["sweep"]) == len(autotune.WAVES) + 2
    assert sorted({e["waves"] for e in rep["sweep"]}) == sorted(autotune.WAVES)
    assert rep["waves"] in autotune.WAVES and rep["tuned_ms"] <= rep["default_ms"] and not rep["cached"]
    assert bl.get_tiles() == tiles == [tuple(t) for t in rep["tiles"]]
    assert set(rep["class_tiles"]) == {"%dx%d" % s[:2] for s in shapes}
    again = autotune.tune_level(bl, shapes, cache_path=path)
    assert again["cached"] and again["waves"] == rep["waves"] and again["tiles"] == rep["tiles"]
    assert all(torch.equal(a, s[0]) for a, s in zip(before, slots))
    h.close()
