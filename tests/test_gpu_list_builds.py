"""The list builds' two-pass scans (scan_words) against the CPU oracle at their
edges: runs of more than 32 candidates and items with more words than the
block holds, periodic boxes from three cells up (images nearer across the
box, split z runs, items away from every face), items that moved more than a
cell, and radii other than their type's."""
import numpy as np
import pytest

from spatial_cell_gb300 import scenes
from tests.helpers import assert_same_counters, assert_same_state

pytestmark = pytest.mark.gpu


def _scene(n, nm, box, periodic, crowd, fast, odd):
    cfg, types, rules, p, m, nid = scenes.test_scene(21, n=n, nm=nm, box=box, species=4, periodic=periodic,
                                                     walls=1 - periodic)
    rng = np.random.default_rng(4)
    if crowd:   # half of the metabolic items and a third of the particles within two cells of one corner
        for s, k in ((m, nm // 2), (p, n // 3)):
            s["pos"][:k] = (rng.random((k, 3)) * 11.0).astype(np.float32)
    if fast:
        m["velocity"][::7] = rng.normal(0.0, 30.0, m["velocity"][::7].shape).astype(np.float32)
    if odd:
        m["radius"][::5] = np.float32(1.25)
        lip = np.nonzero(p["type"] == scenes.LIPID)[0][::3]
        p["radius"][lip] = np.float32(1.5)
    return cfg, types, rules, p, m, nid


@pytest.mark.parametrize("n,nm,box,periodic,crowd,fast,odd", [
    (300, 400, 18.0, 1, 0, 0, 0), (400, 900, 24.5, 1, 0, 1, 1), (600, 1500, 30.0, 1, 1, 0, 0),
    (500, 2500, 43.0, 1, 1, 1, 1), (900, 4000, 66.0, 1, 0, 0, 0), (900, 4000, 66.0, 1, 0, 1, 0),
    (600, 2500, 36.0, 0, 1, 1, 1), (320, 33, 90.0, 0, 0, 0, 0)])
def test_builds(product, n, nm, box, periodic, crowd, fast, odd):
    from oracle.engine import OracleEngine
    cfg, types, rules, p, m, nid = _scene(n, nm, box, periodic, crowd, fast, odd)
    gpu = product.Simulation(cfg, types, rules)
    cpu = OracleEngine("port", cfg, types, rules)
    for e in (gpu, cpu):
        e.load_state(p, m, step=0, next_particle_id=nid)
        e.prepare()
        e.step(2)
    assert_same_state(gpu.export_state(), cpu.export_state(), species=4, what="2 steps")
    assert_same_counters(gpu.counters(), cpu.counters())
