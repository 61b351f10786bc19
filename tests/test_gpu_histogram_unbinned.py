"""The pair histogram after a polymerisation, before the next sort: the new
monomers are in no cell, so they count the neighbours they find in cells and
are nobody's neighbour, whether the two types are the same, differ or are any."""
import numpy as np
import pytest

from spatial_cell_gb300 import abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [0, 1])
@pytest.mark.parametrize("pairs,inactive", [(1, 0), (40, 0), (700, 9)])
def test_new_monomers(product, pairs, inactive, periodic):
    cfg, types, rules, p, m, nid = scenes.polymer_scene(23, pairs, box=max(24.0, 3.0 * (2 * pairs) ** (1 / 3) + 12.0))
    cfg.periodic = periodic
    if inactive:
        p["flags"][1::inactive] = 0
    sim = product.Simulation(cfg, types, rules)
    sim.load_state(p, m, next_particle_id=nid)
    sim.run_phase(abi.PHASE_SORT_PARTICLES)
    sim.run_phase(abi.PHASE_POLYMERIZE)
    q = sim.export_state()[0]
    q = q[q["flags"] & 1 != 0]
    new = q["id"] >= nid
    assert new.sum() == (p["scheduled_polymerization"][p["flags"] & 1 != 0] >= 0).sum()
    x, box = q["pos"].astype(np.float64), np.float64(np.float32(cfg.sim_size))
    d = x[None] - x[:, None]
    if periodic:
        d -= box * np.rint(d / box)
    r = np.sqrt((d * d).sum(2))
    r[:, new] = np.inf          # nobody finds a new monomer
    np.fill_diagonal(r, np.inf)
    bins = 32
    for a, b in ((-1, -1), (scenes.MONO, scenes.MONO), (scenes.MONO, scenes.CTRL), (scenes.CTRL, -1)):
        use = ((a < 0) | (q["type"] == a))[:, None] & ((b < 0) | (q["type"] == b))[None]
        at = (r[use & (r < 5.5)] * bins / 5.5).astype(np.int64)
        assert np.array_equal(sim.pair_histogram(a, b, 5.5, bins), np.bincount(at[at < bins], minlength=bins))
    sim.close()
