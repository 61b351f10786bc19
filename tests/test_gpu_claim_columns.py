"""The pair claim's offers, three open items a warp and a lane per column of
an item's neighbourhood, against the CPU oracle at the edges of that split:
open items filling a warp's three places or not, a block's 24 or not, and more
than the grid takes at once."""
import numpy as np
import pytest

from spatial_cell_gb300 import abi, scenes
from tests.helpers import assert_same_counters, assert_same_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [0, 1])
@pytest.mark.parametrize("opened,n,box", [(1, 60, 20.0), (2, 60, 20.0), (3, 60, 20.0), (4, 60, 20.0), (24, 300, 24.5),
                                          (25, 300, 24.5), (26, 700, 31.0), (4 * 1216 * 24 + 7, 130_000, 200.0)])
def test_open_items(product, opened, n, box, periodic):
    from oracle.engine import OracleEngine
    rng = np.random.default_rng(opened)
    types, rules = scenes.baseline_types(), scenes.baseline_rules()
    p = scenes.uniform_particles(rng, n, box, types)
    p["type"] = scenes.DUMMY
    ids = rng.permutation(n)[:opened]
    p["type"][ids] = np.where(np.arange(opened) % 2, scenes.TYPE_A, scenes.TYPE_B)
    p["radius"], p["hydrophobic"] = types["radius"][p["type"]], types["hydrophobic"][p["type"]]
    if opened < 100:   # each beside the one before
        for a, b in zip(ids, ids[1:]):
            p["pos"][b] = p["pos"][a] + rng.normal(0.0, 2.0, 3)
        p["pos"] = p["pos"].clip(0, np.nextafter(np.float32(box), np.float32(0)))
    m = scenes.uniform_metabolic(rng, 8, box, types, 1)
    cfg = abi.make_config(num_particles=n, num_metabolic_particles=8, sim_size=box, grid_cell_size=6.0,
                          max_interaction_distance=5.5, max_diffusion_distance=6.0, num_metabolites=1, seed=7,
                          periodic=periodic, walls=1 - periodic, pair_claim=1)
    gpu, cpu = product.Simulation(cfg, types, rules), OracleEngine("port", cfg, types, rules)
    for e in (gpu, cpu):
        e.load_state(p, m, next_particle_id=n)
        for ph in (abi.PHASE_SORT_PARTICLES, abi.PHASE_COMPLEXIFY, abi.PHASE_COMPLEXIFY):
            e.run_phase(ph, 0)
    got = gpu.export_state()
    assert_same_state(got, cpu.export_state(), species=1)
    assert_same_counters(gpu.counters(), cpu.counters())
    if opened > 1:
        assert (got[0]["n_active_interactions"] > 0).any()
    gpu.close()
    cpu.close()
