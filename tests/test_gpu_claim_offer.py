"""The pair claim's offers (a warp per open item, a lane per neighbour cell)
against the CPU oracle where the neighbourhood has edges: periodic boxes of
three and four cells, walls on every side, cells holding many items, fewer
open items than a warp and one more than a block's worth of warps."""
import numpy as np
import pytest

from spatial_cell_gb300 import abi, scenes
from tests.helpers import assert_same_counters, assert_same_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,box,periodic,probability", [(1, 18.0, 1, None), (40, 18.5, 1, None), (300, 25.0, 1, 0.5),
                                                        (900, 22.0, 0, 0.5), (9 * 8, 13.0, 0, None),
                                                        (3000, 80.0, 1, 0.1)])
def test_offers(product, n, box, periodic, probability):
    from oracle.engine import OracleEngine
    rng = np.random.default_rng(n)
    types, rules = scenes.baseline_types(), scenes.baseline_rules(probability=probability)
    p = scenes.uniform_particles(rng, n, box, types,
                                 fractions=((scenes.DUMMY, 0.2), (scenes.TYPE_A, 0.4), (scenes.TYPE_B, 0.4)))
    m = scenes.uniform_metabolic(rng, 8, box, types, 4)
    cfg = abi.make_config(num_particles=n, num_metabolic_particles=8, sim_size=box, grid_cell_size=6.0,
                          max_interaction_distance=5.5, max_diffusion_distance=6.0, num_metabolites=4, seed=n,
                          periodic=periodic, walls=1 - periodic, pair_claim=1,
                          rule_probabilities=int(probability is not None))
    gpu, cpu = product.Simulation(cfg, types, rules), OracleEngine("port", cfg, types, rules)
    for e in (gpu, cpu):
        e.load_state(p, m)
        e.prepare()
        for _ in range(3):
            for ph in (abi.PHASE_SORT_PARTICLES, abi.PHASE_APPLY_VELOCITIES, abi.PHASE_COMPLEXIFY, abi.PHASE_END_STEP):
                e.run_phase(ph, 0)
    assert_same_state(gpu.export_state(), cpu.export_state(), species=4)
    assert_same_counters(gpu.counters(), cpu.counters())
    if n >= 40:
        assert (gpu.export_state()[0]["n_active_interactions"] > 0).any()
