"""The lean metabolic sweep of sims that fill the device, whose overflowed
items have a launch of their own, against the CPU oracle, with capped lists;
and either side of the size where their blocks join the sweep's."""
import numpy as np
import pytest

from spatial_cell_gb300 import abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nm,limit", [(1216 // 4 * 256, 2), (1216 // 4 * 256 + 1, 2), (200_000, -1)])
def test_lean_sweep(product, nm, limit):
    from oracle.engine import OracleEngine
    rng = np.random.default_rng(nm)
    types, rules = scenes.baseline_types(), scenes.baseline_rules()
    box = float((nm / 0.04) ** (1 / 3))
    p = scenes.uniform_particles(rng, 1000, box, types)
    m = scenes.uniform_metabolic(rng, nm, box, types, 1)
    m["velocity"] = rng.normal(0.0, 0.2, (nm, 3)).astype(np.float32)
    cfg = abi.make_config(num_particles=1000, num_metabolic_particles=nm, sim_size=box, grid_cell_size=6.0,
                          max_interaction_distance=5.5, max_diffusion_distance=6.0, num_metabolites=1, seed=3, periodic=1)
    cfg.metabolic_pairs, cfg.pair_list_limit = 0, limit
    out = []
    for make in (lambda: product.Simulation(cfg, types, rules), lambda: OracleEngine("port", cfg, types, rules)):
        e = make()
        e.load_state(p, m, next_particle_id=1000)
        for ph in (abi.PHASE_SORT_PARTICLES, abi.PHASE_SORT_METABOLIC, abi.PHASE_RELAX_METAB, abi.PHASE_RELAX_METAB):
            e.run_phase(ph, 0)
        out.append(e.export_state()[1]["velocity"].copy())
        e.close()
    assert np.array_equal(out[0], out[1])
