"""The metabolic sweep's blocks of several 256-item groups, their number a
rule of the sim's size, against the plain relaxation phase of the CPU oracle:
sizes either side of the first two rules' lines and a ragged last block."""
import numpy as np
import pytest

from spatial_cell_gb300 import abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nm", [2 * 2 * 1216 * 256 - 300, 2 * 2 * 1216 * 256 + 1, 3 * 2 * 1216 * 256 + 257])
def test_sweep(product, nm):
    from oracle.engine import OracleEngine
    rng = np.random.default_rng(nm)
    types, rules = scenes.baseline_types(), scenes.baseline_rules()
    box = float((nm / 0.03) ** (1 / 3))
    p = scenes.uniform_particles(rng, 2000, box, types)
    m = scenes.uniform_metabolic(rng, nm, box, types, 1)
    m["velocity"] = rng.normal(0.0, 0.2, (nm, 3)).astype(np.float32)
    cfg = abi.make_config(num_particles=2000, num_metabolic_particles=nm, sim_size=box, grid_cell_size=6.0,
                          max_interaction_distance=5.5, max_diffusion_distance=6.0, num_metabolites=1, seed=3, periodic=1)
    out = []
    for make in (lambda: product.Simulation(cfg, types, rules), lambda: OracleEngine("port", cfg, types, rules)):
        e = make()
        e.load_state(p, m, next_particle_id=2000)
        for ph in (abi.PHASE_SORT_PARTICLES, abi.PHASE_SORT_METABOLIC, abi.PHASE_RELAX_METAB, abi.PHASE_RELAX_METAB):
            e.run_phase(ph, 0)
        out.append(e.export_state()[1]["velocity"].copy())
        e.close()
    assert np.array_equal(out[0], out[1])
