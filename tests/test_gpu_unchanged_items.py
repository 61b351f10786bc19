"""What a sub-iteration leaves alone is written only until both buffers hold
it, and passes that cannot act are left out: against the CPU oracle over odd
and even sub-iteration counts (either buffer ends up current), inactive items
among the active ones, and states with scheduled polymerisations under rule
tables that never schedule one."""
import numpy as np
import pytest

from spatial_cell_gb300 import abi, scenes
from tests.helpers import assert_same_counters, assert_same_state

pytestmark = pytest.mark.gpu


def _engines(product, cfg, types, rules, p, m, nid):
    from oracle.engine import OracleEngine
    es = product.Simulation(cfg, types, rules), OracleEngine("port", cfg, types, rules)
    for e in es:
        e.load_state(p, m, step=0, next_particle_id=nid)
    return es


def _one_nan(state):
    """A state with every NaN the same: a monomer made by the zero rule lies on its parent, and which NaN a machine
    gives for the direction between them is its own."""
    for a in state:
        for f in a.dtype.names:
            if a[f].dtype.kind == "f":
                a[f] = np.where(np.isnan(a[f]), np.float32(np.nan), a[f])
    return state


@pytest.mark.parametrize("counts", [(1, 1, 1), (3, 5, 3), (2, 2, 2), (0, 3, 0)])
@pytest.mark.parametrize("graphs", [0, 1])
def test_sub_iteration_parity(product, counts, graphs):
    cfg, types, rules, p, m, nid = scenes.test_scene(31, n=700, nm=1500, box=40.0, species=8, periodic=1)
    cfg.noise_coordination_steps, cfg.relaxation_steps, cfg.metabolite_diffusion_steps = counts
    cfg.graphs = graphs
    rng = np.random.default_rng(1)
    m["flags"][rng.random(len(m)) < 0.3] = 0
    p["flags"][rng.random(len(p)) < 0.1] = 0
    gpu, cpu = _engines(product, cfg, types, rules, p, m, nid)
    for e in (gpu, cpu):
        e.prepare()
        e.step(3)
    assert_same_state(gpu.export_state(), cpu.export_state(), species=8, what=str(counts))
    assert_same_counters(gpu.counters(), cpu.counters())


@pytest.mark.parametrize("spoly", [-1, 0, 1001])
def test_scheduled_without_polymerising_rules(product, spoly):
    """A loaded state's scheduled polymerisations run whatever the rules."""
    rng = np.random.default_rng(2)
    types, rules = scenes.baseline_types(), scenes.baseline_rules()
    n, box = 400, 40.0
    p = scenes.uniform_particles(rng, n, box, types)
    p["scheduled_polymerization"][::50] = spoly
    m = scenes.uniform_metabolic(rng, 50, box, types, 4)
    cfg = abi.make_config(num_particles=n + 64, num_metabolic_particles=50, sim_size=box, grid_cell_size=6.0,
                          max_interaction_distance=5.5, max_diffusion_distance=6.0, num_metabolites=4, seed=3,
                          periodic=1)
    gpu, cpu = _engines(product, cfg, types, rules, p, m, n)
    for e in (gpu, cpu):
        e.prepare()
        e.step(2)
    states = [_one_nan(e.export_state()) for e in (gpu, cpu)]
    assert_same_state(*states, species=4)
    assert_same_counters(gpu.counters(), cpu.counters())
