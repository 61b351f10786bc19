"""One sim that takes a second state: what a step leaves out follows the state
last loaded, not the one its step graphs were captured under.  States with
scheduled polymerisations under rules that schedule none, loaded after (and
before) states without, against the CPU oracle; and a generated scene after
such a state, against a sim of its own."""
import numpy as np
import pytest

from spatial_cell_gb300 import abi, scenes
from tests.helpers import assert_same_counters, assert_same_state

pytestmark = pytest.mark.gpu

KINDS, MIX = (scenes.LIPID, scenes.DUMMY, scenes.TYPE_A, scenes.TYPE_B), (0.4, 0.4, 0.1, 0.1)


def _scene(pool=-1):
    rng = np.random.default_rng(2)
    types, rules = scenes.baseline_types(), scenes.baseline_rules()
    n, box = 400, 40.0
    plain = scenes.uniform_particles(rng, n, box, types)
    plain["scheduled_polymerization"] = -1
    scheduled = plain.copy()
    scheduled["scheduled_polymerization"][::50] = 1001
    m = scenes.uniform_metabolic(rng, 50, box, types, 4)
    cfg = abi.make_config(num_particles=n + 64, num_metabolic_particles=50, sim_size=box, grid_cell_size=6.0,
                          max_interaction_distance=5.5, max_diffusion_distance=6.0, num_metabolites=4, seed=3,
                          periodic=1, graphs=1, pool_per_item=pool)
    return cfg, types, rules, plain, scheduled, m, n


@pytest.mark.parametrize("steps", [1, 2, 3])
@pytest.mark.parametrize("order", ["psp", "sps", "ppss"])
@pytest.mark.parametrize("pool", [-1, 200])
def test_scheduled_polymerisations_of_a_later_load(product, order, steps, pool):
    from oracle.engine import OracleEngine
    cfg, types, rules, plain, scheduled, m, n = _scene(pool)
    gpu = product.Simulation(cfg, types, rules)
    for k, which in enumerate(order):
        cpu = OracleEngine("port", cfg, types, rules)
        for e in (gpu, cpu):
            e.load_state(scheduled if which == "s" else plain, m, step=0, next_particle_id=n)
            e.prepare()
            e.step(steps)
        assert_same_state(gpu.export_state(), cpu.export_state(), species=4, what=f"load {k}")
        assert_same_counters(gpu.counters(), cpu.counters(), what=f"load {k}")
        cpu.close()
    gpu.close()


def test_resumed_checkpoint(product, tmp_path):
    cfg, types, rules, plain, scheduled, m, n = _scene(200)
    sim = product.Simulation(cfg, types, rules)
    sim.load_state(scheduled, m, next_particle_id=n)
    sim.checkpoint(str(tmp_path / "state"))
    sim.close()
    out = []
    for first in (plain, None):   # in a sim that has stepped another state, and in a new one
        sim = product.Simulation(cfg, types, rules)
        if first is not None:
            sim.load_state(first, m, next_particle_id=n)
            sim.step(2)
        sim.resume(str(tmp_path / "state"))
        sim.step(2)
        out.append(sim.export_state())
        assert sim.counters().n_active_particles == n + 8
        sim.close()
    assert_same_state(*out, species=4)


def test_generated_scene_after_a_scheduled_load(product):
    cfg, types, rules, _, scheduled, m, n = _scene(200)
    cfg.graphs = 0
    out = []
    for load in (True, False):
        sim = product.Simulation(cfg, types, rules)
        if load:
            sim.load_state(scheduled, m, next_particle_id=n)
        before = sim.counters().kernel_launches
        sim.generate_uniform(n, 50, KINDS, MIX, 5)
        sim.step(2)
        out.append((sim.counters().kernel_launches - before, sim.export_state()))
        sim.close()
    assert out[0][0] == out[1][0], "launches of a step with nothing to polymerise"
    assert_same_state(out[0][1], out[1][1], species=4)
