"""Batched sims whose relax classes have a kernel each (class_streams 3: the
form of batches that fill the device), or one launch (1), against each
replica's own sim and the CPU oracle bit for bit, with bonds, chains and
membranes in the replicas."""
import pytest

from spatial_cell_gb300 import abi, scenes
from tests.helpers import assert_same_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("streams", [1, 3])
@pytest.mark.parametrize("periodic,claim,pairs", [(1, 1, 1), (1, 0, 0), (0, 1, 0)])
def test_uniform_replicas(product, streams, periodic, claim, pairs):
    from oracle.engine import OracleEngine
    reps = scenes.batch_replicas(4, seed=17, n_lo=300, n_hi=4000)
    for cfg, *_ in reps:
        cfg.periodic, cfg.walls, cfg.pair_claim, cfg.metabolic_pairs, cfg.class_streams = periodic, 1 - periodic, claim, \
            pairs, streams
        cfg.noise_coordination_steps, cfg.relaxation_steps, cfg.metabolite_diffusion_steps = 3, 5, 3
    cfg, replicas = scenes.batch_of(reps)
    batch = product.Simulation(cfg, reps[0][1], reps[0][2], replicas=replicas)
    batch.load_batch([(p, m) for *_, p, m in reps])
    batch.prepare()
    batch.step(3)
    for r, (c, types, rules, p, m) in enumerate(reps):
        got = batch.export_replica(r)
        cpu = OracleEngine("port", c, types, rules)
        cpu.load_state(p, m)
        cpu.prepare()
        cpu.step(3)
        assert_same_state(got, cpu.export_state(), species=c.num_metabolites, what=f"replica {r}")
        cpu.close()
    batch.close()


@pytest.mark.parametrize("streams", [1, 3])
def test_structured_replicas(product, streams):
    box = 120.0
    groups = scenes.vesicle_groups(box, shell_r=50.0, lipids=3000, interior=2000, complexes=60, complex_size=20)
    n, nm, seeds = abi.scene_particles(groups), 5000, [5, 9, 11]
    cfg = abi.make_config(num_particles=n, num_metabolic_particles=nm, sim_size=box, grid_cell_size=6.0,
                          max_interaction_distance=5.5, max_diffusion_distance=6.0, num_metabolites=8, seed=5,
                          periodic=0, walls=1, pair_claim=1, rule_probabilities=1, noise_coordination_steps=3,
                          relaxation_steps=5, metabolite_diffusion_steps=3, class_streams=streams)
    types, rules = scenes.baseline_types(), scenes.workload_rules()
    batch = product.Simulation(cfg, types, rules, replicas=[abi.Replica(n, nm, box, 0, sd) for sd in seeds])
    batch.generate_scene_batch(groups, nm, seeds)
    batch.prepare()
    batch.step(3)
    for r, sd in enumerate(seeds):
        c = abi.config_from_bytes(bytes(cfg))
        c.seed, c.class_streams = sd, 0
        solo = product.Simulation(c, types, rules)
        solo.generate_scene(groups, nm, sd)
        solo.prepare()
        solo.step(3)
        assert_same_state(batch.export_replica(r), solo.export_state(), species=8, what=f"replica {r}")
        solo.close()
    batch.close()
