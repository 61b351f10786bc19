"""Items that used to be handled one pair or one item at a time, against the
CPU oracle: particles with a test bond, whose relaxation walks their list (or
the cells, when the list overflowed), and polymerisations that share a
particle, whose list mixes them with ones that do not."""
import numpy as np
import pytest

from spatial_cell_gb300 import abi, scenes
from tests.helpers import assert_same_counters, assert_same_state

pytestmark = pytest.mark.gpu


def _both(product, scene, phases):
    from oracle.engine import OracleEngine
    cfg, types, rules, p, m, nid = scene
    gpu = product.Simulation(cfg, types, rules)
    cpu = OracleEngine("port", cfg, types, rules)
    for e in (gpu, cpu):
        e.load_state(p, m, step=0, next_particle_id=nid)
    for ph, arg in phases:
        gpu.run_phase(ph, arg)
        cpu.run_phase(ph, arg)
        assert_same_state(gpu.export_state(), cpu.export_state(), species=cfg.num_metabolites, what=f"phase {ph}")
        assert_same_counters(gpu.counters(), cpu.counters(), what=f"phase {ph}")
    gpu.close()
    cpu.close()


@pytest.mark.parametrize("periodic", [0, 1])
@pytest.mark.parametrize("limit", [None, 0, 12])
def test_test_bonds_relax_from_the_list(product, limit, periodic):
    rng = np.random.default_rng(3)
    types, rules = scenes.baseline_types(), scenes.baseline_rules()
    n, box = 900, 30.0
    p = scenes.uniform_particles(rng, n, box, types)
    p["velocity"] = rng.normal(0.0, 0.2, (n, 3)).astype(np.float32)
    p["angular_velocity"] = scenes.random_quaternions(rng, n)
    ids = rng.permutation(n)[:160]
    for k, (a, b) in enumerate(zip(ids[::2], ids[1::2])):
        p["pos"][b] = p["pos"][a] + rng.normal(0.0, 1.0, 3).astype(np.float32)
        kinds = ((0, 0), (1001, 1001)) if k % 3 == 0 else ((0, 0),)
        for i, j in ((a, b), (b, a)):
            for s, kind in enumerate(kinds):
                p[i]["interactions"][s] = (*kind, p[j]["id"])
            p[i]["n_active_interactions"] = len(kinds)
    p["pos"] = p["pos"].clip(0, np.nextafter(np.float32(box), np.float32(0)))
    m = scenes.uniform_metabolic(rng, 32, box, types, 2)
    cfg = abi.make_config(num_particles=n + 5, num_metabolic_particles=32, sim_size=box, grid_cell_size=6.0,
                          max_interaction_distance=5.5, max_diffusion_distance=6.0, num_metabolites=2, seed=9,
                          periodic=periodic)
    if limit is not None:
        cfg.pair_list_limit = limit
    _both(product, (cfg, types, rules, p, m, n),
          [(abi.PHASE_SORT_PARTICLES, 0), (abi.PHASE_SORT_METABOLIC, 0)] + [(abi.PHASE_RELAX, k) for k in range(3)])


@pytest.mark.parametrize("pairs,sched,shared,twice", [(1, 1, 0, 0), (255, 0, 254, 0), (256, 30, 30, 0),
                                                      (700, 5, 40, 1), (700, 0, 0, 3)])
def test_mixed_polymerisations(product, pairs, sched, shared, twice):
    """Items in the list's first, last and only block that meet others among ones that do not; `twice` controllers
    hold a second bond of their rule's group."""
    cfg, types, rules, p, m, nid = scenes.polymer_scene(17, pairs, scheduled_monomers=sched, shared=shared)
    for c in range(0, 2 * twice, 2):
        j = p[c]["n_active_interactions"]
        p[c]["interactions"][j] = (1022, 1020, p[c + 3]["id"])
        p[c]["n_active_interactions"] = j + 1
    _both(product, (cfg, types, rules, p, m, nid),
          [(abi.PHASE_SORT_PARTICLES, 0), (abi.PHASE_SORT_METABOLIC, 0), (abi.PHASE_POLYMERIZE, 0)])
