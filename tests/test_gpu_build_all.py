"""The relaxation's pair lists built in one launch, in sims small enough for
it, against the oracle: whole steps launched directly and as graphs, without
relaxation or diffusion sub-iterations, of sets with one item, and with capped
lists."""
import pytest

from spatial_cell_gb300 import scenes
from tests.helpers import assert_same_counters, assert_same_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [0, 1])
@pytest.mark.parametrize("n,nm,relax,diffuse,limit", [(600, 1200, 4, 3, -1), (600, 1200, 0, 2, -1), (600, 1200, 3, 0, 3),
                                                      (300, 1, 1, 1, -1), (1, 700, 2, 2, -1), (700, 700, 2, 1, -1)])
def test_steps(product, n, nm, relax, diffuse, limit, graphs):
    from oracle.engine import OracleEngine
    cfg, types, rules, p, m, nid = scenes.test_scene(4, n=max(n, 300), nm=max(nm, 60), box=36.0)
    p, m = p[:n], m[:nm]
    cfg.relaxation_steps, cfg.metabolite_diffusion_steps, cfg.graphs = relax, diffuse, graphs
    cfg.pair_list_limit = limit
    gpu = product.Simulation(cfg, types, rules)
    cpu = OracleEngine("port", cfg, types, rules)
    for e in (gpu, cpu):
        e.load_state(p, m, step=0, next_particle_id=nid)
        e.step(3)
    assert_same_state(gpu.export_state(), cpu.export_state(), species=cfg.num_metabolites, what="3 steps")
    assert_same_counters(gpu.counters(), cpu.counters(), what="3 steps")
    gpu.close()
    cpu.close()
