"""The relax kernels by work class, against the CPU oracle, where their blocks
and lists have edges: bonded items filling the last block of two-thread items
or not, lists shorter and longer than the entries whose geometry is kept,
more than one bond per item, and angular velocities the identity product
does not leave alone (signed zeros, infinities)."""
import numpy as np
import pytest

from spatial_cell_gb300 import abi, scenes
from tests.helpers import diff_fields, mask_state

pytestmark = pytest.mark.gpu


def _scene(bonded, n, box, periodic, seed=5):
    """n particles of lipid / dummy / A / B in a dense box, `bonded` of them in rule-bonded pairs and, for an odd
    count, one serially chain-bonded triple."""
    rng = np.random.default_rng(seed)
    types, rules = scenes.baseline_types(), scenes.baseline_rules()
    p = scenes.uniform_particles(rng, n, box, types)
    p["velocity"] = rng.normal(0.0, 0.3, (n, 3)).astype(np.float32)
    p["angular_velocity"] = scenes.random_quaternions(rng, n)
    free = np.nonzero(p["type"] == scenes.DUMMY)[0]
    p["angular_velocity"][free[:4]] = [[0.0, -0.0, 0.5, -0.8], [-0.0, -0.0, -0.0, -1.0], [-0.0, 0.6, -0.8, 0.0],
                                       [-0.0, -0.3, -0.0, -0.0]]
    p["angular_velocity"][free[4]] = [np.inf, 0.1, -0.0, 1.0]
    ids = rng.permutation(np.setdiff1d(np.arange(n), free[:5]))[:bonded]
    at = 0

    def bond(i, j, kind, group):
        k = p[i]["n_active_interactions"]
        p[i]["interactions"][k] = (kind, group, p[j]["id"])
        p[i]["n_active_interactions"] = k + 1

    if bonded % 2:
        for a, b in ((0, 1), (1, 2)):
            bond(ids[a], ids[b], abi.INTERACTION_TYPE_CHAIN, abi.INTERACTION_GROUP_FORWARD)
            bond(ids[b], ids[a], abi.INTERACTION_TYPE_CHAIN, abi.INTERACTION_GROUP_BACKWARD)
            p["pos"][ids[b]] = p["pos"][ids[a]] + np.float32(0.9)
        at = 3
    for a, b in zip(ids[at::2], ids[at + 1::2]):
        bond(a, b, 1001, 1001)
        bond(b, a, 1001, 1001)
        p["pos"][b] = p["pos"][a] + rng.normal(0.0, 1.0, 3).astype(np.float32)
    p["pos"] = p["pos"].clip(0, np.nextafter(np.float32(box), np.float32(0)))
    m = scenes.uniform_metabolic(rng, 64, box, types, 4)
    cfg = abi.make_config(num_particles=n + 3, num_metabolic_particles=64, sim_size=box, grid_cell_size=6.0,
                          max_interaction_distance=5.5, max_diffusion_distance=6.0, num_metabolites=4, seed=11,
                          periodic=periodic)
    return cfg, types, rules, p, m, n


@pytest.mark.parametrize("streams", [1, 3])
@pytest.mark.parametrize("bonded,n,box,periodic", [(0, 40, 40.0, 0), (127, 400, 60.0, 1), (128, 700, 30.0, 1),
                                                   (129, 700, 42.0, 0), (257, 1300, 36.0, 1)])
def test_relax_classes(product, bonded, n, box, periodic, streams):
    from oracle.engine import OracleEngine
    scene = _scene(bonded, n, box, periodic)
    scene[0].class_streams = streams
    cfg, types, rules, p, m, nid = scene
    gpu = product.Simulation(cfg, types, rules)
    cpu = OracleEngine("port", cfg, types, rules)
    phases = [(abi.PHASE_SORT_PARTICLES, 0), (abi.PHASE_SORT_METABOLIC, 0), (abi.PHASE_RELAX, 0), (abi.PHASE_RELAX, 1),
              (abi.PHASE_RELAX, 2), (abi.PHASE_RELAX, 3), (abi.PHASE_APPLY_NOISE, 0), (abi.PHASE_RELAX, 4),
              (abi.PHASE_RELAX, 5), (abi.PHASE_RELAX, 6)]
    for e in (gpu, cpu):
        e.load_state(p, m, next_particle_id=nid)
    for k, (ph, arg) in enumerate(phases):
        gpu.run_phase(ph, arg)
        cpu.run_phase(ph, arg)
        a, b = mask_state(*gpu.export_state(), species=4)[0], mask_state(*cpu.export_state(), species=4)[0]
        for s in (a, b):   # one NaN for another is no difference
            for f in ("angular_velocity", "angular_noise"):
                s[f] = np.where(np.isnan(s[f]), np.float32(np.nan), s[f])
        assert not diff_fields(a, b), f"phase {k} ({ph})"
