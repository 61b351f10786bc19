"""Periodic boxes holding positions outside the box (unwrapped coordinates; an
item's cell is the one on the face its index is clamped to): such items and
those in the box find each other through the nearest image, against the CPU
oracle.  Groups of two particles and two metabolic items lie alone in cells on
the faces, so that the neighbourhood is the clamped cell itself."""
import numpy as np
import pytest

from spatial_cell_gb300 import abi, scenes
from tests.helpers import assert_same_counters, assert_same_state, step_phases

pytestmark = pytest.mark.gpu

BOX = 60.0   # ten cells


def _scene(shift, seed=4):
    """shift: which of each group lie a box length outside -- "one" of the two particles and metabolic items, the
    "lipids" alone, the "metabolic" items alone, "all" of them, or "slight": one of them just past its face."""
    rng = np.random.default_rng(seed)
    types, rules = scenes.baseline_types(), scenes.baseline_rules()
    sites = []
    for axis in range(3):
        for u in (10.0, 30.0):
            for v in (10.0, 30.0):
                high = (u == v) != (axis == 1)
                c = np.insert([u, v], axis, BOX - 3.0 if high else 3.0)
                sites.append((c, np.eye(3)[axis] * (BOX if high else -BOX)))
    n = 2 * len(sites)
    p = scenes.uniform_particles(rng, n, BOX, types)
    m = scenes.uniform_metabolic(rng, n, BOX, types, 4)
    pairs = [(scenes.LIPID, scenes.LIPID), (scenes.DUMMY, scenes.DUMMY), (scenes.TYPE_A, scenes.TYPE_B),
             (scenes.LIPID, scenes.DUMMY)]
    for k, (c, out) in enumerate(sites):
        for s in (0, 1):
            i = 2 * k + s
            p["type"][i] = pairs[k % 4][s]
            for a in (p, m):
                a["pos"][i] = c + rng.uniform(-1.0, 1.0, 3)
            one = out if shift != "slight" else out / BOX * 3.5   # from 2 to 4 nm off the face
            if shift == "all" or shift == "lipids" or (shift in ("one", "slight") and s):
                p["pos"][i] += one
            if shift == "all" or shift == "metabolic" or (shift in ("one", "slight") and s):
                m["pos"][i] += one
    p["radius"], p["hydrophobic"] = types["radius"][p["type"]], types["hydrophobic"][p["type"]]
    p["velocity"] = rng.normal(0.0, 0.1, (n, 3)).astype(np.float32)
    m["velocity"] = rng.normal(0.0, 0.1, (n, 3)).astype(np.float32)
    for i, j in ((2 * k + s, 2 * k + 1 - s) for k in range(2, len(sites), 8) for s in (0, 1)):   # bonds across the face
        p[i]["interactions"][0] = (1001, 1001, p[j]["id"])
        p[i]["n_active_interactions"] = 1
    cfg = abi.make_config(num_particles=n, num_metabolic_particles=n, sim_size=BOX, grid_cell_size=6.0,
                          max_interaction_distance=5.5, max_diffusion_distance=6.0, num_metabolites=4, seed=seed,
                          periodic=1, noise_coordination_steps=3, relaxation_steps=5, metabolite_diffusion_steps=2)
    return cfg, types, rules, p, m, n


@pytest.mark.parametrize("shift", ["one", "lipids", "metabolic", "all", "slight"])
@pytest.mark.parametrize("pairs,streams", [(1, 0), (0, 3)])
def test_steps(product, shift, pairs, streams):
    from oracle.engine import OracleEngine
    cfg, types, rules, p, m, nid = _scene(shift)
    cfg.metabolic_pairs, cfg.class_streams = pairs, streams
    gpu, cpu = product.Simulation(cfg, types, rules), OracleEngine("port", cfg, types, rules)
    for e in (gpu, cpu):
        e.load_state(p, m, step=0, next_particle_id=nid)
        e.step(2)
    assert_same_state(gpu.export_state(), cpu.export_state(), species=4, what="2 steps")
    assert_same_counters(gpu.counters(), cpu.counters(), what="2 steps")
    gpu.close()
    cpu.close()


@pytest.mark.parametrize("shift", ["one", "lipids", "metabolic", "all", "slight"])
def test_phases(product, shift):
    from oracle.engine import OracleEngine
    cfg, types, rules, p, m, nid = _scene(shift)
    gpu, cpu = product.Simulation(cfg, types, rules), OracleEngine("port", cfg, types, rules)
    for e in (gpu, cpu):
        e.load_state(p, m, step=0, next_particle_id=nid)
    for k, (ph, arg) in enumerate(step_phases(cfg)):
        gpu.run_phase(ph, arg)
        cpu.run_phase(ph, arg)
        assert_same_state(gpu.export_state(), cpu.export_state(), species=4, what=f"phase {k} ({ph})")
        if ph == abi.PHASE_RELAX_PARTNERS:
            assert all(c >= len(p) // 4 for c in gpu.pair_counts()[:3])
    gpu.close()
    cpu.close()
