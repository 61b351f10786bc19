"""Phases on a sim whose other item set has not been sorted since the sim was
made: it lies in no cell, so the sorted set's items are the only neighbours,
against the CPU oracle.  A sim of the same size runs first, so that buffers
come with what it left in them."""
import numpy as np
import pytest

from spatial_cell_gb300 import abi, scenes
from tests.helpers import assert_same_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lean", [0, 1])
@pytest.mark.parametrize("periodic", [0, 1])
@pytest.mark.parametrize("sort", [abi.PHASE_SORT_PARTICLES, abi.PHASE_SORT_METABOLIC, None])
def test_phases_with_one_set_sorted(product, sort, periodic, lean):
    from oracle.engine import OracleEngine
    cfg, types, rules, p, m, nid = scenes.test_scene(8, n=900, nm=1700, box=40.0, species=4, periodic=periodic)
    cfg.metabolic_pairs = 1 - lean
    first = product.Simulation(cfg, types, rules)
    first.load_state(p, m, next_particle_id=nid)
    first.prepare()
    first.step(1)
    first.sync()
    first.close()
    gpu, cpu = product.Simulation(cfg, types, rules), OracleEngine("port", cfg, types, rules)
    for e in (gpu, cpu):
        e.load_state(p, m, next_particle_id=nid)
    phases = [abi.PHASE_RELAX, abi.PHASE_RELAX_METAB, abi.PHASE_RELAX_PARTNERS, abi.PHASE_RELAX_METAB, abi.PHASE_DIFFUSE]
    for ph in ([] if sort is None else [sort]) + phases:
        gpu.run_phase(ph, 0)
        cpu.run_phase(ph, 0)
        assert_same_state(gpu.export_state(), cpu.export_state(), species=4, what=f"phase {ph}")
    if sort == abi.PHASE_SORT_PARTICLES:   # the metabolic items met lipids
        now = gpu.export_state()[1]
        assert (now["velocity"][:len(m)] != m["velocity"]).any()
    gpu.close()
    cpu.close()
