"""The cell sort at the sizes where its tiles change (four, eight and sixteen
keys per thread), against numpy's stable sort of the same keys."""
import ctypes

import numpy as np
import pytest

from spatial_cell_gb300 import abi, scenes

pytestmark = pytest.mark.gpu


def _keys(pos, active, box, cell, n_axis):
    g = np.minimum((pos / np.float32(cell)).astype(np.int64), n_axis - 1)
    return np.where(active, (g[:, 0] * n_axis + g[:, 1]) * n_axis + g[:, 2], 1 << 40)


@pytest.mark.parametrize("n", [1, 255, 1024, 1025, 152 * 1024, 152 * 1024 + 1, 262144])
def test_static_sort(product, n):
    import torch
    rng = np.random.default_rng(n)
    box = 90.0
    cfg = abi.make_config(sim_size=box, grid_cell_size=6.0)
    n_axis, _, cells = abi.grid_dims(cfg)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = np.minimum((rng.random((n, 3)) * box).astype(np.float32), np.nextafter(np.float32(box), np.float32(0)))
    info = np.zeros((n, 4), np.int32)
    info[:, 2] = rng.random(n) < 0.9
    d = [torch.from_numpy(x).cuda() for x in (pos, info)]
    perm = torch.zeros(n, dtype=torch.int32, device="cuda")
    starts = torch.zeros(cells + 1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    rc = product.lib().sc_sort_cells_static(ctypes.byref(cfg), *[ctypes.c_void_p(x.data_ptr()) for x in d], n,
                                            ctypes.c_void_p(perm.data_ptr()), ctypes.c_void_p(starts.data_ptr()), None)
    assert rc == 0
    key = _keys(pos[:, :3], info[:, 2] != 0, box, 6.0, n_axis)
    want = np.argsort(key, kind="stable")
    assert np.array_equal(perm.cpu().numpy(), want)
    assert np.array_equal(starts.cpu().numpy(), np.searchsorted(key[want], np.arange(cells + 1)))


@pytest.mark.parametrize("n", [152 * 2048, 152 * 2048 + 1, 400001])
def test_sim_sort(product, n):
    box = float((n / 0.02) ** (1 / 3))
    cfg = abi.make_config(num_particles=n, num_metabolic_particles=8, sim_size=box, grid_cell_size=6.0,
                          max_interaction_distance=5.5, max_diffusion_distance=6.0, num_metabolites=1, seed=1)
    sim = product.Simulation(cfg, scenes.baseline_types(), scenes.baseline_rules())
    sim.generate_uniform(n, 8, (0, 1, 2, 3), (0.25,) * 4, 7)
    before = sim.export_state()[0]
    sim.run_phase(abi.PHASE_SORT_PARTICLES)
    _, perm = sim.export_grid(0)
    key = _keys(before["pos"], before["flags"] & 1 != 0, box, 6.0, abi.grid_dims(cfg)[0])
    assert np.array_equal(perm, np.argsort(key, kind="stable"))
    sim.close()


@pytest.mark.parametrize("n,nm", [(5, 155648), (155648, 300), (70000, 140000), (300, 155649)])
def test_both_sets_of_a_step(product, n, nm):
    """A step's sorts, in the same launches up to 155,648 items a set."""
    box = float((max(n, nm) / 0.02) ** (1 / 3))
    cfg = abi.make_config(num_particles=n, num_metabolic_particles=nm, sim_size=box, grid_cell_size=6.0,
                          max_interaction_distance=5.5, max_diffusion_distance=6.0, num_metabolites=1, seed=1,
                          noise_coordination_steps=0, relaxation_steps=0, metabolite_diffusion_steps=0)
    sim = product.Simulation(cfg, scenes.baseline_types(), scenes.baseline_rules())
    sim.generate_uniform(n, nm, (0, 1, 2, 3), (0.25,) * 4, 7)
    before = sim.export_state()
    sim.step(1)
    for which, state in enumerate(before):
        _, perm = sim.export_grid(which)
        key = _keys(state["pos"], state["flags"] & 1 != 0, box, 6.0, abi.grid_dims(cfg)[0])
        assert np.array_equal(perm, np.argsort(key, kind="stable"))
    sim.close()
