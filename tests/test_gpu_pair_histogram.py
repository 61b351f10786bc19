"""The pair histogram against all pairs in double precision: boxes of three
cells up, walled and periodic, items on the faces, pairs of one type, of two
and of any, and distances on the bins' edges."""
import numpy as np
import pytest

from spatial_cell_gb300 import abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,box,periodic,bins", [(300, 18.0, 1, 64), (500, 25.0, 1, 33), (400, 26.0, 0, 64),
                                                 (900, 61.0, 1, 128)])
def test_histogram(product, n, box, periodic, bins):
    rng = np.random.default_rng(n)
    types = scenes.baseline_types()
    p = scenes.uniform_particles(rng, n, box, types)
    p["pos"][:6] = [[0, 0, 0], [box, box, box], [0, box, 1], [box, 0, 1], [3, 3, 0], [3, 3, box]]
    p["pos"][20:40] = p["pos"][6] + np.arange(20, dtype=np.float32)[:, None] * np.float32([0, 0.25, 0])
    p["pos"] = p["pos"].clip(0, box)
    p["flags"][::9] = 0
    m = scenes.uniform_metabolic(rng, 4, box, types, 1)
    cfg = abi.make_config(num_particles=n, num_metabolic_particles=4, sim_size=box, grid_cell_size=6.0,
                          max_interaction_distance=5.5, max_diffusion_distance=6.0, num_metabolites=1, seed=1,
                          periodic=periodic)
    sim = product.Simulation(cfg, types, scenes.baseline_rules())
    sim.load_state(p, m)
    x = p["pos"].astype(np.float64)
    d = x[None] - x[:, None]
    if periodic:
        d -= np.float64(np.float32(box)) * np.rint(d / np.float64(np.float32(box)))
    r = np.sqrt((d * d).sum(2))
    act = p["flags"] & 1 != 0
    for a, b in ((-1, -1), (scenes.TYPE_A, scenes.TYPE_B), (scenes.LIPID, -1)):
        use = (act & ((a < 0) | (p["type"] == a)))[:, None] & (act & ((b < 0) | (p["type"] == b)))[None]
        np.fill_diagonal(use, False)
        near = r[use & (r < 5.5)]
        at = (near * bins / 5.5).astype(np.int64)
        assert np.array_equal(sim.pair_histogram(a, b, 5.5, bins), np.bincount(at[at < bins], minlength=bins))
    sim.close()
