"""Device memory a sim holds before its pools grow, against the sum of its
buffers' bytes per item; the metabolic list's candidates take none of their
own where the diffusion buffer has room for them, and none in the tiled
sweep."""
import pytest

from spatial_cell_gb300 import abi, scenes

pytestmark = pytest.mark.gpu

# Two buffers of the state 480, sort 16, polymerisation 16, particle list 544, bond matches 36, kept geometry 128, bond
# records 16, lipid-metabolic pool 192, the rest 13; with the pair claim 8.
PARTICLE = 1441
# State 236 at eight amounts, sort 16, diffusion buffer 768, list counts, order and overflow 45; 16 bytes per pool entry.
METABOLIC = 1065


@pytest.mark.parametrize("n,nm,tiles", [(65536, 131072, 0), (65536, 262144, 0), (131072, 20000, 0), (65536, 262144, 1)])
def test_bytes_per_item(product, n, nm, tiles):
    box = 200.0
    cfg = abi.make_config(num_particles=n, num_metabolic_particles=nm, sim_size=box, grid_cell_size=6.0,
                          max_interaction_distance=5.5, max_diffusion_distance=6.0, num_metabolites=8, seed=1,
                          periodic=1, pair_claim=1, tiles=tiles)
    sim = product.Simulation(cfg, scenes.baseline_types(), scenes.baseline_rules())
    pool = 4 * 160 if tiles else 12 * 16
    # the lipid list's scratch, where the diffusion buffer is smaller; starts of the cells; look-back words and tables
    rest = (192 * n if 48 * n > 192 * nm else 0) + 8 * abi.grid_dims(cfg)[2] + (1 << 19)
    assert sim.device_bytes() <= n * PARTICLE + nm * (METABOLIC + pool) + rest
    sim.close()
