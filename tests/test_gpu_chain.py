"""The kernel chain of the binned sort (k_bin, k_scan, k_pairs_cells,
k_pairs_big, k_match), on grids of more cells than k_resident takes or with
a panel, GPU against the oracle bit for bit.  Bits are compared, so there is no
tolerance."""
import numpy as np
import pytest

from gpusmoldyn_gb300 import _lib as L
from gpusmoldyn_gb300.configs import rng, uniform_positions
from gpusmoldyn_gb300.system import System
from test_gpu_parity import run_parity
from test_gpu_resident import system

pytestmark = pytest.mark.gpu

CELLS = 54  # 157,464 cells of edge 0.25


@pytest.mark.parametrize("births,kernels", [(0.7, 5), (40.0, 5), (499.0, 5), (501.0, 6), (2000.0, 6)])
def test_bins_overflow_beside_births(births, kernels):
    """A cluster overflows its bin while the last CTA of k_bin makes the
    step's births (1,000 by two reactions at most; more are k_zeroth's): the
    step stops whole and is replayed with larger bins."""
    s = system(3000, CELLS, births=births)
    g = rng(17)
    pos = uniform_positions(g, 3000, (0, 0, 0), (0.25 * CELLS,) * 3)
    pos[:400] = uniform_positions(g, 400, (0.3,) * 3, (0.4,) * 3)
    s.set_particles(pos, (np.arange(3000) % 3).astype(np.int32))
    assert s.kernels_per_step() == kernels
    run_parity(s, 6, batch=3)
    s.close()


@pytest.mark.parametrize("sort", ["binned", "compact"])
@pytest.mark.parametrize("n", [2048, 2049, 4097, 65537])
def test_large_cells_without_second_order_reactions(n, sort):
    """Cells cut into units (2,048 records) and joined by one merge pass, or
    by two above 32 units, in a network that has no pairs to find."""
    s = System((-0.75,) * 3, (1.25,) * 3, dt=1e-3, seed=83, normals="table", sort=sort, cell_size=0.5)
    A, B = s.add_species(0.2), s.add_species(0.1)
    s.add_reaction(1, [A], [B], 30.0)
    s.add_reaction(1, [B], [A, A], 20.0)
    if sort == "binned":  # a panel nothing meets, so that the steps are the chain's
        f = s.add_surface()
        s.set_surface_action(f, L.BD_ALL_SPECIES, "both", "transmit")
        s.add_panel(f, "rect", [1.2, -0.75, -0.75, 2.0, 2.0], axis=0)
    s.finalize()
    g = rng(83)
    pos = np.concatenate([uniform_positions(g, n, (-0.15,) * 3, (0.15,) * 3),
                          uniform_positions(g, 300, (0.4,) * 3, (1.25,) * 3)])
    s.set_particles(pos, g.integers(0, 2, len(pos)).astype(np.int32))
    assert s.kernels_per_step() > 1
    run_parity(s, 2)
    s.close()


@pytest.mark.parametrize("n,cells,kernels", [
    (50000, 26, 1),       # 17,576 cells
    (50000, 27, 5),       # 19,683
    (100000, 26, 1),      # the most particles
    (100001, 26, 5),
    (60000, 35, 1),       # 42,875 cells: 1.4 a cell
    (3456, 3, 1),         # 128 a cell
    (3457, 3, 5),         # and one more: large cells are the rule
], ids=lambda v: str(v))
def test_the_line_between_k_resident_and_the_chain(n, cells, kernels):
    s = system(n, cells, kon=0.2)
    assert s.kernels_per_step() == kernels
    run_parity(s, 4, batch=2)
    s.close()
